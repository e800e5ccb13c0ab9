// The routed experts on the tensor cores.
//
// Stands where the reference's prefill entry multiplies items of up to 64 rows with warp-level MMAs
// (kernel/src/moe_prefill.cu:252-262, kernels :405 and :421) and its decode entry walks the records
// with vector dot products (moe_decode.cu:325-399). Under skewed routing a few experts see
// hundreds of rows; here a work item is up to 192 sorted rows of one expert, and every item is
// multiplied with its expert's record by the kernel core of trellis_tc.cuh: the rows rotated once
// into plain fp16 rows with one scale per row, the record's trellis tiles decoded into
// tensor memory, tcgen05.mma kind::f16 with the accumulator beside them, and the output
// Hadamard in the epilogue. Five launches behind the grouping:
//
//   moe_tc_rotate_x_kernel    x o suh (the row's expert's gate|up record), Hadamard, fp16 rows
//   moe_tc_gemm_kernel<0>     rows x gate|up record -> gu fp32 [row][2 inter] (gate columns, then up)
//   moe_tc_rotate_h_kernel    silu(g) u o suh (the down record), Hadamard, fp16 rows
//   moe_tc_gemm_kernel<1>     rows x down record, times the routing weight -> fp32 [token][rank][hidden]
//   moe_tc_fold_kernel        a token's products as 2^-32 fixed-point integers, summed, added to the
//                             token's int64 accumulator row (84 M atomic additions into the
//                             accumulator from the product's epilogue took two thirds of that launch)
//
// A row's arithmetic does not depend on the item it is in or on the rows beside it, so results are
// reproducible bit for bit whatever the grouping order.
#include "moe_internal.cuh"
#include "trellis_tc.cuh"

namespace b200q {
namespace {

using namespace trellis_tc;
static_assert(kMoeTcItemRows == Shape<2>::kMaxRows, "an item is what a CTA takes");

// The sorted rows' activations (rotate_row, trellis_device.cuh), a CTA going from row to row: the token's `hidden` values times the
// expert's suh, the 128-wide Hadamard per block, one power-of-two scale per row, fp16. A lane holds 32 values, so that five of
// the seven Hadamard stages are additions of two values an instruction. (Four values a lane: 102 us for 40 960 rows of 2048 inputs
// against 77.) THREADS: the most a launch has.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) moe_tc_rotate_x_kernel(const __grid_constant__ ExpertParams p, const uint32_t *offsets) {
  __shared__ float warp_max[2][32];
  griddep_launch_dependents();
  griddep_wait();
  const uint32_t in = p.hidden;
  const uint32_t rows = offsets[p.experts];   // fewer than the launch may have been sized for
  float *const inv = p.x_scale;
  struct Source {
    uint32_t a;
    ignis_moe_slot slot;
  };
  auto source = [&](uint32_t row) {   // four loads that depend on one another: for the next row while this one is transformed
    Source s = {};
    if (row < rows) {
      s.a = p.sorted[row];
      s.slot = p.slots[static_cast<uint32_t>(p.ids[s.a]) * 2u];
    }
    return s;
  };
  Source here = source(blockIdx.x);
  for (uint32_t row = blockIdx.x, turn = 0; row < rows; row += gridDim.x, turn ^= 1u) {
    const Source next = source(row + gridDim.x);
    const ignis_moe_slot slot = here.slot;
    uint16_t *const to = p.x_rows + static_cast<size_t>(row) * in;
    if (slot.record == nullptr || !(slot.k2 == 4 || slot.k2 == 5 || slot.k2 == 6 || slot.k2 == 8)) {
      // an absent record: the product kernel flags it and skips the item; leave finite rows behind
      for (uint32_t i = threadIdx.x * 4u; i < in; i += 4u * blockDim.x) *reinterpret_cast<uint2 *>(to + i) = make_uint2(0u, 0u);
      if (threadIdx.x == 0) inv[row] = 0.0f;
      __syncthreads();   // as a rotated row would: the turn after the next writes its maxima where the turn before wrote its own
    } else {
      const uint64_t trellis_bytes = static_cast<uint64_t>(in) * 2u * p.inter * slot.k2 / 16u;
      const uint16_t *suh = reinterpret_cast<const uint16_t *>(static_cast<const uint8_t *>(slot.record) + trellis_bytes);
      const uint16_t *x = p.x + static_cast<size_t>(here.a / p.top_k) * in;
      rotate_row(in, to, inv + row, warp_max[turn],
                 [&](uint32_t k, float2 (&v)[4]) { scaled_inputs(ldg128_coherent(x + k), __ldg(reinterpret_cast<const uint4 *>(suh + k)), v); });
    }
    here = next;
  }
}

// silu(g) u of a sorted row's gate|up products, rotated for the down record: a CTA of two warps per row, a warp per 128-input
// block, the row's values waiting in shared memory for its scale. Bound by the sigmoid and the division as much as by the
// transform: 70 us for 40 960 rows of 768, where rotate_row takes 76 (a warp with a quarter of its lanes idle) and 108 from row
// to row.
constexpr uint32_t kRotateThreads = 64;
__global__ void __launch_bounds__(kRotateThreads) moe_tc_rotate_h_kernel(const __grid_constant__ ExpertParams p, const uint32_t *offsets) {
  extern __shared__ __align__(16) float rot[];
  __shared__ float warp_max[kRotateThreads / 32];
  griddep_launch_dependents();
  griddep_wait();
  const uint32_t row = blockIdx.x;
  if (row >= offsets[p.experts]) return;   // fewer rows than the launch was sized for
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t a = p.sorted[row];
  const uint32_t expert = static_cast<uint32_t>(p.ids[a]);
  const ignis_moe_slot slot = p.slots[expert * 2u + 1u];
  const uint32_t in = p.inter;
  uint16_t *dst = p.h_rows + static_cast<size_t>(row) * in;
  float *inv = p.h_scale + row;
  if (slot.record == nullptr || !(slot.k2 == 4 || slot.k2 == 5 || slot.k2 == 6 || slot.k2 == 8)) {
    // an absent record: the product kernel flags it and skips the item; leave finite rows behind
    for (uint32_t i = threadIdx.x * 4u; i < in; i += 4u * kRotateThreads) *reinterpret_cast<uint2 *>(dst + i) = make_uint2(0u, 0u);
    if (threadIdx.x == 0) *inv = 0.0f;
    return;
  }
  const uint64_t trellis_bytes = static_cast<uint64_t>(in) * p.hidden * slot.k2 / 16u;
  const uint16_t *suh = reinterpret_cast<const uint16_t *>(static_cast<const uint8_t *>(slot.record) + trellis_bytes);
  const uint32_t nblk = in / 128u;
  float m = 0.0f;
  for (uint32_t bl = static_cast<uint32_t>(warp); bl < nblk; bl += kRotateThreads / 32u) {
    const size_t k0 = static_cast<size_t>(bl) * 128u + 4u * lane;
    const uint2 sb = *reinterpret_cast<const uint2 *>(suh + k0);
    const __half2 s01 = *reinterpret_cast<const __half2 *>(&sb.x), s23 = *reinterpret_cast<const __half2 *>(&sb.y);
    const float sv[4] = {__low2float(s01), __high2float(s01), __low2float(s23), __high2float(s23)};
    float v[4];
    const float *g = p.gu + static_cast<size_t>(row) * 2u * p.inter + k0;
    const uint4 gb = ldg128_coherent(g), ub = ldg128_coherent(g + p.inter);
    const float gv[4] = {__uint_as_float(gb.x), __uint_as_float(gb.y), __uint_as_float(gb.z), __uint_as_float(gb.w)};
    const float uv[4] = {__uint_as_float(ub.x), __uint_as_float(ub.y), __uint_as_float(ub.z), __uint_as_float(ub.w)};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = gv[i] / (1.0f + __expf(-gv[i])) * uv[i] * sv[i];
    hadamard128(v, lane);
    *reinterpret_cast<float4 *>(rot + k0) = make_float4(v[0], v[1], v[2], v[3]);
    m = fmaxf(m, fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if (lane == 0) warp_max[warp] = m;
  __syncthreads();
  m = warp_max[0];
#pragma unroll
  for (uint32_t i = 1; i < kRotateThreads / 32u; ++i) m = fmaxf(m, warp_max[i]);
  // m in [2^(e-1), 2^e) with e = (exponent field) - 126: the scale 2^(14 - e), held to what a float carries
  int shift = 0;
  if (m > 0.0f && m <= 3.0e38f) shift = max(-126, min(126, 140 - static_cast<int>(__float_as_uint(m) >> 23)));
  const float scale = __uint_as_float(static_cast<uint32_t>(shift + 127) << 23);
  if (threadIdx.x == 0) *inv = __uint_as_float(static_cast<uint32_t>(127 - shift) << 23);
  for (uint32_t i = threadIdx.x * 4u; i < in; i += 4u * kRotateThreads) {
    const float4 v = *reinterpret_cast<const float4 *>(rot + i);
    const __half2 h01 = __floats2half2_rn(v.x * scale, v.y * scale), h23 = __floats2half2_rn(v.z * scale, v.w * scale);
    uint2 packed;
    packed.x = *reinterpret_cast<const uint32_t *>(&h01);
    packed.y = *reinterpret_cast<const uint32_t *>(&h23);
    *reinterpret_cast<uint2 *>(dst + i) = packed;
  }
}

// PHASE 0: gate | up products of an item into gu. PHASE 1: down, weighted, into the rows the fold
// kernel adds up. One CTA per (item, 128 output columns); no CTA waits for another.
constexpr uint32_t kBoxRows = 32;   // rows of one TMA load: an item loads as many as it has rows for

template <int PHASE>
__global__ void __launch_bounds__(Shape<2>::kThreads, 2) moe_tc_gemm_kernel(const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ ExpertParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t in = PHASE == 0 ? p.hidden : p.inter;
  const uint32_t out_plane = PHASE == 0 ? 2u * p.inter : p.hidden;
  const uint32_t col_tiles = out_plane / 128u;
  const uint32_t item_index = blockIdx.x / col_tiles, col_tile = blockIdx.x % col_tiles;
  griddep_launch_dependents();
  griddep_wait();   // the item list and the rotated rows come from the kernels before
  if (item_index >= p.n_items[0]) return;
  const Item item = p.items[item_index];
  const ignis_moe_slot slot = p.slots[item.expert * 2u + PHASE];
  if (slot.record == nullptr || !(slot.k2 == 4 || slot.k2 == 5 || slot.k2 == 6 || slot.k2 == 8)) {
    if (threadIdx.x == 0 && col_tile == 0) atomicOr(p.status, kStatusAbsentRecord);
    return;
  }
  Job job;
  job.trellis = static_cast<const uint32_t *>(slot.record);
  job.k2 = slot.k2;
  job.tile_stride = out_plane / 16u;
  job.stage0 = 0u;
  job.stage1 = in / 64u;
  job.blk = col_tile;
  job.row0 = item.first;
  job.rows = item.count;
  job.box = kBoxRows;
  const Core c = core_setup<2>(smem_raw, job, kWhole);
  const uint64_t trellis_bytes = static_cast<uint64_t>(in) * out_plane * slot.k2 / 16u;
  const uint16_t *svh = reinterpret_cast<const uint16_t *>(static_cast<const uint8_t *>(slot.record) + trellis_bytes) + in;
  const float *inv_rows = PHASE == 0 ? p.x_scale : p.h_scale;
  const bool decoded = core_roles<2>(c, job, &map_rows, p.status + 1);   // word 1 of the status line: waits of this kernel that ran out
  struct Row {
    float *y;
    float weight;   // PHASE 1: the routing weight
  };
  core_finish_rows<2>(
      c, job, kWhole, decoded, p.status + 1, [&](uint32_t r) { return inv_rows[item.first + r]; },
      [&](uint32_t r) {
        const uint32_t row = item.first + r;
        if (PHASE == 0) return Row{p.gu + static_cast<size_t>(row) * 2u * p.inter + col_tile * 128u, 1.0f};
        const uint32_t a = p.sorted[row];   // which assignment (token, rank) the row is
        return Row{p.down_rows + static_cast<size_t>(a) * p.hidden + col_tile * 128u, p.weights[a]};
      },
      [](const Row &, uint32_t) { return 0u; },
      [&](const Row &row, uint32_t col, uint32_t, const float4 &v) {
        const float4 sv = four_halves(__ldg(reinterpret_cast<const uint2 *>(svh + col_tile * 128u + col)));
        float4 o = make_float4(v.x * sv.x, v.y * sv.y, v.z * sv.z, v.w * sv.w);
        if (PHASE == 1) o = make_float4(row.weight * o.x, row.weight * o.y, row.weight * o.z, row.weight * o.w);
        *reinterpret_cast<float4 *>(row.y + col) = o;
      });
}

// One CTA per token, several with few tokens: the token's weighted down products (one row per choice that had an expert with a
// record) become 2^-32 fixed-point integers and are added to the token's accumulator row. Integer
// sums do not depend on their order: the bits are those of adding every product on its own. SHARED: by atomic additions, so that
// calls on several streams may add into one accumulator; wide calls read and write the row, whose calls must be ordered.
template <bool SHARED>
__global__ void __launch_bounds__(256) moe_tc_fold_kernel(const __grid_constant__ ExpertParams p, uint32_t tokens) {
  griddep_launch_dependents();
  griddep_wait();
  const uint32_t token = blockIdx.x;
  if (token >= tokens) return;
  __shared__ uint32_t present[64];
  const uint32_t top_k = p.top_k < 64u ? p.top_k : 64u;
  if (threadIdx.x < top_k) {
    const int32_t e = p.ids[static_cast<size_t>(token) * p.top_k + threadIdx.x];
    bool ok = e >= 0 && static_cast<uint32_t>(e) < p.experts;
    if (ok) {
      const ignis_moe_slot slot = p.slots[static_cast<uint32_t>(e) * 2u + 1u];
      ok = slot.record != nullptr && (slot.k2 == 4 || slot.k2 == 5 || slot.k2 == 6 || slot.k2 == 8);
    }
    present[threadIdx.x] = ok ? 1u : 0u;
  }
  __syncthreads();
  bool range = false;
  // four columns per thread and trip (hidden is a multiple of 128), the choices' loads issued together
  const float4 *rows4 = reinterpret_cast<const float4 *>(p.down_rows + static_cast<size_t>(token) * p.top_k * p.hidden);
  const uint32_t quads = p.hidden / 4u;
  for (uint32_t c4 = blockIdx.y * 256u + threadIdx.x; c4 < quads; c4 += gridDim.y * 256u) {
    long long sum[4] = {0, 0, 0, 0};
    for (uint32_t k0 = 0; k0 < top_k; k0 += 8u) {
      float4 v[8];
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) {
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k0 + j < top_k && present[k0 + j] != 0u) v[j] = __ldcs(rows4 + static_cast<size_t>(k0 + j) * quads + c4);
      }
#pragma unroll
      for (uint32_t j = 0; j < 8u; ++j) {
        const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (!(fabsf(e[i]) < 2147483648.0f)) {   // also catches NaN
            range = true;
          } else {
            // times 2^32 is exact in a float (the magnitude is below 2^31): the integer a double product would round to
            sum[i] += __float2ll_rn(e[i] * 4294967296.0f);
          }
        }
      }
    }
    long long *dst = p.acc + static_cast<size_t>(token) * p.hidden + 4u * c4;   // the caller's buffer: 8-byte alignment is all it promises
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (SHARED) atomicAdd(reinterpret_cast<unsigned long long *>(dst + i), static_cast<unsigned long long>(sum[i]));
      else dst[i] += sum[i];
    }
  }
  if (range) atomicOr(p.status, kStatusRange);
}

constexpr uint32_t kRotateMaxIn = 51200;   // inputs of a row the route takes

}  // namespace

int32_t moe_tc_prepare(ErrorSlot &slot) {
  cudaError_t err = cudaFuncSetAttribute(moe_tc_gemm_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<2>::kSmemBytes));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(moe_tc_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<2>::kSmemBytes));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(moe_tc_rotate_h_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRotateMaxIn * 4u));
  if (err != cudaSuccess) return fail(slot, "MoE tensor-core kernel attributes: %s", cudaGetErrorString(err));
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
  return 0;
}

int32_t moe_tc_experts(ErrorSlot &slot, const DeviceState &dev, const ExpertParams &p, uint32_t rows, uint32_t items_max,
                       const uint32_t *offsets, cudaStream_t stream, const char *what) {
  const bool pdl = dev.pdl != 0;
  const uint32_t tokens = rows / p.top_k;
  if (p.top_k > 64u) return fail(slot, "%s: more than 64 choices per token on the tensor-core route", what);
  for (int phase = 0; phase < 2; ++phase) {
    const uint32_t in = phase == 0 ? p.hidden : p.inter;
    const uint32_t out_plane = phase == 0 ? 2u * p.inter : p.hidden;
    if (in > kRotateMaxIn) return fail(slot, "%s: a dimension is too long for the tensor-core route", what);
    const uint32_t threads = 32u * rotate_warps(in), at_once = static_cast<uint32_t>(dev.sm_count) * (threads <= 256u ? 1024u / threads : 1u);
    cudaError_t err = phase != 0 ? launch(moe_tc_rotate_h_kernel, dim3(rows), dim3(kRotateThreads), static_cast<size_t>(in) * 4u, stream, pdl, p, offsets)
                                 : launch(threads <= 256u ? moe_tc_rotate_x_kernel<256> : moe_tc_rotate_x_kernel<1024>, dim3(rows < at_once ? rows : at_once),
                                          dim3(threads), 0, stream, pdl, p, offsets);
    if (err != cudaSuccess) return fail(slot, "%s: rotation launch failed: %s", what, cudaGetErrorString(err));
    CUtensorMap map_rows;
    if (!make_rows_map(&map_rows, phase == 0 ? p.x_rows : p.h_rows, rows, in, kBoxRows)) {
      return fail(slot, "%s: tensor map encoding failed", what);
    }
    const dim3 grid(items_max * (out_plane / 128u));
    err = phase == 0 ? launch(moe_tc_gemm_kernel<0>, grid, dim3(Shape<2>::kThreads), Shape<2>::kSmemBytes, stream, pdl, map_rows, p)
                     : launch(moe_tc_gemm_kernel<1>, grid, dim3(Shape<2>::kThreads), Shape<2>::kSmemBytes, stream, pdl, map_rows, p);
    if (err != cudaSuccess) return fail(slot, "%s: expert launch failed: %s", what, cudaGetErrorString(err));
  }
  const cudaError_t err = launch(tokens <= kMoeNarrowTokens ? moe_tc_fold_kernel<true> : moe_tc_fold_kernel<false>, dim3(tokens, tokens < static_cast<uint32_t>(dev.sm_count) ? (p.hidden + 1023u) / 1024u : 1u), dim3(256), 0, stream, pdl, p, tokens);
  if (err != cudaSuccess) return fail(slot, "%s: fold launch failed: %s", what, cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q
