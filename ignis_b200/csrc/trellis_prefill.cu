// Dense trellis linear beyond 64 tokens: the prefill route on the tensor cores.
//
// Stands where the reference switches from its decode kernel to its prefill kernel
// (kernel/src/trellis_linear.cu: rotate_kernel + prefill_kernel, trellis_linear_prefill.cu:162-279;
// the route needs the workspace, as theirs does). Two launches: `trellis_rotate_rows_kernel` writes
// the rotated activations as fp16 rows with one scale per token into the workspace, and
// `trellis_tc_dense_kernel` multiplies them with the trellis plane on tcgen05 (trellis_tc.cuh).
// SwiGLU runs the gate product first (BF16 into h, as the reference's prefill route stores the gate
// between its passes: ignis_trellis_linear.h:43-44) and the up product with an epilogue that
// multiplies by silu of what it finds there.
#include "../../include/ignis_trellis_linear.h"

#include "trellis_internal.cuh"
#include "trellis_tc.cuh"

namespace b200q {
namespace {

using namespace trellis_tc;

__device__ uint32_t g_trellis_tc_status = 0;

// ---- rotation: one CTA per token ------------------------------------------------------------------
// x o suh, the 128-wide Hadamard per block (a warp per block, fp32), one power-of-two scale for the
// whole token (largest magnitude in [2^13, 2^14)), fp16. The token's rotated values wait in shared
// memory between the two passes (4 bytes per input).
__global__ void __launch_bounds__(256) trellis_rotate_rows_kernel(const uint16_t *x, const uint16_t *suh, uint32_t in,
                                                                  uint16_t *rows_f16, float *inv) {
  extern __shared__ __align__(16) float rot[];
  __shared__ float warp_max[8];
  griddep_launch_dependents();
  griddep_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t token = blockIdx.x;
  const uint32_t nblk = in / 128u;
  float m = 0.0f;
  for (uint32_t bl = static_cast<uint32_t>(warp); bl < nblk; bl += 8u) {
    const size_t k0 = static_cast<size_t>(bl) * 128u + 4u * lane;
    const uint2 xb = ldg64_coherent(x + static_cast<size_t>(token) * in + k0);
    const uint2 sb = *reinterpret_cast<const uint2 *>(suh + k0);
    const __half2 s01 = *reinterpret_cast<const __half2 *>(&sb.x), s23 = *reinterpret_cast<const __half2 *>(&sb.y);
    float v[4];
    v[0] = bf16_bits_to_f32(xb.x & 0xFFFFu) * __low2float(s01);
    v[1] = __uint_as_float(xb.x & 0xFFFF0000u) * __high2float(s01);
    v[2] = bf16_bits_to_f32(xb.y & 0xFFFFu) * __low2float(s23);
    v[3] = __uint_as_float(xb.y & 0xFFFF0000u) * __high2float(s23);
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
  for (int i = 1; i < 8; ++i) m = fmaxf(m, warp_max[i]);
  // m in [2^(e-1), 2^e) with e = (exponent field) - 126: the scale 2^(14 - e), held to what a float carries
  int shift = 0;
  if (m > 0.0f && m <= 3.0e38f) shift = max(-126, min(126, 140 - static_cast<int>(__float_as_uint(m) >> 23)));
  const float scale = __uint_as_float(static_cast<uint32_t>(shift + 127) << 23);
  if (threadIdx.x == 0) inv[token] = __uint_as_float(static_cast<uint32_t>(127 - shift) << 23);
  uint16_t *dst = rows_f16 + static_cast<size_t>(token) * in;
  for (uint32_t i = threadIdx.x * 4u; i < in; i += 1024u) {
    const float4 v = *reinterpret_cast<const float4 *>(rot + i);
    const __half2 h01 = __floats2half2_rn(v.x * scale, v.y * scale), h23 = __floats2half2_rn(v.z * scale, v.w * scale);
    uint2 packed;
    packed.x = *reinterpret_cast<const uint32_t *>(&h01);
    packed.y = *reinterpret_cast<const uint32_t *>(&h23);
    *reinterpret_cast<uint2 *>(dst + i) = packed;
  }
}

// ---- the product -----------------------------------------------------------------------------------
constexpr uint32_t kEpiStore = 0, kEpiAdd = 1, kEpiSiluMul = 2;   // kEpiSiluMul: y = BF16(silu(float(y)) * v)

struct DenseParams {
  const uint32_t *trellis;
  const uint16_t *svh;
  const float *inv;      // the tokens' inverse scales
  uint16_t *y;           // BF16 [tokens][ldy]
  uint32_t k2, tile_stride, in, out, tokens, ldy, epilogue;
  uint32_t tile;         // tokens per CTA
  uint32_t ranks;        // the CTAs of a cluster share an item's K stages (1: no cluster)
};

__global__ void __launch_bounds__(kThreads, 2) trellis_tc_dense_kernel(const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ DenseParams p) {
  extern __shared__ uint8_t smem_raw[];
  // Token tiles run fastest over the grid, so the CTAs at work at one time decode the same columns
  // of the plane (read from HBM once, then from the L2).
  const uint32_t row_tiles = (p.tokens + p.tile - 1u) / p.tile;
  const Split split = {p.ranks, p.ranks == 1u ? 0u : cluster_ctarank()};
  const uint32_t item = blockIdx.x / p.ranks;
  Job job;
  job.trellis = p.trellis;
  job.k2 = p.k2;
  job.tile_stride = p.tile_stride;
  const uint32_t stages = p.in / 64u;
  job.stage0 = stages * split.rank / p.ranks;
  job.stage1 = stages * (split.rank + 1u) / p.ranks;
  job.blk = item / row_tiles;
  job.row0 = item % row_tiles * p.tile;
  job.rows = min(p.tokens - job.row0, p.tile);
  job.box = p.tile;
  const Core c = core_setup(smem_raw, job, split);
  const bool decoded = core_roles(c, job, &map_rows, &g_trellis_tc_status);
  const uint32_t col = job.blk * 128u + 4u * static_cast<uint32_t>(c.lane);
  const float4 sv = four_halves(p.svh + col);
  uint16_t *out = p.y + static_cast<size_t>(job.row0) * p.ldy + col;
  core_finish_rows(
      c, job, split, decoded, &g_trellis_tc_status, [&](uint32_t r) { return p.inv[job.row0 + r]; },
      [&](uint32_t r) { return p.epilogue != kEpiStore ? *reinterpret_cast<const uint2 *>(out + static_cast<size_t>(r) * p.ldy) : make_uint2(0u, 0u); },
      [&](uint32_t r, const uint2 &old, const float4 &o) {
        float v[4] = {o.x * sv.x, o.y * sv.y, o.z * sv.z, o.w * sv.w};
        if (p.epilogue != kEpiStore) {
          const float was[4] = {bf16_bits_to_f32(old.x & 0xFFFFu), __uint_as_float(old.x & 0xFFFF0000u), bf16_bits_to_f32(old.y & 0xFFFFu),
                                __uint_as_float(old.y & 0xFFFF0000u)};
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = p.epilogue == kEpiAdd ? v[e] + was[e] : was[e] / (1.0f + __expf(-was[e])) * v[e];
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
        *reinterpret_cast<uint2 *>(out + static_cast<size_t>(r) * p.ldy) =
            make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
      });
}

uint64_t align256(uint64_t v) { return (v + 255u) & ~static_cast<uint64_t>(255u); }

constexpr size_t kRotateMaxSmem = 200 * 1024;   // 4 bytes per input: in <= 51200

bool aligned_to(const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

}  // namespace

uint64_t trellis_tc_workspace_bytes(uint32_t in, uint32_t weights, uint32_t tokens) {
  // a status line, then per weight the rotated rows (fp16) and the tokens' inverse scales
  return 256u + static_cast<uint64_t>(weights) * (align256(static_cast<uint64_t>(tokens) * in * 2u) + align256(static_cast<uint64_t>(tokens) * 4u));
}

namespace {
// The CTAs of a cluster that share the K stages of an item.
constexpr uint32_t kMaxRanks = 8;

cudaLaunchConfig_t dense_config(uint32_t items, uint32_t ranks, cudaStream_t stream, bool pdl, cudaLaunchAttribute (&attr)[2]) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(items * ranks);
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kSmemBytes;
  config.stream = stream;
  unsigned n = 0;
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (ranks > 1u) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = ranks;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  config.attrs = attr;
  config.numAttrs = n;
  return config;
}

// How many CTAs share an item: the count for which a model of the launch gives the least time. In microseconds, from
// measurements of four shapes at 70 to 2000 tokens: a stage takes 1.17 with two CTAs on the SM, 0.72 alone (0.95 in a cluster,
// whose CTAs may share an SM all the same); the epilogue 3 per row tile of 128 and 0.9 more per rank (its reads from the other
// CTAs' shared memory). The last wave is counted for what is left in it. Few items leave SMs idle and walk all of K alone
// (17408 -> 5120 at 128 tokens: 40 items of 272 stages, 190 us; six ranks each: 63), a last wave that is nearly empty costs as
// much as a full one (the same at 1000 tokens: 160 items, 306 us; three ranks: 250); many items need no sharing. At least eight
// stages per rank: what a CTA spends before its first and after its last stage is as long.
uint32_t dense_ranks(const DeviceState &dev, uint32_t items, uint32_t stages, uint32_t row_tiles128) {
  uint32_t best = 1u;
  float least = 0.0f;
  for (uint32_t ranks = 1; ranks <= kMaxRanks && (ranks == 1u || stages / ranks >= 8u); ++ranks) {
    const uint32_t at_once = ranks == 1u ? 2u * static_cast<uint32_t>(dev.sm_count) : static_cast<uint32_t>(dev.trellis_clusters[ranks]);
    if (at_once == 0u) continue;
    const uint32_t waves = items / at_once, left = items % at_once;
    const float epilogue = static_cast<float>(row_tiles128) * (3.0f + 0.9f * static_cast<float>(ranks));
    const float walked = static_cast<float>((stages + ranks - 1u) / ranks);
    const bool alone = left * ranks <= static_cast<uint32_t>(dev.sm_count);
    float t = static_cast<float>(waves) * (1.17f * walked + epilogue);
    if (left != 0u) t += (!alone ? 1.17f : ranks == 1u ? 0.72f : 0.95f) * walked + epilogue;
    if (ranks == 1u || t < least) least = t, best = ranks;
  }
  return best;
}
}  // namespace

int32_t trellis_tc_prepare(ErrorSlot &slot) {
  DeviceState *dev = device_state(slot);
  if (dev == nullptr) return -1;
  cudaError_t err = cudaFuncSetAttribute(trellis_tc_dense_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemBytes));
  if (err == cudaSuccess) {
    err = cudaFuncSetAttribute(trellis_rotate_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRotateMaxSmem));
  }
  if (err != cudaSuccess) return fail(slot, "trellis prefill kernel attributes: %s", cudaGetErrorString(err));
  for (uint32_t ranks = 2; ranks <= kMaxRanks && !dev->counted; ++ranks) {
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t config = dense_config(1u, ranks, nullptr, false, attr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, trellis_tc_dense_kernel, &config) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    dev->trellis_clusters[ranks] = clusters;
  }
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
  return 0;
}

bool trellis_tc_takes(const DeviceState &dev, uint32_t in, uint32_t tokens, uint32_t weights, const ignis_trellis_workspace *workspace) {
  if (dev.trellis_tc == 0 || tokens <= IGNIS_TRELLIS_DECODE_MAX_TOKENS) return false;
  if (static_cast<size_t>(in) * 4u > kRotateMaxSmem) return false;
  if (workspace == nullptr || workspace->base == nullptr || !aligned_to(workspace->base, 256)) return false;
  return workspace->bytes >= trellis_tc_workspace_bytes(in, weights, tokens);
}

namespace {
int32_t one_product(ErrorSlot &slot, const DeviceState &dev, const ignis_trellis_weight *w, const uint16_t *x, uint32_t tokens, uint16_t *y,
                    uint32_t ldy, uint32_t epilogue, uint8_t *region, cudaStream_t stream, const char *what) {
  uint16_t *rows = reinterpret_cast<uint16_t *>(region);
  float *inv = reinterpret_cast<float *>(region + align256(static_cast<uint64_t>(tokens) * w->in * 2u));
  cudaError_t err = launch(trellis_rotate_rows_kernel, dim3(tokens), dim3(256), static_cast<size_t>(w->in) * 4u, stream, dev.pdl != 0, x,
                           static_cast<const uint16_t *>(w->suh), w->in, rows, inv);
  if (err != cudaSuccess) return fail(slot, "%s: rotation launch failed: %s", what, cudaGetErrorString(err));
  const uint32_t row_tiles = (tokens + kMaxRows - 1u) / kMaxRows;
  CUtensorMap map_rows;
  const uint32_t tile = ((tokens + row_tiles - 1u) / row_tiles + 15u) / 16u * 16u;
  if (!make_rows_map(&map_rows, rows, tokens, w->in, tile)) return fail(slot, "%s: tensor map encoding failed", what);
  DenseParams p = {};
  p.trellis = static_cast<const uint32_t *>(w->trellis);
  p.svh = static_cast<const uint16_t *>(w->svh);
  p.inv = inv;
  p.y = y;
  p.k2 = w->k2;
  p.tile_stride = w->tile_stride ? w->tile_stride : w->out / 16u;
  p.in = w->in;
  p.out = w->out;
  p.tokens = tokens;
  p.ldy = ldy;
  p.epilogue = epilogue;
  p.tile = tile;
  const uint32_t items = w->out / 128u * ((tokens + p.tile - 1u) / p.tile);
  p.ranks = dense_ranks(dev, items, w->in / 64u, p.tile > 128u ? 2u : 1u);
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t config = dense_config(items, p.ranks, stream, dev.pdl != 0, attr);
  err = cudaLaunchKernelEx(&config, trellis_tc_dense_kernel, map_rows, p);
  if (err != cudaSuccess) return fail(slot, "%s: launch failed: %s", what, cudaGetErrorString(err));
  return 0;
}
}  // namespace

int32_t trellis_tc_linear(ErrorSlot &slot, const DeviceState &dev, const ignis_trellis_weight *w, const ignis_trellis_weight *up,
                          const void *x, uint32_t tokens, void *y, uint32_t ldy, uint32_t epilogue,
                          const ignis_trellis_workspace *workspace, cudaStream_t stream, const char *what) {
  uint8_t *base = static_cast<uint8_t *>(workspace->base) + 256;
  const uint16_t *xs = static_cast<const uint16_t *>(x);
  uint16_t *ys = static_cast<uint16_t *>(y);
  if (up == nullptr) return one_product(slot, dev, w, xs, tokens, ys, ldy, epilogue == 1u ? kEpiAdd : kEpiStore, base, stream, what);
  // SwiGLU: the gate product into h, then the up product times silu of what it finds there
  if (one_product(slot, dev, w, xs, tokens, ys, ldy, kEpiStore, base, stream, what) != 0) return -1;
  uint8_t *second = base + align256(static_cast<uint64_t>(tokens) * w->in * 2u) + align256(static_cast<uint64_t>(tokens) * 4u);
  return one_product(slot, dev, up, xs, tokens, ys, ldy, kEpiSiluMul, second, stream, what);
}

int32_t trellis_tc_status(ErrorSlot &slot, cudaStream_t stream, uint32_t *status) {
  cudaError_t err = cudaMemcpyFromSymbolAsync(status, g_trellis_tc_status, sizeof(uint32_t), 0, cudaMemcpyDeviceToHost, stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
  if (err != cudaSuccess) return fail(slot, "b200q_trellis_device_status: %s", cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q
