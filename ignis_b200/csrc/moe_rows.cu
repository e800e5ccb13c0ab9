// The dense products of an MoE block that are narrow in rows: the router's logits (BF16 weight
// [experts][hidden], fp32 out), the router's selection, and the shared expert's FP8 row-scale
// products (kernel/include/ignis_fp8_linear.h:4-10) of calls the tcgen05 kernels do not take.
//
// One kernel serves all three products, `moe_rows_kernel<KIND, NT>`. A CTA owns 16 output rows and up
// to 64 tokens; its eight warps split K, so that a weight of a few hundred rows still spreads over
// the device (512 experts: 32 CTAs, 256 warps), and their partial sums meet in shared memory in
// warp order. The products run on mma.sync m16n8k16 (BF16 x BF16, fp32 accumulation): inside a chunk
// of 64 columns the MMA's k slots are dealt so that a lane needs 16 contiguous weights of its two
// rows and 16 contiguous activations of its token, all loaded straight from global memory in
// 16-byte pieces - at these widths a weight is read once and nothing is gained by staging it.
// E4M3 codes widen exactly to BF16. The first weights are requested before the wait for the
// previous kernel. Bound by latency: the router's 2 MB at 8 tokens take 3.6 us (one CTA per token
// walking all experts took 98), the shared expert's 4.7 MB 7.8 us (a warp per row: 40).
//
// `moe_router_tile_kernel` is the router's product for many tokens: 128 experts x 128 tokens a CTA,
// operands staged by cp.async, each of the eight K slices summed from zero and added in slice order, so
// a token's logits carry the same bits whichever kernel ran (a token's result must not depend on
// how many tokens share the call). 4096 tokens x 512 experts x 2048: 40 us (the kernel before: 807).
#include "moe_internal.cuh"

namespace b200q {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kRowTile = 16;
enum Kind { kRouter = 0, kGateUp = 1, kDown = 2 };

struct RowsParams {
  const void *w0, *w1;  // kRouter: BF16 [rows][cols]; kGateUp: FP8 gate, up; kDown: FP8 down
  const uint16_t *x;    // BF16 [tokens][cols]
  void *y;              // [tokens][rows]: fp32, or BF16 (kGateUp)
  uint32_t rows, cols, tokens;
  uint32_t x16;         // x is 16-byte aligned (8 is all the shared expert's h promises)
};

// Two E4M3 codes (the low 16 bits of `pair`) as BF16 x 2, exactly: the fp16 bits moved down three
// places are a BF16 with an exponent 112 too small, which one BF16 multiply restores.
__device__ __forceinline__ uint32_t e4m3x2_to_bf16x2(uint32_t pair) {
  const uint32_t h = e4m3x2_to_half2(pair);
  const uint32_t tiny = ((h & 0x7FFF7FFFu) >> 3) | (h & 0x80008000u);
  const __nv_bfloat162 up = __floats2bfloat162_rn(5.192296858534828e33f, 5.192296858534828e33f);   // 2^112
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&tiny), up);
  return *reinterpret_cast<const uint32_t *>(&v);
}

// A lane's weights of one chunk of 64 columns: 16 of row g and 16 of row g + 8.
template <int KIND>
struct Chunk {
  static constexpr int S = KIND == kGateUp ? 2 : 1;
  static constexpr int Q = KIND == kRouter ? 2 : 1;   // 16-byte pieces of 16 weights
  uint4 v[S][2][Q];
};

template <int KIND>
__device__ __forceinline__ void load_chunk(Chunk<KIND> &c, const uint8_t *const (&rows)[2][2], uint32_t chunk, int t, bool lo, bool hi) {
#pragma unroll
  for (int s = 0; s < Chunk<KIND>::S; ++s)
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
      for (int q = 0; q < Chunk<KIND>::Q; ++q) {
        const uint32_t at = KIND == kRouter ? chunk * 128u + 32u * t + 16u * q : chunk * 64u + 16u * t;
        c.v[s][half][q] = (half == 0 ? lo : hi) ? __ldg(reinterpret_cast<const uint4 *>(rows[s][half] + at)) : make_uint4(0u, 0u, 0u, 0u);
      }
}

// The A fragments of MMA j of the chunk: k slots 2t, 2t + 1 are the lane's weights 4 j, 4 j + 1, slots
// 2t + 8, 2t + 9 its 4 j + 2, 4 j + 3.
template <int KIND>
__device__ __forceinline__ void chunk_frag(const Chunk<KIND> &c, int s, int j, uint32_t (&a)[4]) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    if (KIND == kRouter) {
      const uint4 q = c.v[s][half][Chunk<KIND>::Q == 2 ? (j >> 1) : 0];
      a[half] = (j & 1) ? q.z : q.x;
      a[2 + half] = (j & 1) ? q.w : q.y;
    } else {
      const uint4 q = c.v[s][half][0];
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      a[half] = e4m3x2_to_bf16x2(w[j] & 0xFFFFu);
      a[2 + half] = e4m3x2_to_bf16x2(w[j] >> 16);
    }
  }
}

// A lane's 16 activations of one token (columns 16 t .. of a chunk).
__device__ __forceinline__ void load_activations(uint4 (&xb)[2], const uint16_t *src, bool x16) {
  if (x16) {
    xb[0] = ldg128_coherent(src);
    xb[1] = ldg128_coherent(src + 8);
  } else {
    const uint2 v0 = ldg64_coherent(src), v1 = ldg64_coherent(src + 4), v2 = ldg64_coherent(src + 8), v3 = ldg64_coherent(src + 12);
    xb[0] = make_uint4(v0.x, v0.y, v1.x, v1.y);
    xb[1] = make_uint4(v2.x, v2.y, v3.x, v3.y);
  }
}

constexpr int kAhead = 4;   // chunks of weights a warp requests before it waits for the previous kernel

template <int KIND, int NT>
__global__ void __launch_bounds__(kThreads) moe_rows_kernel(const __grid_constant__ RowsParams p) {
  constexpr int S = Chunk<KIND>::S;
  extern __shared__ __align__(16) float red[];   // [warp][weight][token tile][lane][4]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t row0 = blockIdx.x * kRowTile, tok0 = blockIdx.y * (8u * NT);
  const uint32_t chunks = p.cols / 64u;
  const uint32_t c0 = chunks * static_cast<uint32_t>(warp) / kWarps, c1 = chunks * (static_cast<uint32_t>(warp) + 1u) / kWarps;
  const bool lo = row0 + g < p.rows, hi = row0 + g + 8u < p.rows;
  const size_t row_bytes = static_cast<size_t>(p.cols) * (KIND == kRouter ? 2u : 1u);
  const uint8_t *rows[2][2];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      rows[s][half] = static_cast<const uint8_t *>(s == 0 ? p.w0 : p.w1) + (row0 + g + 8u * half) * row_bytes;
    }
  Chunk<KIND> ring[kAhead];
#pragma unroll
  for (int d = 0; d < kAhead; ++d) {
    if (c0 + d < c1) load_chunk<KIND>(ring[d], rows, c0 + d, t, lo, hi);
  }
  griddep_launch_dependents();
  griddep_wait();   // the activations may come from the previous kernel

  float acc[S][NT][4];
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[s][nt][e] = 0.0f;
  for (uint32_t base = c0; base < c1; base += kAhead) {
#pragma unroll
    for (int d = 0; d < kAhead; ++d) {
      if (base + d >= c1) break;
      uint4 xb[NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint32_t token = tok0 + nt * 8u + g;
        xb[nt][0] = xb[nt][1] = make_uint4(0u, 0u, 0u, 0u);
        if (token < p.tokens) load_activations(xb[nt], p.x + static_cast<size_t>(token) * p.cols + (base + d) * 64u + 16u * t, p.x16 != 0u);
      }
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t a[4];
          chunk_frag<KIND>(ring[d], s, j, a);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const uint4 q = xb[nt][j >> 1];
            mma_bf16_f32(acc[s][nt], a[0], a[1], a[2], a[3], (j & 1) ? q.z : q.x, (j & 1) ? q.w : q.y);
          }
        }
      if (base + d + kAhead < c1) load_chunk<KIND>(ring[d], rows, base + d + kAhead, t, lo, hi);
    }
  }
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      reinterpret_cast<float4 *>(red)[((warp * S + s) * NT + nt) * 32 + lane] = make_float4(acc[s][nt][0], acc[s][nt][1], acc[s][nt][2], acc[s][nt][3]);
    }
  __syncthreads();
  const uint64_t scale_off = (static_cast<uint64_t>(p.rows) * p.cols + 255u) & ~static_cast<uint64_t>(255u);   // behind the FP8 codes
  for (uint32_t o = threadIdx.x; o < kRowTile * 8u * NT; o += kThreads) {   // 16 consecutive rows of a token side by side
    const uint32_t r = o % kRowTile, tl = o / kRowTile;
    const uint32_t row = row0 + r, token = tok0 + tl;
    if (row >= p.rows || token >= p.tokens) continue;
    const uint32_t at = ((tl >> 3) * 32u + (r & 7u) * 4u + ((tl & 7u) >> 1)) * 4u + (tl & 1u) + 2u * (r >> 3);
    float v[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      v[s] = red[s * NT * 128 + at];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) v[s] += red[(w * S + s) * NT * 128 + at];
    }
    const size_t out = static_cast<size_t>(token) * p.rows + row;
    if (KIND == kRouter) {
      static_cast<float *>(p.y)[out] = v[0];
    } else {
      const float s0 = bf16_bits_to_f32(reinterpret_cast<const uint16_t *>(static_cast<const uint8_t *>(p.w0) + scale_off)[row]);
      if (KIND == kDown) {
        static_cast<float *>(p.y)[out] = v[0] * s0;
      } else {
        const float s1 = bf16_bits_to_f32(reinterpret_cast<const uint16_t *>(static_cast<const uint8_t *>(p.w1) + scale_off)[row]);
        const float gv = v[0] * s0, uv = v[S - 1] * s1;
        static_cast<__nv_bfloat16 *>(p.y)[out] = __float2bfloat16_rn(gv / (1.0f + __expf(-gv)) * uv);
      }
    }
  }
}

template <int KIND, int NT>
cudaError_t rows_launch_nt(const RowsParams &p, cudaStream_t stream, bool pdl) {
  const size_t smem = static_cast<size_t>(kWarps) * Chunk<KIND>::S * NT * 512u;
  return launch(moe_rows_kernel<KIND, NT>, dim3((p.rows + kRowTile - 1u) / kRowTile, (p.tokens + 8u * NT - 1u) / (8u * NT)), dim3(kThreads), smem,
                stream, pdl, p);
}

// Token tiles per CTA: the fewest that hold the call, up to 64 tokens (then side by side in the grid).
template <int KIND>
cudaError_t rows_launch(const RowsParams &p, cudaStream_t stream, bool pdl) {
  if (p.tokens <= 8u) return rows_launch_nt<KIND, 1>(p, stream, pdl);
  if (p.tokens <= 16u) return rows_launch_nt<KIND, 2>(p, stream, pdl);
  if (p.tokens <= 32u) return rows_launch_nt<KIND, 4>(p, stream, pdl);
  return rows_launch_nt<KIND, 8>(p, stream, pdl);
}

// ---- the router's logits for many tokens ------------------------------------------------------------
constexpr int kTile = 128;            // experts and tokens per CTA
constexpr int kTileStages = 4;
constexpr uint32_t kTileBytes = kTile * 128u;   // one operand of a stage: 128 rows x 64 BF16
constexpr size_t kTileSmem = static_cast<size_t>(kTileStages) * 2u * kTileBytes;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16u : 0u) : "memory");
}

// A slice's sums are added to the running total and start again from zero.
__device__ __forceinline__ void close_slice(float (&total)[4][4][4], float (&acc)[4][4][4], bool first) {
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        total[m][n][e] = first ? acc[m][n][e] : total[m][n][e] + acc[m][n][e];
        acc[m][n][e] = 0.0f;
      }
}

// Warp (wm, wn) of 2 x 4 owns 64 experts x 32 tokens. A stage is a chunk of 64 columns; a row's eight
// 16-byte pieces are exchanged by the row's low bits, so that the fragment reads (8 lanes: two rows,
// pieces 0, 2, 4, 6 or 1, 3, 5, 7) touch all bank groups once.
__global__ void __launch_bounds__(kThreads, 1) moe_router_tile_kernel(const __grid_constant__ RowsParams p) {
  extern __shared__ __align__(16) uint8_t tile_smem[];
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(tile_smem));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t e0 = blockIdx.x * kTile, tok0 = blockIdx.y * kTile;
  const uint32_t wm = static_cast<uint32_t>(warp) & 1u, wn = static_cast<uint32_t>(warp) >> 1;
  const uint32_t chunks = p.cols / 64u;
  griddep_launch_dependents();
  griddep_wait();
  auto request = [&](uint32_t chunk) {
    if (chunk < chunks) {
      const uint32_t stage = base + (chunk % kTileStages) * 2u * kTileBytes;
#pragma unroll
      for (int i = 0; i < 8; ++i) {   // 1024 pieces of each operand over 256 threads
        const uint32_t piece = threadIdx.x + 256u * (i & 3), r = piece >> 3, q = piece & 7u;
        const bool a = i < 4;
        const uint32_t row = (a ? e0 : tok0) + r, limit = a ? p.rows : p.tokens;
        const uint16_t *src = (a ? static_cast<const uint16_t *>(p.w0) : p.x) + static_cast<size_t>(row < limit ? row : 0u) * p.cols + chunk * 64u + q * 8u;
        cp_async16(stage + (a ? 0u : kTileBytes) + r * 128u + ((q ^ (r & 7u)) << 4), src, row < limit);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[4][4][4], total[4][4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = total[m][n][e] = 0.0f;
  for (int s = 0; s < kTileStages - 1; ++s) request(s);
  uint32_t slice = 0;   // the K slice (a warp's of moe_rows_kernel) that the chunk belongs to
  for (uint32_t c = 0; c < chunks; ++c) {
    for (; c >= chunks * (slice + 1u) / kWarps; ++slice) close_slice(total, acc, slice == 0u);
    asm volatile("cp.async.wait_group %0;" ::"n"(kTileStages - 2) : "memory");
    __syncthreads();
    request(c + kTileStages - 1);
    const uint8_t *sa = tile_smem + (c % kTileStages) * 2u * kTileBytes, *sb = sa + kTileBytes;
    uint4 b[4][2];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const uint32_t r = wn * 32u + n * 8u + g;
#pragma unroll
      for (int q = 0; q < 2; ++q) b[n][q] = *reinterpret_cast<const uint4 *>(sb + r * 128u + (((2u * t + q) ^ (r & 7u)) << 4));
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      uint4 a[2][2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint32_t r = wm * 64u + m * 16u + half * 8u + g;
#pragma unroll
        for (int q = 0; q < 2; ++q) a[half][q] = *reinterpret_cast<const uint4 *>(sa + r * 128u + (((2u * t + q) ^ (r & 7u)) << 4));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 a_lo = a[0][j >> 1], a_hi = a[1][j >> 1];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const uint4 q = b[n][j >> 1];
          if (j & 1) mma_bf16_f32(acc[m][n], a_lo.z, a_hi.z, a_lo.w, a_hi.w, q.z, q.w);
          else mma_bf16_f32(acc[m][n], a_lo.x, a_hi.x, a_lo.y, a_hi.y, q.x, q.y);
        }
      }
    }
  }
  for (; slice < kWarps; ++slice) close_slice(total, acc, slice == 0u);   // the last slice, and the empty ones of a short K
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t row = e0 + wm * 64u + m * 16u + g + 8u * (e >> 1), token = tok0 + wn * 32u + n * 8u + 2u * t + (e & 1u);
        if (row < p.rows && token < p.tokens) static_cast<float *>(p.y)[static_cast<size_t>(token) * p.rows + row] = total[m][n][e];
      }
}

// ---- the router's selection ----------------------------------------------------------------------------
// One warp per token: the top_k largest BF16-rounded logits, ties to the lower id, then the softmax over
// the selected ones in fp32, rounded to BF16 and stored as fp32. A lane keeps its experts as 32-bit keys
// (the value's order-preserving bits above the complement of the id), so a round is an integer
// maximum over the lane's keys and one warp reduction; the keys are read once. A NaN is never selected.
template <int PER>
__global__ void __launch_bounds__(kThreads) moe_router_select_kernel(const float *logits, uint32_t tokens, uint32_t experts,
                                                                     uint32_t top_k, int32_t *ids, float *weights) {
  griddep_launch_dependents();
  griddep_wait();
  const uint32_t t = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31u;
  if (t >= tokens) return;
  const float *row = logits + static_cast<size_t>(t) * experts;
  uint32_t key[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint32_t e = lane + 32u * i;
    key[i] = 0u;
    if (e < experts) {
      const float v = row[e];
      uint32_t bits = __bfloat16_as_ushort(__float2bfloat16_rn(v));
      if (bits == 0x8000u) bits = 0u;   // both zeros are one value
      bits = (bits & 0x8000u) ? (~bits & 0xFFFFu) : (bits | 0x8000u);
      if (v == v) key[i] = (bits << 16) | (0xFFFFu - e);
    }
  }
  float mine = -INFINITY;   // lane r keeps the value of choice r
  int32_t mine_id = 0x7FFFFFFF;
  uint32_t best = 0xFFFFFFFFu;
  for (uint32_t r = 0; r < top_k; ++r) {
    uint32_t m = 0u;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (key[i] == best) key[i] = 0u;   // the previous round's choice (ids make keys unique)
      m = max(m, key[i]);
    }
    best = __reduce_max_sync(0xFFFFFFFFu, m);
    if (lane == r && best != 0u) {
      const uint32_t bits = best >> 16;
      mine = bf16_bits_to_f32((bits & 0x8000u) ? (bits & 0x7FFFu) : (~bits & 0xFFFFu));
      mine_id = static_cast<int32_t>(0xFFFFu - (best & 0xFFFFu));
    }
    if (best == 0u) best = 0xFFFFFFFFu;   // nothing is left to choose
  }
  const float mx = __shfl_sync(0xFFFFFFFFu, mine, 0);
  const float ex = expf(mine - mx);
  float sum = 0.0f;
  for (uint32_t r = 0; r < top_k; ++r) sum += __shfl_sync(0xFFFFFFFFu, ex, static_cast<int>(r));
  if (lane < top_k) {
    ids[static_cast<size_t>(t) * top_k + lane] = mine_id;
    weights[static_cast<size_t>(t) * top_k + lane] = __bfloat162float(__float2bfloat16_rn(ex / sum));
  }
}

}  // namespace

int32_t moe_rows_prepare(ErrorSlot &slot) {
  cudaError_t err = cudaFuncSetAttribute(moe_router_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTileSmem));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(moe_rows_kernel<kGateUp, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWarps * 2 * 8 * 512);
  if (err != cudaSuccess) return fail(slot, "MoE row kernels: %s", cudaGetErrorString(err));
  return 0;
}

constexpr uint32_t kRouterRowCtas = 768;

cudaError_t moe_router_logits_launch(const DeviceState &dev, const uint16_t *x, const uint16_t *w, uint32_t tokens, uint32_t hidden,
                                     uint32_t experts, float *logits, cudaStream_t stream) {
  const RowsParams p = {w, nullptr, x, logits, experts, hidden, tokens, 1u};
  // The tile form re-reads its operands least, but has only experts / 128 x tokens / 128 CTAs, each a walk down all of
  // `hidden`: its time hardly depends on the call until they fill the device. The row form has 16 times as many, and its time
  // grows with them. The line lies where they meet at 512 experts: five waves of the row form's CTAs, 1536 tokens there.
  // Logits and selection from a cold L2, rows against tiles in us: 512 experts x 2048 at 1536 / 1537 tokens 60 / 52, 256 x 7168 at
  // 2048 99 / 130, 128 x 2048 at 4096 42 / 48, 8 x 4096 at 2048 24 / 77.
  const uint32_t row_ctas = (experts + kRowTile - 1u) / kRowTile * ((tokens + 63u) / 64u);
  if (row_ctas > kRouterRowCtas) {
    return launch(moe_router_tile_kernel, dim3((experts + kTile - 1) / kTile, (tokens + kTile - 1) / kTile), dim3(kThreads), kTileSmem, stream,
                  dev.pdl != 0, p);
  }
  return rows_launch<kRouter>(p, stream, dev.pdl != 0);
}

cudaError_t moe_router_select_launch(const DeviceState &dev, const float *logits, uint32_t tokens, uint32_t experts, uint32_t top_k,
                                     int32_t *ids, float *weights, cudaStream_t stream) {
  const dim3 grid((tokens + kWarps - 1) / kWarps), block(kThreads);
  const bool pdl = dev.pdl != 0;
  if (experts <= 256u) return launch(moe_router_select_kernel<8>, grid, block, 0, stream, pdl, logits, tokens, experts, top_k, ids, weights);
  if (experts <= 512u) return launch(moe_router_select_kernel<16>, grid, block, 0, stream, pdl, logits, tokens, experts, top_k, ids, weights);
  if (experts <= 1024u) return launch(moe_router_select_kernel<32>, grid, block, 0, stream, pdl, logits, tokens, experts, top_k, ids, weights);
  return launch(moe_router_select_kernel<128>, grid, block, 0, stream, pdl, logits, tokens, experts, top_k, ids, weights);
}

cudaError_t moe_rows_shared_expert(const DeviceState &dev, const uint8_t *gate, const uint8_t *up, const uint8_t *down, const uint16_t *x,
                                   uint32_t tokens, uint32_t hidden, uint32_t inter, void *h, float *shared, cudaStream_t stream) {
  const RowsParams p = {gate, up, x, h, inter, hidden, tokens, 1u};
  cudaError_t err = rows_launch<kGateUp>(p, stream, dev.pdl != 0);
  if (err == cudaSuccess) {
    const RowsParams d = {down, nullptr, static_cast<const uint16_t *>(h), shared, hidden, inter, tokens,
                          (reinterpret_cast<uintptr_t>(h) & 15u) == 0u ? 1u : 0u};
    err = rows_launch<kDown>(d, stream, dev.pdl != 0);
  }
  return err;
}

}  // namespace b200q
