// NVFP4 prefill route (W4A4): out[t][r] = bf16(alpha * sum_k E2M1(a) E4M3(sa) E2M1(w) E4M3(sw)),
// alpha = 1 / (d_in d_w), on the 5th-generation tensor cores.
//
// Stands where the reference quantizes activations and runs its FP4 GEMMs
// (kernel/vendor/src/ops/linear/nvfp4/nvfp4_w4a4_mma.cuh:203-436, nvfp4_w4a4_tma.cuh:264-508,
// launch_problem nvfp4_w4a4.cu:74-110) - warp-level mma.sync on its RTX target. Here:
//
//  1. `quantize_swizzled_kernel` turns the BF16 activations into E2M1 codes [T_pad][K/2] and E4M3
//     scales, bit for bit the reference's rule (nvfp4_codec.cuh:81-110), the scales written in the
//     same 512-byte (128 rows x 4 groups) tiles the weight plane uses - which is the scale-factor
//     atom the block-scaled MMA reads, so neither operand's scales are ever reshuffled.
//  2. `w4a4_gemm_pair_kernel` - clusters of two CTAs, one CTA per SM, walk 256-token x 256-row tiles
//     (tcgen05 cta_group::2): a producer warp streams K in stages of 256 (TMA 2-D tiles of codes with the
//     128-byte swizzle, scale tiles beside them) into an mbarrier ring that keeps running across tile
//     boundaries; two warps copy each stage's scale atoms to tensor memory (tcgen05.cp); one issues
//     tcgen05.mma kind::mxf4nvf4 block_scale scale_vec::4X (M 256, N 256, K 64) with the fp32
//     accumulator in tensor memory; four warps pull the accumulator (tcgen05.ld), hand tensor
//     memory back and store under the next tile's MMAs. Calls whose tiles would leave most of the
//     device idle take the narrow kernel instead (nvfp4_w4a4_narrow.cu).
//
// Every wait on an mbarrier is bounded: after the limit the thread records a status bit in the
// workspace, stops issuing and the CTA tears down (tensor memory freed) instead of hanging.
#include "../../include/b200q_nvfp4.h"

#include "nvfp4_internal.cuh"
#include "nvfp4_tc.cuh"
#include "w4a4_pair_control.h"

#include <cmath>
#include <mutex>

namespace b200q {
namespace {

constexpr int kBM = 128;          // tokens per tile (MMA M)
constexpr int kBKBytes = 128;     // bytes of codes per row per stage: 256 values along K
constexpr uint32_t kABytes = kBM * kBKBytes;        // 16 KB
constexpr uint32_t kSfaBytes = 4 * 512;             // 4 K-atoms of one 128-row tile

constexpr uint32_t kStatusProducerTimeout = 1u, kStatusMmaTimeout = 2u, kStatusEpilogueTimeout = 4u;

// ---- activation quantizer, scales in tile order -------------------------------------------------
// One thread per (token row of the padded range, 32 values): two blocks of 16, i.e. 64 bytes in,
// 16 bytes of codes and two of the four scale bytes that lie side by side in a scale tile out. The
// kernel is bound by instruction issue as much as by memory (about 13 instructions per value), so a
// thread is kept small: 48 registers, five CTAs an SM, their load and arithmetic phases interleaved
// (four blocks a thread at 65 registers and three CTAs: 2.6 % slower on a step of 8192 tokens, 5120 -> 17408 -> 5120).
// Rows at and beyond `tokens` get zero codes and zero scales.
__global__ void __launch_bounds__(256, 5) quantize_swizzled_kernel(const uint16_t *x, uint32_t tokens, uint32_t tokens_pad,
                                                                   uint32_t k, float d_in, uint8_t *codes, uint8_t *scales) {
  griddep_launch_dependents();
  griddep_wait();
  const uint32_t halves = k / 32u, quads = k / 64u;
  const uint64_t total = static_cast<uint64_t>(tokens_pad) * halves;
  for (uint64_t hi = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; hi < total;
       hi += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t t = static_cast<uint32_t>(hi / halves), h = static_cast<uint32_t>(hi % halves);
    uint2 c[2];
    uint32_t sw = 0;
    if (t < tokens) {
      const uint16_t *src = x + static_cast<uint64_t>(t) * k + h * 32u;
      uint4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = ldg128_coherent(src + 8 * j);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        uint8_t s;
        quantize_block16(v[2 * b], v[2 * b + 1], d_in, c[b], s);
        sw |= static_cast<uint32_t>(s) << (8 * b);
      }
    } else {
#pragma unroll
      for (int b = 0; b < 2; ++b) c[b] = make_uint2(0u, 0u);
    }
    *reinterpret_cast<uint4 *>(codes + hi * 16u) = make_uint4(c[0].x, c[0].y, c[1].x, c[1].y);
    const uint32_t q = h >> 1;
    const uint64_t so = (static_cast<uint64_t>(t >> 7) * quads + q) * 512u + (t & 31u) * 16u + ((t & 127u) >> 5) * 4u + (h & 1u) * 2u;
    *reinterpret_cast<uint16_t *>(scales + so) = static_cast<uint16_t>(sw);
  }
}

// One weight of a launch (row ranges of one parent share the activations), with its first 256-row tile in the grid's walk.
struct W4A4Weight {
  void *y;
  uint32_t n, ldy;
  float alpha;
  uint32_t tile_begin;
};
struct W4A4Params {
  W4A4Weight w[kMaxGroup];
  uint32_t count, n_tiles;   // n_tiles: 256-row tiles of all weights
  uint32_t *status;
  uint32_t tokens, k;
  uint32_t epilogue;  // STORE / ADD / OUT_F32, or the fused SwiGLU (the tile's columns 0..127 are gate rows, 128..255 the up rows)
  uint8_t *q_codes;   // kEpilogueQuant: h as the next product's operand, codes [pad tokens][n / 4] ...
  uint8_t *q_scales;  // ... and scales in 512-byte tiles
  float q_din;        // the next weight's input divisor
};
struct W4A4Maps {
  CUtensorMap b[kMaxGroup], sfb[kMaxGroup];   // the weights' codes and scales
};

// The weight that 256-row tile `n_tile` of the launch belongs to.
__device__ __forceinline__ uint32_t weight_of(const W4A4Params &p, uint32_t n_tile) {
  uint32_t wi = 0;
  for (uint32_t i = 1; i < p.count; ++i) {
    if (n_tile >= p.w[i].tile_begin) wi = i;
  }
  return wi;
}

// The epilogue pulls the whole accumulator into registers (as packed BF16: 128 registers a thread - the
// CTA has the SM's register file to itself), hands tensor memory back to the MMA warp and only
// then stores, under the next tile's MMAs. What a tile costs beyond its MMAs is the pull alone.
// ---- the epilogue of one CTA's 128-token x 256-row half of a tile --------------------------------
// The calling warp q owns accumulator lanes (tokens) 32 q .. 32 q + 31 at `lane_base`. `release()`
// hands tensor memory back to the MMA thread; it is called as soon as the accumulator has been
// read, so that whatever follows runs under the next tile's MMAs.
template <class Release>
__device__ __forceinline__ void w4a4_epilogue_tile(const W4A4Params &p, const W4A4Weight &w, uint32_t lane_base, int warp, int lane, uint32_t m_tile,
                                                   uint32_t n_tile, bool swiglu, Release release) {
  constexpr int kBN = 256;
  const float alpha = w.alpha;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t token = m_tile * kBM + warp * 32 + lane;
  if (p.epilogue & (kEpilogueF32 | kEpilogueAdd)) {
    // float32 rows do not fit the register file, and a residual has to be read before the one
    // rounding: these forms store chunk by chunk, then release
#pragma unroll 1
    for (uint32_t c = 0; c < kBN; c += 32) {
      uint32_t r[32];
      tmem_ld32(lane_base + c, r);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const uint32_t row0 = n_tile * kBN + c;
      if (token < p.tokens && row0 < w.n) {
        const bool add = (p.epilogue & kEpilogueAdd) != 0u;
        if (p.epilogue & kEpilogueF32) {
          float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(w.y) + static_cast<size_t>(token) * w.ldy + row0);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 o = make_float4(__uint_as_float(r[4 * j]) * alpha, __uint_as_float(r[4 * j + 1]) * alpha,
                                   __uint_as_float(r[4 * j + 2]) * alpha, __uint_as_float(r[4 * j + 3]) * alpha);
            if (add) {
              const float4 old = dst[j];
              o.x += old.x, o.y += old.y, o.z += old.z, o.w += old.w;
            }
            dst[j] = o;
          }
        } else {
          uint4 *dst = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(w.y) + static_cast<size_t>(token) * w.ldy + row0);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 old = dst[j];
            const uint32_t ow[4] = {old.x, old.y, old.z, old.w};
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(
                  __uint_as_float(r[8 * j + 2 * e]) * alpha + bf16_bits_to_f32(ow[e] & 0xFFFFu),
                  __uint_as_float(r[8 * j + 2 * e + 1]) * alpha + __uint_as_float(ow[e] & 0xFFFF0000u));
              o[e] = *reinterpret_cast<const uint32_t *>(&h);
            }
            dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    release();
    return;
  }
  // The thread's row as packed BF16: 256 columns of the product, or (SwiGLU) BF16(g alpha) in
  // [0, 64) and BF16(u alpha) in [64, 128) - the two roundings the reference's formula makes first.
  uint32_t out[128];
#pragma unroll
  for (uint32_t c = 0; c < kBN; c += 32) {
    uint32_t r[32];
    tmem_ld32(lane_base + c, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[2 * j]) * alpha, __uint_as_float(r[2 * j + 1]) * alpha);
      out[c / 2 + j] = *reinterpret_cast<const uint32_t *>(&h);
    }
  }
  // tensor memory is free for the next tile's MMAs; the rest runs under them
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  release();
  // Rows past the call's tokens: nothing of them is read (as operand rows of the next product they only reach output rows
  // that are not stored), and their zeros would take the divisions' slow paths (242 -> 175 us a layer at 300 tokens).
  if (token >= p.tokens) return;
  if (swiglu) {
    // h = BF16(silu(BF16(g)) * BF16(u)), in place over the gate half
#pragma unroll
    for (int j = 0; j < 64; ++j) {
      const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&out[j]));
      const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&out[64 + j]));
      const __nv_bfloat162 h = __floats2bfloat162_rn(g.x / (1.0f + __expf(-g.x)) * u.x, g.y / (1.0f + __expf(-g.y)) * u.y);
      out[j] = *reinterpret_cast<const uint32_t *>(&h);
    }
  }
  if (swiglu && (p.epilogue & kEpilogueQuant)) {
    // h leaves as the down product's operand: 8 blocks of 16 along its K, quantized as the
    // standalone quantizer would from the BF16 values
    const uint32_t inter = w.n / 2u, g0 = n_tile * 8u;
    uint32_t sc[2] = {0u, 0u};
    uint4 *code_dst = reinterpret_cast<uint4 *>(p.q_codes + static_cast<uint64_t>(token) * (inter / 2u) + n_tile * 64u);
#pragma unroll
    for (int b = 0; b < 8; b += 2) {
      uint2 c0, c1;
      uint8_t s0, s1;
      quantize_block16(make_uint4(out[8 * b], out[8 * b + 1], out[8 * b + 2], out[8 * b + 3]),
                       make_uint4(out[8 * b + 4], out[8 * b + 5], out[8 * b + 6], out[8 * b + 7]), p.q_din, c0, s0);
      quantize_block16(make_uint4(out[8 * b + 8], out[8 * b + 9], out[8 * b + 10], out[8 * b + 11]),
                       make_uint4(out[8 * b + 12], out[8 * b + 13], out[8 * b + 14], out[8 * b + 15]), p.q_din, c1, s1);
      code_dst[b / 2] = make_uint4(c0.x, c0.y, c1.x, c1.y);
      sc[b >> 2] |= (static_cast<uint32_t>(s0) << (8 * (b & 3))) | (static_cast<uint32_t>(s1) << (8 * ((b + 1) & 3)));
    }
    const uint64_t atom = (static_cast<uint64_t>(token >> 7) * (inter / 64u) + (g0 >> 2)) * 512u + (token & 31u) * 16u +
                          ((token & 127u) >> 5) * 4u;
    *reinterpret_cast<uint32_t *>(p.q_scales + atom) = sc[0];
    *reinterpret_cast<uint32_t *>(p.q_scales + atom + 512u) = sc[1];
    return;
  }
  const uint32_t width = swiglu ? 128u : kBN;
  const uint32_t col0 = n_tile * width;
  const uint32_t limit = swiglu ? w.n / 2u : w.n;
  __nv_bfloat16 *row = static_cast<__nv_bfloat16 *>(w.y) + static_cast<size_t>(token) * w.ldy + col0;
#pragma unroll
  for (uint32_t c = 0; c < kBN; c += 8) {
    if (c < width && col0 + c < limit) {  // n is a multiple of 128: an 8-column piece is whole
      *reinterpret_cast<uint4 *>(row + c) = make_uint4(out[c / 2], out[c / 2 + 1], out[c / 2 + 2], out[c / 2 + 3]);
    }
  }
}

// ---- the product on CTA pairs --------------------------------------------------------------------
// Two CTAs of a cluster share a 256-token x 256-row tile (tcgen05 cta_group::2): each CTA holds its
// 128 tokens' codes and accumulator rows, and only half of the weight rows - the tensor cores read
// the other half from the peer's shared memory - so a CTA brings 38 KB per K stage. The token tile index
// runs fastest, so the pairs at work share weight rows in the L2. Every load
// of both CTAs reports to the barrier of the pair's first CTA, whose MMA warp issues for both;
// its commits arrive at both CTAs' barriers (two plain commits, one per CTA). The scale tiles
// travel as TMA tiles too (a bulk copy cannot report to the peer's barrier): the scale planes as
// [tile][128] words.
constexpr uint32_t kPairBBytes = 128 * kBKBytes;                                   // this CTA's half of the weight rows
constexpr uint32_t kPairStageBytes = kABytes + kPairBBytes + kSfaBytes + 2 * 2048;  // + token scales + both halves' weight scales
constexpr uint32_t kPairSmemBytes = kPairStages * kPairStageBytes + kPairControlBytes + 1024;
constexpr uint32_t kPairSfCols = 48;  // per stage: 16 columns of token scales, 32 of weight scales
// The shared::cluster address of this CTA's `addr` in the cluster's CTA `rank`.
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  return remote;
}

__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_cp_sf_pair(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
__device__ __forceinline__ void mma_mxf4nvf4_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                                  uint32_t accumulate) {
  asm volatile("{ .reg .pred p; setp.ne.u32 p, %6, 0;\n"
               "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p; }"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
               : "memory");
}
// Arrives at `bar` (a shared::cluster address: this CTA's or the peer's) once the pair's MMAs so far have retired.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__global__ void __launch_bounds__(256, 1) w4a4_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a,
                                                               const __grid_constant__ CUtensorMap map_sfa,
                                                               const __grid_constant__ W4A4Maps maps,
                                                               const __grid_constant__ W4A4Params p) {
  constexpr int kBN = 256;
  constexpr int kStages = kPairStages;
  constexpr uint32_t kTmemCols = 512;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;   // the same offset in both CTAs: they run the same kernel
  uint8_t *base_ptr = smem_raw + (base - raw);
  const uint32_t control = base + kStages * kPairStageBytes;   // barriers and the tensor-memory slot (PairControl)
  const uint32_t bars = control + kPairFull, bars_empty = control + kPairEmpty;
  const uint32_t bar_acc_full = control + kPairAccFull, bar_acc_empty = control + kPairAccEmpty, bar_sf_ready = control + kPairSfReady;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base_ptr + kStages * kPairStageBytes + kPairTmemSlot);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // 0: the pair's first CTA, which issues the MMAs
  const uint32_t k_iters = p.k / 256u, k_atoms = p.k / 64u;
  const bool swiglu = (p.epilogue & kEpilogueSwiglu) != 0u;
  const uint32_t m_tiles = (p.tokens + kBM - 1) / kBM, m_pairs = (m_tiles + 1u) / 2u;
  const uint32_t tiles = m_pairs * p.n_tiles;
  const uint32_t first = blockIdx.x / 2u, step = gridDim.x / 2u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bars + 8 * s, 1);               // the first CTA's: its producer's expect_tx arrival (the bytes of both CTAs)
      mbar_init(bars_empty + 8 * s, 1);         // one commit
    }
    mbar_init(bar_acc_full, 1);
    mbar_init(bar_acc_empty, 8);                // the first CTA's: one arrival per epilogue warp of the pair
    for (int s = 0; s < kStages; ++s) mbar_init(bar_sf_ready + 8 * s, 2);   // the two scale copiers' commits
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist before anything is sent to them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);

  griddep_launch_dependents();
  griddep_wait();  // the quantized activations come from the previous kernel in the stream

  // The issuing roles run in whole warps with an elected lane (elect_one, nvfp4_tc.cuh).
  if (warp == 4) {
    // ---- producer (both CTAs): own tokens, own half of the weight rows, the scales of both halves ----
    RingAt at;
    const uint32_t full0 = in_cta(bars, 0u);   // the first CTA's barriers collect both CTAs' bytes
    bool ok = true;
    for (uint32_t tile = first; tile < tiles && ok; tile += step) {
      const uint32_t m_tile = 2u * (tile % m_pairs) + rank, wi = weight_of(p, tile / m_pairs), n_tile = tile / m_pairs - p.w[wi].tile_begin;
      const CUtensorMap *map_b = &maps.b[wi], *map_sfb = &maps.sfb[wi];
      const uint32_t row_a = swiglu ? n_tile * 128u : n_tile * kBN;
      const uint32_t row_b = swiglu ? p.w[wi].n / 2u + n_tile * 128u : n_tile * kBN + 128u;
      const int32_t row = static_cast<int32_t>(rank == 0u ? row_a : row_b);
      const uint32_t sfa0 = m_tile * k_atoms, sfb0 = row_a / 128u * k_atoms, sfb1 = row_b / 128u * k_atoms;
      for (uint32_t it = 0; it < k_iters; ++it, at.advance(1u, kStages)) {
        if (!mbar_wait(bars_empty + 8 * at.slot, at.phase ^ 1u)) {
          if (lane == 0) atomicOr(p.status, kStatusProducerTimeout);
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t full = full0 + 8 * at.slot, stage = base + at.slot * kPairStageBytes;
          if (rank == 0u) mbar_expect_tx(bars + 8 * at.slot, 2u * kPairStageBytes);
          tma_load_2d_pair(stage, &map_a, full, static_cast<int32_t>(it * kBKBytes), static_cast<int32_t>(m_tile * kBM));
          tma_load_2d_pair(stage + kABytes, map_b, full, static_cast<int32_t>(it * kBKBytes), row);
          tma_load_2d_pair(stage + kABytes + kPairBBytes, &map_sfa, full, 0, static_cast<int32_t>(sfa0 + it * 4u));
          tma_load_2d_pair(stage + kABytes + kPairBBytes + kSfaBytes, map_sfb, full, 0, static_cast<int32_t>(sfb0 + it * 4u));
          tma_load_2d_pair(stage + kABytes + kPairBBytes + kSfaBytes + 2048u, map_sfb, full, 0, static_cast<int32_t>(sfb1 + it * 4u));
        }
        __syncwarp();
      }
    }
  } else if (warp == 5) {
    // ---- MMA issuer of the pair: M 256 (128 per CTA), N 256, K 64 ----
    if (rank == 0u) {
      const uint32_t idesc = (1u << 7) | (1u << 10) | ((kBN >> 3) << 17) | ((256u >> 4) << 24);
      const uint32_t own_empty = in_cta(bars_empty, 0u), peer_empty = in_cta(bars_empty, 1u);
      const uint32_t own_acc = in_cta(bar_acc_full, 0u), peer_acc = in_cta(bar_acc_full, 1u);
      const uint64_t desc0 = smem_desc(base, 1024u, 2u);
      RingAt at;
      uint32_t tile_i = 0;
      bool ok = true;
      for (uint32_t tile = first; tile < tiles && ok; tile += step, ++tile_i) {
        if (!mbar_wait(bar_acc_empty, (tile_i & 1u) ^ 1u)) {   // both CTAs have pulled the previous tile out of tensor memory
          if (lane == 0) atomicOr(p.status, kStatusMmaTimeout);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (uint32_t it = 0; it < k_iters; ++it, at.advance(1u, kStages)) {
          if (!mbar_wait(bar_sf_ready + 8 * at.slot, at.phase)) {   // operands landed in both CTAs and scales copied
            if (lane == 0) atomicOr(p.status, kStatusMmaTimeout);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (elect_one()) {
            const uint32_t sf_cols = tmem + kBN + at.slot * kPairSfCols;
            const uint64_t a_desc = desc0 + at.slot * (kPairStageBytes >> 4), b_desc = a_desc + (kABytes >> 4);
#pragma unroll
            for (uint32_t kb = 0; kb < 4; ++kb) {
              mma_mxf4nvf4_pair(tmem, a_desc + 2u * kb, b_desc + 2u * kb, idesc, sf_cols + kb * 4u, sf_cols + 16u + kb * 8u,
                                (it | kb) != 0u ? 1u : 0u);
            }
            mma_commit_pair(own_empty + 8 * at.slot);    // this CTA's stage ...
            mma_commit_pair(peer_empty + 8 * at.slot);   // ... and the peer's
          }
          __syncwarp();
        }
        if (ok && elect_one()) {
          mma_commit_pair(own_acc);
          mma_commit_pair(peer_acc);
        }
        __syncwarp();
      }
    }
  } else if (warp >= 6) {
    // ---- scale copiers of the pair (one copy instruction serves both CTAs): warp 6 the first two
    //      K-atoms of a stage, warp 7 the other two ----
    if (rank == 0u) {
      const uint32_t kb0 = static_cast<uint32_t>(warp - 6) * 2u;
      const uint32_t my_tiles = tiles > first ? (tiles - first + step - 1u) / step : 0u;
      const uint32_t total = my_tiles * k_iters, ready = in_cta(bar_sf_ready, 0u);
      const uint64_t sfa0 = smem_desc(base + kABytes + kPairBBytes, 128u, 0u);
      RingAt at;
      for (uint32_t g = 0; g < total; ++g, at.advance(1u, kStages)) {
        if (!mbar_wait(bars + 8 * at.slot, at.phase)) {
          if (lane == 0) atomicOr(p.status, kStatusMmaTimeout);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint32_t sf_cols = tmem + kBN + at.slot * kPairSfCols + kb0 * 4u;
          const uint64_t sfa = sfa0 + at.slot * (kPairStageBytes >> 4) + kb0 * 32u, sfb = sfa + (kSfaBytes >> 4);
#pragma unroll
          for (uint32_t kb = 0; kb < 2u; ++kb) {
            tmem_cp_sf_pair(sf_cols + kb * 4u, sfa + kb * 32u);
            tmem_cp_sf_pair(sf_cols + 16u + kb0 * 4u + kb * 8u, sfb + kb * 32u);
            tmem_cp_sf_pair(sf_cols + 20u + kb0 * 4u + kb * 8u, sfb + 128u + kb * 32u);
          }
          mma_commit_pair(ready + 8 * at.slot);
        }
        __syncwarp();
      }
    }
  } else if (warp < 4) {
    // ---- epilogue (both CTAs): warp q owns this CTA's accumulator lanes (tokens) 32 q .. 32 q + 31 ----
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const uint32_t acc_empty_first = in_cta(bar_acc_empty, 0u);
    uint32_t tile_i = 0;
    for (uint32_t tile = first; tile < tiles; tile += step, ++tile_i) {
      const uint32_t m_tile = 2u * (tile % m_pairs) + rank, wi = weight_of(p, tile / m_pairs), n_tile = tile / m_pairs - p.w[wi].tile_begin;
      if (!mbar_wait(bar_acc_full, tile_i & 1u)) {
        if (lane == 0) atomicOr(p.status, kStatusEpilogueTimeout);
        break;
      }
      if (m_tile >= m_tiles) {   // the odd pair's second CTA: nothing of this tile is its to store
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_first);
        continue;
      }
      w4a4_epilogue_tile(p, p.w[wi], lane_base, warp, lane, m_tile, n_tile, swiglu, [&] {
        if (lane == 0) mbar_arrive_cluster(acc_empty_first);
      });
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves while the other may still reach its shared memory or barriers
  if (warp == 5) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---- host side --------------------------------------------------------------------------------
// A scale plane of 512-byte tiles as a 2-D tensor [tiles][128 words] with boxes of four tiles (one K stage).
bool make_scale_map(CUtensorMap *map, const void *scales, uint64_t tiles) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {128, tiles};
  const cuuint64_t strides[1] = {512};
  const cuuint32_t box[2] = {128, 4};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(scales), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

uint32_t w4a4_tokens_pad(uint32_t tokens) { return (tokens + kBM - 1) / kBM * kBM; }

// Workspace of a W4A4 call: one status line, then the codes, then the scale tiles.
uint64_t w4a4_workspace_bytes(uint32_t k, uint32_t tokens) {
  const uint64_t pad = w4a4_tokens_pad(tokens);
  return 256u + pad * (k / 2u) + pad * (k / 16u);
}

bool w4a4_shape_ok(uint32_t n, uint32_t k) { return (k % 256u) == 0 && (n % 128u) == 0; }

int32_t w4a4_prepare(ErrorSlot &slot) {
  const cudaError_t err = cudaFuncSetAttribute(w4a4_gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPairSmemBytes));
  if (err != cudaSuccess) return fail(slot, "nvfp4 prefill kernel attributes: %s", cudaGetErrorString(err));
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
  return w4a4_narrow_prepare(slot);
}

namespace {
struct QuantTarget {
  uint8_t *codes = nullptr;
  uint8_t *scales = nullptr;
  float d_in = 1.0f;
};

// Which kernel a product takes: the cheaper by a model of each, in SM cycles, fitted to products whose weights come from HBM.
// The pair kernel: waves of 256 x 256 tiles on half as many pairs as SMs, 820 cycles a stage of 256 and 3000 a tile (a gate|up
// parent, whose epilogue multiplies, rounds and quantizes: 8600, and 47 500 a launch, a fit whose cause has not been taken
// apart), never faster than the weights come from HBM; `w4a4_narrow_cycles` beside its kernel. The narrow kernel has to be ahead by 15 %: where the models are that
// close, products on different kernels in a row cost more (200 tokens: gate|up on the pair kernel and down on the narrow one
// 89 us, both on the narrow one 71, both on the pair kernel 85).
// Both forced, an MLP with its residual, in us, narrow / pair, the rule's choice last:
//   tokens   5120 x 17408          4096 x 14336          2048 x 6144
//     128    44.8 /  84.6 n        38.5 /  76.0 n        26.4 / 39.7 n
//     200    70.9 /  84.8 n        61.2 /  77.4 n        28.2 / 39.5 n
//     384    93.6 / 113.0 n        84.5 / 104.4 n        39.4 / 53.3 n
//     640   158.6 / 144.8 p       124.6 / 120.9 p        48.9 / 53.8 n
//    1024   244.3 / 197.8 p       182.9 / 142.7 p        65.3 / 68.3 n
bool narrow_is_cheaper(const DeviceState &dev, const A4Item *items, uint32_t count, uint32_t k, uint32_t tokens, bool swiglu) {
  if (dev.w4a4_pair >= 0) return dev.w4a4_pair == 0;
  uint32_t row_tiles = 0, n_tiles = 0;
  for (uint32_t i = 0; i < count; ++i) {
    row_tiles += items[i].n / (swiglu ? 256u : 128u);
    n_tiles += (items[i].n + 255u) / 256u;
  }
  const double tiles = static_cast<double>(n_tiles) * ((tokens + 255u) / 256u);
  const double walk = ceil(tiles / (dev.sm_count / 2)) * ((k / 256u) * 820.0 + (swiglu ? 8600.0 : 3000.0)) + (swiglu ? 47500.0 : 0.0);
  const double stream = row_tiles * (swiglu ? 144.0 : 72.0) * k / 3150.0;
  return w4a4_narrow_cycles(dev, row_tiles, k, tokens, swiglu) * 1.15 < 8500.0 + (walk > stream ? walk : stream);
}

int32_t quantize_rows(ErrorSlot &slot, const DeviceState &dev, const uint16_t *x, uint32_t tokens, uint32_t k, float d_in, uint8_t *codes,
                      uint8_t *scales, cudaStream_t stream) {
  const uint32_t pad = w4a4_tokens_pad(tokens);
  const uint64_t total = static_cast<uint64_t>(pad) * (k / 32u);
  const uint32_t grid = static_cast<uint32_t>(total / 256u < 148u * 24u ? (total + 255u) / 256u : 148u * 24u);
  const cudaError_t err = launch(quantize_swizzled_kernel, dim3(grid), dim3(256), 0, stream, dev.pdl != 0, x, tokens, pad, k, d_in, codes, scales);
  if (err != cudaSuccess) return fail(slot, "nvfp4 activation quantizer launch: %s", cudaGetErrorString(err));
  return 0;
}

// The products of `count` weights that share k over the operand at `a_codes` / `a_scales`, in one launch; `x` non-NULL
// is quantized there first.
int32_t w4a4_products(ErrorSlot &slot, const DeviceState &dev, const A4Item *items, uint32_t count, uint32_t k, const uint16_t *x,
                      uint32_t tokens, uint32_t epilogue, uint32_t *status, uint8_t *a_codes, uint8_t *a_scales, const QuantTarget &q,
                      cudaStream_t stream) {
  const uint32_t pad = w4a4_tokens_pad(tokens);
  if (x != nullptr && quantize_rows(slot, dev, x, tokens, k, items[0].d_in, a_codes, a_scales, stream) != 0) return -1;
  const bool swiglu = (epilogue & kEpilogueSwiglu) != 0u;
  if (narrow_is_cheaper(dev, items, count, k, tokens, swiglu)) {
    return w4a4_narrow_launch(slot, dev, items, count, k, tokens, epilogue, a_codes, a_scales, status, q.codes, q.scales, q.d_in, stream);
  }
  W4A4Params p = {};
  W4A4Maps maps = {};
  CUtensorMap map_a, map_sfa;
  bool encoded = make_code_map(&map_a, a_codes, pad, k / 2u, kBM) &&
                 make_scale_map(&map_sfa, a_scales, static_cast<uint64_t>(pad / kBM) * (k / 64u));
  p.count = count;
  for (uint32_t i = 0; i < count; ++i) {
    const A4Item &it = items[i];
    p.w[i] = W4A4Weight{it.y, it.n, it.ldy, 1.0f / (it.d_in * it.d_w), p.n_tiles};
    p.n_tiles += (it.n + 255u) / 256u;
    encoded = encoded && make_code_map(&maps.b[i], it.codes, it.n, k / 2u, 128u) &&
              make_scale_map(&maps.sfb[i], it.scales, static_cast<uint64_t>(it.n / 128u) * (k / 64u));
  }
  if (!encoded) return fail(slot, "nvfp4 prefill: tensor map encoding failed");
  p.status = status;
  p.tokens = tokens;
  p.k = k;
  p.epilogue = epilogue;
  p.q_codes = q.codes;
  p.q_scales = q.scales;
  p.q_din = q.d_in;
  const uint32_t tiles = (pad / kBM + 1u) / 2u * p.n_tiles;
  const uint32_t pairs_max = static_cast<uint32_t>(dev.sm_count) / 2u;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(2u * (tiles < pairs_max ? tiles : pairs_max), 1, 1);
  config.blockDim = dim3(256, 1, 1);
  config.dynamicSmemBytes = kPairSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = dev.pdl ? 2 : 1;
  const cudaError_t err = cudaLaunchKernelEx(&config, w4a4_gemm_pair_kernel, map_a, map_sfa, maps, p);
  if (err != cudaSuccess) return fail(slot, "nvfp4 prefill launch: %s", cudaGetErrorString(err));
  return 0;
}
}  // namespace

int32_t w4a4_launch_parts(ErrorSlot &slot, const DeviceState &dev, const A4Item *parts, uint32_t count, uint32_t k, const uint16_t *x,
                          uint32_t tokens, uint32_t epilogue, uint8_t *workspace, cudaStream_t stream) {
  uint8_t *a_codes = workspace + 256;
  uint8_t *a_scales = a_codes + static_cast<uint64_t>(w4a4_tokens_pad(tokens)) * (k / 2u);
  return w4a4_products(slot, dev, parts, count, k, x, tokens, epilogue, reinterpret_cast<uint32_t *>(workspace), a_codes, a_scales, QuantTarget(),
                       stream);
}

int32_t w4a4_launch(ErrorSlot &slot, const DeviceState &dev, const uint8_t *w_codes, const uint8_t *w_scales, uint32_t n,
                    uint32_t k, float d_w, float d_in, const uint16_t *x, uint32_t tokens, void *y, uint32_t ldy,
                    uint32_t epilogue, uint8_t *workspace, cudaStream_t stream) {
  const A4Item item = {w_codes, w_scales, y, n, ldy, d_w, d_in};
  return w4a4_launch_parts(slot, dev, &item, 1, k, x, tokens, epilogue, workspace, stream);
}

// Quantizes tokens [token_begin, token_begin + token_count) of a call of `tokens_total` tokens into
// their place of the operand in `workspace` (token_begin a multiple of 128: whole scale tiles);
// `x_rows` points at the first of those tokens. Rows between the range's end and the next multiple
// of 128 are written as zeros.
int32_t w4a4_quantize_range(ErrorSlot &slot, const DeviceState &dev, const uint16_t *x_rows, uint32_t tokens_total,
                            uint32_t token_begin, uint32_t token_count, uint32_t k, float d_in, uint8_t *workspace,
                            cudaStream_t stream) {
  const uint64_t pad_total = w4a4_tokens_pad(tokens_total);
  uint8_t *codes = workspace + 256 + static_cast<uint64_t>(token_begin) * (k / 2u);
  uint8_t *scales = workspace + 256 + pad_total * (k / 2u) + static_cast<uint64_t>(token_begin / 128u) * (k / 64u) * 512u;
  return quantize_rows(slot, dev, x_rows, token_count, k, d_in, codes, scales, stream);
}

// Workspace of the MLP: the status line, x quantized (K = k), h quantized (K = inter).
uint64_t w4a4_mlp_workspace_bytes(uint32_t k, uint32_t inter, uint32_t tokens) {
  const uint64_t pad = w4a4_tokens_pad(tokens);
  return 256u + pad * (k / 2u) + pad * (k / 16u) + pad * (inter / 2u) + pad * (inter / 16u);
}

int32_t w4a4_mlp_launch(ErrorSlot &slot, const DeviceState &dev, const uint8_t *gu_codes, const uint8_t *gu_scales, uint32_t gu_n,
                        uint32_t k, float gu_dw, float gu_din, const uint8_t *dn_codes, const uint8_t *dn_scales, uint32_t dn_n,
                        float dn_dw, float dn_din, const uint16_t *x, uint32_t tokens, void *y, uint32_t ldy, uint32_t epilogue,
                        uint8_t *workspace, cudaStream_t stream) {
  const uint64_t pad = w4a4_tokens_pad(tokens);
  const uint32_t inter = gu_n / 2u;
  uint32_t *status = reinterpret_cast<uint32_t *>(workspace);
  uint8_t *x_codes = workspace + 256;
  uint8_t *x_scales = x_codes + pad * (k / 2u);
  QuantTarget h;
  h.codes = x_scales + pad * (k / 16u);
  h.scales = h.codes + pad * (inter / 2u);
  h.d_in = dn_din;
  const A4Item gate_up = {gu_codes, gu_scales, nullptr, gu_n, 0, gu_dw, gu_din}, down = {dn_codes, dn_scales, y, dn_n, ldy, dn_dw, dn_din};
  if (w4a4_products(slot, dev, &gate_up, 1, k, x, tokens, kEpilogueSwiglu | kEpilogueQuant, status, x_codes, x_scales, h, stream) != 0) return -1;
  return w4a4_products(slot, dev, &down, 1, inter, nullptr, tokens, epilogue, status, h.codes, h.scales, QuantTarget(), stream);
}

}  // namespace b200q

// ---- the entry that allocates nothing ------------------------------------------------------------
//
// The W4A4 route keeps the quantized activations and a status line in scratch memory. Here that
// scratch is a fixed array inside the library's own device image instead of a caller-supplied
// workspace, for callers that have no way to hand over device memory when they call.
namespace b200q {
namespace {

static __device__ __align__(256) uint8_t g_static_scratch[B200Q_NVFP4_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxScratchDevices = 64;
// The array's address on each device. In host code the symbol `g_static_scratch` itself is only a
// handle for the runtime, never a device pointer: the address a kernel can use comes from
// cudaGetSymbolAddress, asked once per device while that device is current.
uint8_t *g_scratch_address[kMaxScratchDevices] = {};
std::mutex g_scratch_mutex;

int32_t static_scratch(ErrorSlot &slot, uint8_t **out) {
  int device = -1;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return fail(slot, "b200q_nvfp4_linear_noalloc: no CUDA device: %s", cudaGetErrorString(err));
  if (device < 0 || device >= kMaxScratchDevices) return fail(slot, "b200q_nvfp4_linear_noalloc: device ordinal %d is out of range", device);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_address[device] == nullptr) {
    void *address = nullptr;
    err = cudaGetSymbolAddress(&address, g_static_scratch);
    if (err != cudaSuccess || address == nullptr) {
      return fail(slot, "b200q_nvfp4_linear_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(err));
    }
    // The status line needs no clearing: a file-scope __device__ array is zero when the module is
    // loaded, the kernels only ever OR bits into it, and everything behind it is rewritten by
    // every call before it is read.
    g_scratch_address[device] = static_cast<uint8_t *>(address);
  }
  *out = g_scratch_address[device];
  return 0;
}

bool is_aligned(const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

}  // namespace

// The status line of the built-in scratch array on the current device, after `stream` has
// finished: 0 when b200q_nvfp4_linear_noalloc has not run on this device yet.
int32_t w4a4_noalloc_status(ErrorSlot &slot, cudaStream_t stream, uint32_t *status) {
  *status = 0;
  int device = -1;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return fail(slot, "b200q_nvfp4_device_status: no CUDA device: %s", cudaGetErrorString(err));
  const uint8_t *address = nullptr;
  if (device >= 0 && device < kMaxScratchDevices) {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    address = g_scratch_address[device];
  }
  if (address == nullptr) return 0;
  err = cudaMemcpyAsync(status, address, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
  if (err != cudaSuccess) return fail(slot, "b200q_nvfp4_device_status: %s", cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q

extern "C" int32_t b200q_nvfp4_linear_noalloc(const b200q_nvfp4_weight *w, const void *x, uint32_t tokens, void *y,
                                              uint32_t ldy, uint32_t epilogue, void *stream) {
  using namespace b200q;
  ErrorSlot &slot = nvfp4_error();
  const char *what = "b200q_nvfp4_linear_noalloc";
  if (w == nullptr || w->codes == nullptr || w->scales == nullptr) return fail(slot, "%s: weight is NULL", what);
  if (w->n == 0 || (w->n % 128u) != 0) return fail(slot, "%s: n = %u is not a positive multiple of 128", what, w->n);
  if (w->k == 0 || (w->k % 256u) != 0) return fail(slot, "%s: k = %u is not a positive multiple of 256", what, w->k);
  if (!is_aligned(w->codes, 32) || !is_aligned(w->scales, 16)) return fail(slot, "%s: weight planes are misaligned", what);
  if (!std::isfinite(w->weight_scale_divisor) || !(w->weight_scale_divisor > 0.0f) ||
      !std::isfinite(w->input_scale_divisor) || !(w->input_scale_divisor > 0.0f)) {
    return fail(slot, "%s: both scale divisors must be finite and positive", what);
  }
  if (tokens == 0) return fail(slot, "%s: tokens must be positive", what);
  if ((epilogue & ~static_cast<uint32_t>(B200Q_NVFP4_OUT_F32)) != 0u) return fail(slot, "%s: only STORE (optionally OUT_F32) is served", what);
  if (x == nullptr || !is_aligned(x, 16)) return fail(slot, "%s: x is NULL or not 16-byte aligned", what);
  if (y == nullptr || !is_aligned(y, 16) || (ldy % 8u) != 0 || ldy < w->n) {
    return fail(slot, "%s: y must be 16-byte aligned, ldy a multiple of 8 and at least n", what);
  }
  const uint64_t need = w4a4_workspace_bytes(w->k, tokens);
  if (need > B200Q_NVFP4_NOALLOC_SCRATCH_BYTES) {
    return fail(slot, "%s: %u tokens at k = %u need %llu bytes of scratch, the built-in array holds %llu", what, tokens, w->k,
                static_cast<unsigned long long>(need), static_cast<unsigned long long>(B200Q_NVFP4_NOALLOC_SCRATCH_BYTES));
  }
  const DeviceState *dev = device_state(slot);
  if (dev == nullptr) return -1;
  if (!dev->prepared) return fail(slot, "%s: the device was not prepared (call b200q_nvfp4_prepare at load)", what);
  uint8_t *scratch = nullptr;
  if (static_scratch(slot, &scratch) != 0) return -1;
  return w4a4_launch(slot, *dev, static_cast<const uint8_t *>(w->codes), static_cast<const uint8_t *>(w->scales), w->n, w->k,
                     w->weight_scale_divisor, w->input_scale_divisor, static_cast<const uint16_t *>(x), tokens, y, ldy,
                     epilogue, scratch, static_cast<cudaStream_t>(stream));
}

