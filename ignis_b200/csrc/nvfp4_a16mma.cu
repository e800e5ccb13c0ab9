// NVFP4 A16 products on the tensor cores: y[t][r] = sum_k w[r][k] x[t][k] with BF16 activations
// kept as they are and the weights decoded exactly, for token counts where the decode kernel's
// warp-level MMAs become the limit (more than 8 tokens) up to prefill widths. Stands where the
// reference runs nvfp4_small_t_kernel above a few tokens and nvfp4_a16_mma_kernel from 64 tokens
// (kernel/vendor/src/ops/linear/nvfp4/nvfp4_small_t.cuh:211-377, kernel/src/linear.cu:119-124);
// the design is not theirs.
//
//  * A CTA owns one or two tiles of 128 weight rows (the MMA's M) and a token tile of up to 256 (the MMA's N, a
//    multiple of 16), and walks K in stages of 64. Two tiles share the token tile, an accumulator each:
//    consecutive tiles of a plain product, or a fused SwiGLU's gate rows and their up rows.
//  * One warp brings the packed weights: per four stages 128 bytes of codes of each row (TMA, 128-byte swizzle)
//    and the scale tiles (a bulk copy) into a ring of their own, independent of the previous kernel.
//  * Groups of four decoder warps share the half stages (32 values along K). Thread r of a group owns row r of a tile:
//    it reads the row's 16 bytes of codes and its 2 scale bytes from that ring, widens them to BF16 exactly (widen_half)
//    and stores them to TENSOR MEMORY, from where the MMA takes its A operand: row r is lane r, a column two values. (The
//    decoded tile in shared memory cost a store of 16 KB and a read of 16 KB per stage and tile there, 256 cycles of the
//    128-byte port beside the activations' traffic.) A half stage is widened into registers before its columns are free.
//  * One warp streams the activations: one TMA load of the token tile x 64 BF16 values per stage, 128-byte swizzle,
//    straight from the caller's [tokens][k] matrix (tokens past the end read as zero). Nothing is converted or scaled:
//    BF16 x BF16 products are exact in the FP32 accumulator.
//  * One warp owns tensor memory and issues tcgen05.mma kind::f16 (A and B BF16, M 128, K 16, two per half stage and
//    tile), then commits the columns and the stage back to their writers. The issuing roles run in whole warps with an
//    elected lane (nvfp4_tc.cuh, elect_one).
//  * K can be split over the CTAs of a cluster (narrow weights cannot fill the device otherwise): every CTA pushes its
//    partial sums to the rank that finishes a token, where they are added in rank order: bit-reproducible, no global
//    scratch.
//  * Measured on one layer (q | k | v, o, MLP), decoded weights in shared memory before, in tensor memory now: 99.6 -> 81 us
//    at 17 tokens, 120 -> 102 at 100, 172 -> 145 at 200, 450 -> 380 at 600, 668 -> 624 at 1000. At few tokens the decoder
//    warps bound it (380 cycles a stage and tile), at many the tensor core and, over a whole layer, the power cap.
//  * Every mbarrier wait is bounded; a wait that runs out sets a bit in the library's status word
//    (b200q_nvfp4_device_status) and the CTA falls through to the common exit, frees its tensor
//    memory and returns.
#include "nvfp4_internal.cuh"
#include "nvfp4_tc.cuh"

#include <mutex>

namespace b200q {
namespace {

constexpr int kBM = 128;             // weight rows per CTA
constexpr uint32_t kHalfCols = 16;   // tensor-memory columns of a half stage of BF16 weights: 32 values a row
constexpr uint32_t kProducerTimeout = 0x10u, kMmaTimeout = 0x20u, kEpilogueTimeout = 0x40u, kDecodeTimeout = 0x80u, kReduceTimeout = 0x8000u;

__device__ uint32_t g_a16_status = 0;

struct A16Weight {
  const uint8_t *codes;
  const uint8_t *scales;
  void *y;
  uint32_t n, ldy;
  float inv_dw;
  uint32_t block_begin;  // first CTA of this weight
};

struct A16Maps {
  CUtensorMap m[kMaxGroup];   // the weights' code planes
};

struct A16Params {
  A16Weight w[kMaxGroup];
  uint32_t count;
  uint32_t k, tokens;                 // all tokens of the call; token tile y covers [bn y, bn y + bn)
  uint32_t bn;                        // token tile
  uint32_t a_slots;                   // pieces of decoded weights in tensor memory, a stage or half a stage each
  uint32_t x_stages, raws;            // ring depths in shared memory: activations, packed weights
  uint32_t acc_stride;                // tensor-memory columns from the first accumulator to the second
  uint32_t tmem_cols;
  uint32_t kc;                        // cluster size: K slices
  uint32_t epilogue;                  // STORE / ADD / OUT_F32, or the fused SwiGLU
};

constexpr uint32_t kRawCodes = 128 * 128;                   // four stages of a tile's codes: 128 rows x 256 values
constexpr uint32_t kRawTileBytes = kRawCodes + 4 * 512;     // and its scale tiles

constexpr float kWeightScale = 128.0f;                // the decoded tiles hold weights times 2^-7

constexpr int kGroups = 4, kDecoders = 4 * kGroups;   // groups of four decoder warps
constexpr int kA16Threads = (kDecoders + 3) * 32;     // and a warp each for the activations, the MMAs and the packed weights

// One row's 32 weights of a half stage, widened into the 16 columns of its lane. Both operands of the MMA are BF16, so the
// weights leave as BF16(code * scale * 2^-7): exact, at most 6 significant bits. A code's three magnitude bits on the
// low exponent bits and the top significand bit of a BF16 are the code's value times 2^-126 (0.5 as a
// subnormal, which the multiply takes); one BF16 multiply by scale * 2^119 (448 * 2^119 is the largest and
// still finite) gives the rest. A word beside itself shifted by one code has neighbouring codes 16 bits apart, so a pair
// of them takes two shifts and two logic operations, or one and two: 21 operations for eight codes with the multiplies
// (pairs of codes four apart and a byte permute of each product took 23).
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, __nv_bfloat162 b) {
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&a), b);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ void widen_half(const uint4 codes, float f0, float f1, uint32_t *col) {
  const uint32_t words[4] = {codes.x, codes.y, codes.z, codes.w};
#pragma unroll
  for (int c = 0; c < 4; ++c) {   // word c: values 8 c .. 8 c + 7 of the half stage
    const float f = c < 2 ? f0 : f1;
    const __nv_bfloat162 sg = __floats2bfloat162_rn(f, f);
    const uint32_t w = words[c], w4 = w << 4;
#pragma unroll
    for (int h = 0; h < 2; ++h) {   // codes 4 h .. 4 h + 3: bits 4..7 of the two halves hold the first pair, bits 12..15 the second
      const uint32_t u = __byte_perm(w4, w, h == 0 ? 0x5410 : 0x7632);
      col[4 * c + 2 * h] = bf16x2_mul(((u << 2) & 0x01C001C0u) | ((u << 8) & 0x80008000u), sg);
      col[4 * c + 2 * h + 1] = bf16x2_mul(((u >> 6) & 0x01C001C0u) | (u & 0x80008000u), sg);
    }
  }
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}

// `coef`: the weight's inverse divisor times what the A tiles leave out.
// `bits`: what the residual add found there, as the stored type's bits.
__device__ __forceinline__ void a16_store(const A16Weight &W, uint32_t epilogue, size_t at, float acc, float coef, uint32_t bits) {
  const float val = __fmul_rn(acc, coef);  // not contracted into the residual add: one value for every epilogue
  const float old = __uint_as_float((epilogue & kEpilogueF32) ? bits : bits << 16);
  if (epilogue & kEpilogueF32) {
    static_cast<float *>(W.y)[at] = (epilogue & kEpilogueAdd) ? old + val : val;
  } else {
    static_cast<__nv_bfloat16 *>(W.y)[at] = __float2bfloat16_rn((epilogue & kEpilogueAdd) ? val + old : val);
  }
}
// The residuals of several of a tile's `live` tokens, `step` apart (past the last one: the last), requested together before any
// of them is needed. One at a time, each behind its own branches, they are round trips one after another.
template <int N>
__device__ __forceinline__ void a16_residuals(uint32_t (&bits)[N], const A16Weight &W, uint32_t epilogue, size_t row, uint32_t tok0, uint32_t first,
                                              uint32_t step, uint32_t live) {
  if (!(epilogue & kEpilogueAdd)) return;
  if (epilogue & kEpilogueF32) {
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) bits[j] = static_cast<const uint32_t *>(W.y)[static_cast<size_t>(tok0 + min(first + j * step, live - 1u)) * W.ldy + row];
  } else {
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) bits[j] = static_cast<const uint16_t *>(W.y)[static_cast<size_t>(tok0 + min(first + j * step, live - 1u)) * W.ldy + row];
  }
}
__device__ __forceinline__ void a16_store_swiglu(const A16Weight &W, size_t at, float acc_g, float acc_u, float coef) {
  const float g = acc_g * coef, u = acc_u * coef;
  static_cast<__nv_bfloat16 *>(W.y)[at] = __float2bfloat16_rn(g / (1.0f + __expf(-g)) * u);
}

// TILES: row tiles per CTA (a fused SwiGLU has two: gate rows and their up rows). HALVES: half stages a piece of decoded
// weights has. A whole stage takes fewer instructions; half ones still fit two tiles beside accumulators of up to 224 columns.
template <int TILES, int HALVES>
__global__ void __launch_bounds__(kA16Threads, 1) nvfp4_a16_mma_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                    const __grid_constant__ A16Maps maps,
                                                                    const __grid_constant__ A16Params p) {
  constexpr uint32_t kRawBytes = TILES * kRawTileBytes, kCols = HALVES * kHalfCols, kSlotCols = TILES * kCols;
  constexpr uint32_t kPerTile = kGroups / TILES;       // groups at work on a tile; at most a_slots of them (one parity tells two uses of a slot apart)
  constexpr uint32_t kPieces = 8 / HALVES;             // pieces of a quad of stages
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw);
  const uint32_t x_bytes = p.bn * 128u;                       // one stage of activations
  // rings: activations [x_stages], packed weights [raws], and in tensor memory decoded weights [a_slots]; each with its
  // full and empty barriers
  const uint32_t raw_ring = base + p.x_stages * x_bytes, bars = raw_ring + p.raws * kRawBytes;
  const uint32_t bar_a = bars, bar_a_empty = bar_a + 8u * p.a_slots, bar_x = bar_a_empty + 8u * p.a_slots, bar_x_empty = bar_x + 8u * p.x_stages,
                 bar_raw = bar_x_empty + 8u * p.x_stages, bar_raw_empty = bar_raw + 8u * p.raws, bar_acc = bar_raw_empty + 8u * p.raws,
                 bar_sums = bar_acc + 8u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base_ptr + (bar_sums - base) + 8u);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), kc = p.kc;

  // Which weight, row tiles and token tile this CTA serves. Without a K split the grid is walked
  // token tile first, so the CTAs running at one time share weight rows (read from HBM once, then
  // from the L2) rather than activations.
  uint32_t bx = blockIdx.x, by = blockIdx.y;
  if (kc == 1u) {
    const uint32_t id = blockIdx.y * gridDim.x + blockIdx.x;
    by = id % gridDim.y;
    bx = id / gridDim.y;
  }
  uint32_t wi = 0;
#pragma unroll
  for (uint32_t i = 1; i < kMaxGroup; ++i) {
    if (i < p.count && bx >= p.w[i].block_begin) wi = i;
  }
  const A16Weight &W = p.w[wi];
  const bool swiglu = TILES == 2 && (p.epilogue & kEpilogueSwiglu) != 0u;
  const uint32_t block = (bx - W.block_begin) / kc;
  const uint32_t tile_a = TILES == 2 && !swiglu ? 2u * block : block;      // 128-row tiles of the weight
  const uint32_t tile_b = swiglu ? W.n / 256u + block : tile_a + 1u;       // the second, with two
  const uint32_t k_stages = p.k / 64u, k_quads = (k_stages + 3u) / 4u;     // K is split in whole groups of four stages
  const uint32_t q0 = static_cast<uint32_t>(static_cast<uint64_t>(k_quads) * rank / kc);
  const uint32_t q1 = static_cast<uint32_t>(static_cast<uint64_t>(k_quads) * (rank + 1) / kc);
  const uint32_t s0 = 4u * q0, stages = min(4u * q1, k_stages) - s0;       // this CTA's stages
  const uint32_t tok0 = by * p.bn;

  const uint32_t live = min(p.tokens - tok0, p.bn);   // tokens of the tile
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < p.a_slots; ++s) {
      mbar_init(bar_a + 8 * s, 4 * TILES);      // the four decoder warps of each tile
      mbar_init(bar_a_empty + 8 * s, 1);        // the MMA warp's commit
    }
    for (uint32_t s = 0; s < p.x_stages; ++s) {
      mbar_init(bar_x + 8 * s, 1);              // the producer's expect_tx arrival
      mbar_init(bar_x_empty + 8 * s, 1);
    }
    for (uint32_t d = 0; d < p.raws; ++d) {
      mbar_init(bar_raw + 8 * d, 1);
      mbar_init(bar_raw_empty + 8 * d, kDecoders);
    }
    mbar_init(bar_acc, 1);
    mbar_init(bar_sums, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // every rank of the cluster sends its sums of the tokens that this one finishes
    if (kc > 1u) mbar_expect_tx(bar_sums, kc * ((live + kc - 1u - rank) / kc) * TILES * 512u);
  }
  if (warp == kDecoders + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
  const uint32_t tmem_a = tmem + TILES * p.acc_stride;   // decoded weights behind the accumulators

  if (warp < kDecoders) {
    // ---- row threads: the groups of a tile decode its half stages in turn ----
    const uint32_t r = threadIdx.x & 127u, group = static_cast<uint32_t>(warp) / 4u, sw = r & 7u;
    const uint32_t tile = TILES == 2 ? group & 1u : 0u, g = TILES == 2 ? group >> 1 : group;
    const uint32_t code_off = tile * kRawTileBytes + r * 128u, scale_off = tile * kRawTileBytes + kRawCodes + (r & 31u) * 16u + (r >> 5) * 4u;
    const uint32_t cols = tmem_a + tile * kCols + ((static_cast<uint32_t>(warp) & 3u) << 21);   // the warp's 32 lanes
    griddep_launch_dependents();
    RingAt at, from;
    at.step(g, p.a_slots);
    for (uint32_t it = g; it < 2u / HALVES * stages; it += kPerTile, at.step(kPerTile, p.a_slots)) {
      const uint32_t j = it % kPieces, raw_at = raw_ring + from.slot * kRawBytes;   // piece j of its quad
      if (!mbar_wait(bar_raw + 8 * from.slot, from.phase)) {
        if (lane == 0) atomicOr(&g_a16_status, kDecodeTimeout);
        break;
      }
      uint32_t col[HALVES * kHalfCols], scales[HALVES];
      uint4 codes[HALVES];
#pragma unroll
      for (uint32_t h = 0; h < HALVES; ++h) {
        const uint32_t half = HALVES * j + h;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(codes[h].x), "=r"(codes[h].y), "=r"(codes[h].z), "=r"(codes[h].w) : "r"(raw_at + code_off + ((half ^ sw) << 4)));
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(scales[h]) : "r"(raw_at + scale_off + (half >> 1) * 512u + (half & 1u) * 2u));
      }
#pragma unroll
      for (uint32_t h = 0; h < HALVES; ++h) {
        const uint32_t s01 = e4m3x2_to_half2(scales[h]);
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&s01));
        const float up = 6.646139978924579e35f;  // 2^119
        widen_half(codes[h], f.x * up, f.y * up, col + h * kHalfCols);
      }
      if (j + kPerTile >= kPieces) {   // the group's last piece of the quad
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_raw_empty + 8 * from.slot);
        from.step(1u, p.raws);
      }
      if (!mbar_wait(bar_a_empty + 8 * at.slot, at.phase ^ 1u)) {
        if (lane == 0) atomicOr(&g_a16_status, kDecodeTimeout);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if constexpr (HALVES == 2) tmem_st32(cols + at.slot * kSlotCols, col);
      else tmem_st16(cols + at.slot * kSlotCols, col);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_a + 8 * at.slot);
    }
    griddep_wait();   // the epilogue reads and writes what the previous kernels may use
  } else if (warp == kDecoders) {
    // ---- producer of the activation tiles ----
    griddep_launch_dependents();
    griddep_wait();   // the activations may come from the previous kernel
    RingAt at;
    for (uint32_t s = 0; s < stages; ++s, at.step(1u, p.x_stages)) {
      if (!mbar_wait(bar_x_empty + 8 * at.slot, at.phase ^ 1u)) {
        if (lane == 0) atomicOr(&g_a16_status, kProducerTimeout);
        break;
      }
      if (elect_one()) {
        mbar_expect_tx(bar_x + 8 * at.slot, x_bytes);
        tma_load_2d(base + at.slot * x_bytes, &map_x, bar_x + 8 * at.slot, static_cast<int32_t>((s0 + s) * 64u), static_cast<int32_t>(tok0));
      }
      __syncwarp();
    }
  } else if (warp == kDecoders + 2) {
    // ---- producer of the packed weights: they never depend on the previous kernel ----
    griddep_launch_dependents();
    const uint64_t policy = l2_evict_first_policy();
    const bool once = gridDim.y == 1u;   // several token tiles read the same weights: leave them in the L2
    const CUtensorMap *map = &maps.m[wi];
    RingAt at;
    for (uint32_t q = q0; q < q1; ++q, at.step(1u, p.raws)) {
      if (!mbar_wait(bar_raw_empty + 8 * at.slot, at.phase ^ 1u)) {
        if (lane == 0) atomicOr(&g_a16_status, kProducerTimeout);
        break;
      }
      if (elect_one()) {
        const uint32_t full = bar_raw + 8 * at.slot, dst = raw_ring + at.slot * kRawBytes;
        const uint32_t scale_bytes = (min(4u * q + 4u, k_stages) - 4u * q) * 512u;
        mbar_expect_tx(full, TILES * (kRawCodes + scale_bytes));
#pragma unroll
        for (int t = 0; t < TILES; ++t) {
          const uint32_t tile = t == 0 ? tile_a : tile_b;
          if (once) tma_load_2d_hint(dst + t * kRawTileBytes, map, full, static_cast<int32_t>(q * 128u), static_cast<int32_t>(tile * 128u), policy);
          else tma_load_2d(dst + t * kRawTileBytes, map, full, static_cast<int32_t>(q * 128u), static_cast<int32_t>(tile * 128u));
          bulk_load(dst + t * kRawTileBytes + kRawCodes, W.scales + (static_cast<size_t>(tile) * k_stages + 4u * q) * 512u, scale_bytes, full);
        }
      }
      __syncwarp();
    }
  } else {
    // ---- MMA issuer ----
    griddep_launch_dependents();
    // instruction descriptor: FP32 accumulator (bit 4), A and B BF16 (format 1 at bits 7 and
    // 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((p.bn >> 3) << 17) | ((static_cast<uint32_t>(kBM) >> 4) << 24);
    const uint64_t x_desc0 = smem_desc_sw128(base);
    bool ok = true;
    RingAt at, xat;
    for (uint32_t it = 0; it < stages && ok; ++it, xat.step(1u, p.x_stages)) {
      ok = mbar_wait(bar_x + 8 * xat.slot, xat.phase);
#pragma unroll
      for (uint32_t piece = 0; piece < 2u / HALVES; ++piece, at.step(1u, p.a_slots)) {
        ok = ok && mbar_wait(bar_a + 8 * at.slot, at.phase);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint32_t a = tmem_a + at.slot * kSlotCols;
          const uint64_t x_desc = x_desc0 + xat.slot * (x_bytes >> 4) + 4u * piece;
#pragma unroll
          for (uint32_t kb = 0; kb < 2u * HALVES; ++kb) {   // 16 values along K: 8 columns of A, two 16-byte units of x further
            const uint32_t accumulate = (it | piece | kb) != 0u ? 1u : 0u;
            mma_f16_ts(tmem, a + 8u * kb, x_desc + 2u * kb, idesc, accumulate);
            if (TILES == 2) mma_f16_ts(tmem + p.acc_stride, a + kCols + 8u * kb, x_desc + 2u * kb, idesc, accumulate);
          }
          mma_commit(bar_a_empty + 8 * at.slot);
          if (piece + 1u == 2u / HALVES) mma_commit(bar_x_empty + 8 * xat.slot);
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) atomicOr(&g_a16_status, kMmaTimeout);
    if (ok && elect_one()) mma_commit(bar_acc);
    __syncwarp();
  }

  // ---- epilogue: warp w owns accumulator lanes (tile rows) 32 (w % 4) .. + 31; the groups of four warps take
  //      the chunks of 16 tokens in turn ----
  const uint32_t quad = static_cast<uint32_t>(warp) & 3u, group = static_cast<uint32_t>(warp) / 4u;
  const uint32_t r = quad * 32u + static_cast<uint32_t>(lane);
  const size_t row_a = static_cast<size_t>(tile_a) * 128u + r, row_b = static_cast<size_t>(tile_b) * 128u + r;
  const uint32_t lane_base = tmem + ((quad * 32u) << 16);
  const float coef = W.inv_dw * kWeightScale;
  bool have = false;
  if (warp < kDecoders) {
    have = mbar_wait(bar_acc, 0u);
    if (!have && lane == 0) atomicOr(&g_a16_status, kEpilogueTimeout);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (kc == 1u) {
    if (warp < kDecoders && have) {
      for (uint32_t c = group * 16u; c < p.bn && tok0 + c < p.tokens; c += kGroups * 16u) {
        uint32_t v[16], u[16], old[16] = {};
        tmem_ld16(lane_base + c, v);
        if (TILES == 2) tmem_ld16(lane_base + p.acc_stride + c, u);
        a16_residuals(old, W, p.epilogue, row_a, tok0, c, 1u, live);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (swiglu) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (tok0 + c + j < p.tokens) {
              a16_store_swiglu(W, static_cast<size_t>(tok0 + c + j) * W.ldy + row_a, __uint_as_float(v[j]), TILES == 2 ? __uint_as_float(u[j]) : 0.0f, coef);
            }
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (tok0 + c + j < p.tokens) a16_store(W, p.epilogue, static_cast<size_t>(tok0 + c + j) * W.ldy + row_a, __uint_as_float(v[j]), coef, old[j]);
        }
        if (TILES == 2) {
          a16_residuals(old, W, p.epilogue, row_b, tok0, c, 1u, live);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (tok0 + c + j < p.tokens) a16_store(W, p.epilogue, static_cast<size_t>(tok0 + c + j) * W.ldy + row_b, __uint_as_float(u[j]), coef, old[j]);
          }
        }
      }
    }
  } else {
    // Token tl of the tile is finished by rank tl % kc: once every ring of the cluster is idle, every CTA pushes its sums of
    // it over that rank's rings, [sender][turn][tile][128 rows], and the bytes count at the receiver's barrier. Nobody reads
    // another CTA's memory, so nobody waits for a reader before it leaves.
    constexpr uint32_t kAtOnce = 4;   // tokens of a group whose residuals are requested together, the first before the sums are here
    uint32_t old_a[kAtOnce] = {}, old_b[kAtOnce] = {};
    auto residuals = [&](uint32_t i) {
      a16_residuals(old_a, W, p.epilogue, row_a, tok0, i * kc + rank, kGroups * kc, live);
      if (TILES == 2 && !swiglu) a16_residuals(old_b, W, p.epilogue, row_b, tok0, i * kc + rank, kGroups * kc, live);
    };
    if (warp < kDecoders) residuals(group);
    __syncwarp();
    cluster_sync_all();
    const uint32_t turns = (live + kc - 1u) / kc;
    if (warp < kDecoders) {
      const uint32_t mine = base + (rank * turns * TILES * 128u + r) * 4u;
      for (uint32_t c = group * 16u; c < live; c += kGroups * 16u) {
        uint32_t v[16], u[16];
        if (have) {
          tmem_ld16(lane_base + c, v);
          if (TILES == 2) tmem_ld16(lane_base + p.acc_stride + c, u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        uint32_t to = c % kc, at = mine + c / kc * TILES * 512u;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c + j >= live) break;
          const uint32_t bar = cluster_map(bar_sums, to);
          push_f32(cluster_map(at, to), have ? __uint_as_float(v[j]) : 0.0f, bar);
          if (TILES == 2) push_f32(cluster_map(at + 512u, to), have ? __uint_as_float(u[j]) : 0.0f, bar);
          if (++to == kc) to = 0u, at += TILES * 512u;
        }
      }
      if (mbar_wait_pushed(bar_sums)) {
        const float *sums = reinterpret_cast<const float *>(base_ptr) + r;
        for (uint32_t first = group; first * kc + rank < live; first += kAtOnce * kGroups) {
          if (first != group) residuals(first);
#pragma unroll
          for (uint32_t b = 0; b < kAtOnce; ++b) {
            const uint32_t i = first + b * kGroups;
            if (i * kc + rank >= live) break;
            float sum_a = 0.0f, sum_b = 0.0f;
            for (uint32_t q = 0; q < kc; ++q) {   // in rank order
              const float *from = sums + (q * turns + i) * TILES * 128u;
              sum_a = q == 0u ? from[0] : sum_a + from[0];
              if (TILES == 2) sum_b = q == 0u ? from[128] : sum_b + from[128];
            }
            const size_t at = static_cast<size_t>(tok0 + i * kc + rank) * W.ldy;
            if (swiglu) {
              a16_store_swiglu(W, at + row_a, sum_a, sum_b, coef);
            } else {
              a16_store(W, p.epilogue, at + row_a, sum_a, coef, old_a[b]);
              if (TILES == 2) a16_store(W, p.epilogue, at + row_b, sum_b, coef, old_b[b]);
            }
          }
        }
      } else if (lane == 0) {
        atomicOr(&g_a16_status, kReduceTimeout);
      }
    }
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kDecoders + 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

// ---- host side --------------------------------------------------------------------------------
constexpr size_t kA16MaxSmem = 224 * 1024;

struct A16Plan {
  uint32_t tiles, halves, bn, kc, a_slots, x_stages, raws, acc_stride, tmem_cols;
};

size_t a16_ring_bytes(const A16Plan &pl) { return static_cast<size_t>(pl.x_stages) * pl.bn * 128u + static_cast<size_t>(pl.raws) * pl.tiles * kRawTileBytes; }
// What the CTAs of a cluster push to one of them lies over the rings: the tile's tokens in whole turns of the cluster, whose
// ranks finish one each.
constexpr size_t a16_sums_bytes(uint32_t tiles, uint32_t tokens, uint32_t kc) { return static_cast<size_t>(tiles) * ((tokens + kc - 1u) / kc * kc) * 512u; }
static_assert(a16_sums_bytes(1u, 16u, 3u) == 18u * 512u && a16_sums_bytes(2u, 16u, 8u) == 32u * 512u, "whole turns");
size_t a16_smem_bytes(const A16Plan &pl) { return a16_ring_bytes(pl) + 16u * (pl.a_slots + pl.x_stages + pl.raws) + 48u + 1024u; }

// Columns of tensor memory: the accumulators, then as many pieces of decoded weights as fit, up to four stages; half ones
// where two whole ones do not fit. Ring depths: two of each at least, then in turn packed weights (what is in flight there
// hides the latency of HBM) and activations, up to 6 and 8.
bool a16_rings(A16Plan &pl) {
  pl.acc_stride = (pl.bn + 31u) / 32u * 32u;
  const uint32_t per_tile = static_cast<uint32_t>(kGroups) / pl.tiles;
  for (pl.halves = 2u;; --pl.halves) {
    pl.a_slots = pl.tiles * pl.acc_stride < 512u ? (512u - pl.tiles * pl.acc_stride) / (pl.tiles * pl.halves * kHalfCols) : 0u;
    if (pl.a_slots > 8u / pl.halves) pl.a_slots = 8u / pl.halves;
    if (pl.a_slots >= per_tile) break;
    if (pl.halves == 1u || pl.tiles == 1u) return false;
  }
  pl.tmem_cols = 32u;
  while (pl.tmem_cols < pl.tiles * (pl.acc_stride + pl.a_slots * pl.halves * kHalfCols)) pl.tmem_cols <<= 1;
  pl.x_stages = pl.raws = 2u;
  if (a16_smem_bytes(pl) > kA16MaxSmem) return false;
  auto grow = [&](uint32_t &depth, uint32_t most) {
    if (depth >= most) return false;
    ++depth;
    if (a16_smem_bytes(pl) <= kA16MaxSmem) return true;
    --depth;
    return false;
  };
  for (bool grew = true; grew;) {
    grew = grow(pl.raws, 6u);
    grew = grow(pl.x_stages, 8u) || grew;
  }
  return true;
}

// The shape of a CTA for `row_tiles` tiles of 128 rows (of a SwiGLU: gate tiles): the one that costs least in waves of
// CTAs, by a model in cycles fitted to every shape of four weights (8192 x 5120, 5120 x 6144, 34816 x 5120 fused, 5120 x
// 17408) at 17 to 2500 tokens, which it follows within 6 %; the shape it picks is within 4 % of the fastest one measured
// everywhere, 0.1 % on average. A stage costs the slowest of the decoder warps (380 a tile), the tensor core (2.46 bn a
// tile), what the CTA brings from the L2 (128 bytes a token and 4.6 KB a tile at about 61 bytes a cycle) and 400 of barrier
// round trips, and a sixth of the lesser of the first two; a CTA has its epilogue besides and, with a K split, the exchange.
A16Plan a16_plan(const DeviceState &dev, uint32_t row_tiles, uint32_t k_stages, uint32_t tokens, bool swiglu, bool even) {
  A16Plan best = {};
  best.bn = 0;
  double best_cost = 1e30;
  for (uint32_t tiles = swiglu ? 2u : 1u; tiles <= (swiglu || even ? 2u : 1u); ++tiles) {
    const uint32_t nt_min = (tokens + 255u) / 256u;
    for (uint32_t nt = nt_min; nt <= nt_min + nt_min / 2u + 4u; ++nt) {
      A16Plan pl = {};
      pl.tiles = tiles;
      pl.bn = ((tokens + nt - 1u) / nt + 15u) / 16u * 16u;
      if (nt > nt_min && pl.bn < 64u) break;
      if (!a16_rings(pl)) continue;
      const uint32_t token_tiles = (tokens + pl.bn - 1u) / pl.bn, blocks = tiles == 2u && !swiglu ? row_tiles / 2u : row_tiles;
      for (uint32_t kc = 1; kc <= 8u; ++kc) {
        if (kc > 1u && k_stages / kc < 8u) break;
        if (kc > 1u && a16_sums_bytes(tiles, pl.bn, kc) > a16_ring_bytes(pl)) continue;
        const double ctas = static_cast<double>(blocks) * token_tiles * kc, sms = dev.sm_count;
        // Clusters are placed inside one GPC, and how many CTAs that leaves room for differs from size to size and from device
        // to device (135, 132, 130, 132, 105 and 120 of 148 for 3 to 8 on one). With 0.87 of the SMs for the wide ones 16 clusters of 8 were
        // planned as one wave and ran as two: 4096 x 14336 at 9 tokens 36.9 us, 22.6 here (cold), 2048 x 6144 at 16 20.5 and 14.6,
        // 1024 x 5120 at 150 22.5 and 16.3.
        const double waves = ceil(ctas / (dev.a16_slots[kc] > 0 ? dev.a16_slots[kc] : sms * 0.7));
        const double decode = tiles * 380.0, mma = tiles * 2.46 * pl.bn, load = (pl.bn * 128.0 + tiles * 4608.0) / 61.0;
        double stage = 400.0;
        for (const double limit : {decode, mma, load}) stage = stage > limit ? stage : limit;
        const double cost = waves * (ceil(static_cast<double>(k_stages) / kc) * (stage + 0.16 * (decode < mma ? decode : mma)) + 700.0 + tiles * 28.0 * pl.bn +
                                     (kc > 1u ? 4300.0 + tiles * 19.0 * pl.bn : 0.0));
        if (cost < best_cost) {
          best_cost = cost;
          best = pl;
          best.kc = kc;
        }
      }
    }
  }
  return best;
}

}  // namespace

int32_t a16mma_prepare(ErrorSlot &slot) {
  const int most = static_cast<int>(kA16MaxSmem);
  cudaError_t err = cudaFuncSetAttribute(nvfp4_a16_mma_kernel<1, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(nvfp4_a16_mma_kernel<2, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (err == cudaSuccess) err = cudaFuncSetAttribute(nvfp4_a16_mma_kernel<2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (err != cudaSuccess) return fail(slot, "nvfp4 A16 tensor-core kernel attributes: %s", cudaGetErrorString(err));
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
  DeviceState *dev = device_state(slot);
  if (dev == nullptr) return -1;
  for (int kc = 1; kc <= 8 && !dev->counted; ++kc) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(kc) * 1024u, 1, 1);
    config.blockDim = dim3(kA16Threads, 1, 1);
    config.dynamicSmemBytes = kA16MaxSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(kc);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, nvfp4_a16_mma_kernel<1, 2>, &config) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    dev->a16_slots[kc] = clusters * kc;
  }
  return 0;
}

bool a16mma_takes(uint32_t k, const void *x) { return (k % 64u) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0; }

// `count` weights sharing x, any number of tokens: token tiles side by side in the grid.
int32_t a16mma_launch(ErrorSlot &slot, const DeviceState &dev, const GemvWeight *weights, uint32_t count, const uint16_t *x,
                      uint32_t k, uint32_t tokens, uint32_t epilogue, cudaStream_t stream) {
  const bool swiglu = (epilogue & kEpilogueSwiglu) != 0u;
  uint32_t row_tiles = 0;
  bool even = true;
  for (uint32_t i = 0; i < count; ++i) {
    row_tiles += weights[i].n / (swiglu ? 256u : 128u);
    even = even && (weights[i].n % 256u) == 0u;
  }
  const A16Plan pl = a16_plan(dev, row_tiles, k / 64u, tokens, swiglu, even);
  if (pl.bn == 0u) return fail(slot, "nvfp4 A16 tensor-core route: no plan for %u tokens", tokens);
  A16Params p = {};
  p.count = count;
  p.k = k;
  p.tokens = tokens;
  p.bn = pl.bn;
  p.a_slots = pl.a_slots;
  p.x_stages = pl.x_stages;
  p.raws = pl.raws;
  p.acc_stride = pl.acc_stride;
  p.tmem_cols = pl.tmem_cols;
  p.kc = pl.kc;
  p.epilogue = epilogue;
  uint32_t ctas = 0;
  for (uint32_t i = 0; i < count; ++i) {
    A16Weight &g = p.w[i];
    g.codes = weights[i].codes;
    g.scales = weights[i].scales;
    g.y = weights[i].y[0];
    g.n = weights[i].n;
    g.ldy = weights[i].ldy;
    g.inv_dw = weights[i].inv_dw;
    g.block_begin = ctas;
    ctas += weights[i].n / (pl.tiles == 2u ? 256u : 128u) * pl.kc;
  }
  EncodeTiledFn encode = encode_tiled_fn();
  A16Maps maps = {};
  for (uint32_t i = 0; i < count; ++i) {
    if (!make_code_map(&maps.m[i], weights[i].codes, weights[i].n, k / 2u, 128u)) {
      return fail(slot, "nvfp4 A16 tensor-core route: tensor map encoding failed");
    }
  }
  CUtensorMap map_x;
  {
    const cuuint64_t dims[2] = {k, tokens};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2u};
    const cuuint32_t box[2] = {64u, pl.bn};
    const cuuint32_t elem[2] = {1, 1};
    if (encode == nullptr ||
        encode(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(x), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
      return fail(slot, "nvfp4 A16 tensor-core route: tensor map encoding failed");
    }
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(ctas, (tokens + pl.bn - 1u) / pl.bn, 1);
  config.blockDim = dim3(kA16Threads, 1, 1);
  config.dynamicSmemBytes = a16_smem_bytes(pl);
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pl.kc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = dev.pdl ? 2 : 1;
  const auto kernel = pl.tiles == 1u ? nvfp4_a16_mma_kernel<1, 2> : pl.halves == 2u ? nvfp4_a16_mma_kernel<2, 2> : nvfp4_a16_mma_kernel<2, 1>;
  const cudaError_t err = cudaLaunchKernelEx(&config, kernel, map_x, maps, p);
  if (err != cudaSuccess) return fail(slot, "nvfp4 A16 tensor-core launch: %s", cudaGetErrorString(err));
  return 0;
}

int32_t a16mma_status(ErrorSlot &slot, cudaStream_t stream, uint32_t *status) {
  cudaError_t err = cudaMemcpyFromSymbolAsync(status, g_a16_status, sizeof(uint32_t), 0, cudaMemcpyDeviceToHost, stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
  if (err != cudaSuccess) return fail(slot, "b200q_nvfp4_device_status: %s", cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q
