// NVFP4 A16 products on the tensor cores: y[t][r] = sum_k w[r][k] x[t][k] with BF16 activations
// kept as they are and the weights decoded exactly, for token counts where the decode kernel's
// warp-level MMAs become the limit (more than 16 tokens) up to prefill widths. Stands where the
// reference runs nvfp4_small_t_kernel above a few tokens and nvfp4_a16_mma_kernel from 64 tokens
// (kernel/vendor/src/ops/linear/nvfp4/nvfp4_small_t.cuh:211-377, kernel/src/linear.cu:119-124);
// the design is not theirs.
//
//  * A CTA owns one or two tiles of 128 weight rows (the MMA's M) and a token tile of up to 256 (the MMA's N, a
//    multiple of 16), and walks K in stages of 64. Two tiles share the token tile, an accumulator each:
//    consecutive tiles of a plain product, or a fused SwiGLU's gate rows and their up rows.
//  * Warp 18 brings the packed weights: per four stages 128 bytes of codes of each row (TMA, 128-byte swizzle)
//    and the scale tiles (a bulk copy) into a ring of their own, independent of the previous kernel.
//  * Four groups of four decoder warps share the stages. Thread r of a group owns row r of a tile: it reads
//    the row's 32 bytes of codes and its 4 scale bytes (one word of the swizzled plane) from that ring,
//    widens them to BF16 exactly (widen_row) and stores the 128 bytes into the stage's A tile in the K-major
//    128-byte-swizzle layout the tensor core reads. (Codes requested ahead into registers would have to arrive
//    before the fence that hands a tile to the tensor core lets a thread go on.)
//  * Warp 16 streams the activations: one TMA load of the token tile x 64 BF16 values per stage, the
//    same swizzle, straight from the caller's [tokens][k] matrix (tokens past the end read as
//    zero). Nothing is converted or scaled: BF16 x BF16 products are exact in the FP32 accumulator.
//  * Warp 17 owns tensor memory and issues tcgen05.mma kind::f16 (A and B BF16, M 128, K 16, four per stage and
//    tile), then commits the stage back to its writers. The issuing roles run in whole warps with an elected
//    lane (nvfp4_tc.cuh, elect_one): with a branch on the lane the same kernel took 2.5 times as long.
//    Measured on one 27B-style layer: 99 us at 17 tokens, 122 at 100, 458 at 600 (the kernel before: 156, 470, 1786).
//  * K can be split over the CTAs of a cluster (narrow weights cannot fill the device otherwise):
//    every CTA pulls its accumulators to shared memory, the cluster meets in distributed shared
//    memory, and the tokens are dealt to the CTAs, which add the partial sums in rank order:
//    bit-reproducible, no global scratch.
//  * Every mbarrier wait is bounded; a wait that runs out sets a bit in the library's status word
//    (b200q_nvfp4_device_status) and the CTA falls through to the common exit, frees its tensor
//    memory and returns.
#include "nvfp4_internal.cuh"
#include "nvfp4_tc.cuh"

#include <mutex>

namespace b200q {
namespace {

constexpr int kBM = 128;             // weight rows per CTA
constexpr uint32_t kABytes = kBM * 128;  // one stage of BF16 weights: 128 rows x 64 values
constexpr uint32_t kProducerTimeout = 0x10u, kMmaTimeout = 0x20u, kEpilogueTimeout = 0x40u, kDecodeTimeout = 0x80u;

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
  uint32_t a_stages, x_stages, raws;  // ring depths in shared memory: decoded tiles, activations, packed weights
  uint32_t acc_stride;                // tensor-memory columns from the first accumulator to the second
  uint32_t tmem_cols;
  uint32_t kc;                        // cluster size: K slices
  uint32_t epilogue;                  // STORE / ADD / OUT_F32, or the fused SwiGLU
};

struct CodeStage {
  uint32_t c[8];   // 64 codes
  uint32_t sc;     // their 4 scales
};

constexpr uint32_t kRawCodes = 128 * 128;                   // four stages of a tile's codes: 128 rows x 256 values
constexpr uint32_t kRawTileBytes = kRawCodes + 4 * 512;     // and its scale tiles

constexpr int kGroups = 4, kDecoders = 4 * kGroups;   // groups of four decoder warps
constexpr int kA16Threads = (kDecoders + 3) * 32;
constexpr float kWeightScale = 128.0f;                // the A tiles hold weights times 2^-7

// One row's 64 weights of a stage, widened into its 128 bytes of the A tile (`tile`: the row's address,
// `sw`: its low bits). Both operands of the MMA are BF16, so the weights leave as
// BF16(code * scale * 2^-7): exact, at most 6 significant bits. A code's three magnitude bits on the
// low exponent bits and the top significand bit of a BF16 are the code's value times 2^-126 (0.5 as a
// subnormal, which the multiply takes); one BF16 multiply by scale * 2^119 (448 * 2^119 is the largest and
// still finite) gives the rest. Codes four apart lie 16 bits apart in their word, so a pair of them
// takes two shifts and two logic operations; the products change places by byte permutes. 23 operations for
// eight codes; converting bytes by cvt.e2m1x2 to fp16 and moving those bits to BF16 took 27 and more.
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, __nv_bfloat162 b) {
  const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&a), b);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ void widen_row(const CodeStage &st, uint32_t tile, uint32_t sw) {
  const uint32_t s01 = e4m3x2_to_half2(st.sc & 0xFFFFu), s23 = e4m3x2_to_half2(st.sc >> 16);
  const float2 f01 = __half22float2(*reinterpret_cast<const __half2 *>(&s01));
  const float2 f23 = __half22float2(*reinterpret_cast<const __half2 *>(&s23));
  const float up = 6.646139978924579e35f;  // 2^119
  const float fs[4] = {f01.x * up, f01.y * up, f23.x * up, f23.y * up};
#pragma unroll
  for (int g4 = 0; g4 < 4; ++g4) {
    const __nv_bfloat162 sg = __floats2bfloat162_rn(fs[g4], fs[g4]);
#pragma unroll
    for (int c = 2 * g4; c < 2 * g4 + 2; ++c) {   // word c: values 8 c .. 8 c + 7 of the stage
      const uint32_t w = st.c[c];
      const uint32_t p04 = bf16x2_mul(((w << 6) & 0x01C001C0u) | ((w << 12) & 0x80008000u), sg);
      const uint32_t p15 = bf16x2_mul(((w << 2) & 0x01C001C0u) | ((w << 8) & 0x80008000u), sg);
      const uint32_t p26 = bf16x2_mul(((w >> 2) & 0x01C001C0u) | ((w << 4) & 0x80008000u), sg);
      const uint32_t p37 = bf16x2_mul(((w >> 6) & 0x01C001C0u) | (w & 0x80008000u), sg);
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile + ((static_cast<uint32_t>(c) ^ sw) << 4)),
                   "r"(__byte_perm(p04, p15, 0x5410)), "r"(__byte_perm(p26, p37, 0x5410)), "r"(__byte_perm(p04, p15, 0x7632)),
                   "r"(__byte_perm(p26, p37, 0x7632))
                   : "memory");
    }
  }
}

// `coef`: the weight's inverse divisor times what the A tiles leave out.
__device__ __forceinline__ void a16_store(const A16Weight &W, uint32_t epilogue, size_t at, float acc, float coef) {
  const float val = __fmul_rn(acc, coef);  // not contracted into the residual add: one value for every epilogue
  if (epilogue & kEpilogueF32) {
    float *y = static_cast<float *>(W.y);
    y[at] = (epilogue & kEpilogueAdd) ? y[at] + val : val;
  } else {
    __nv_bfloat16 *y = static_cast<__nv_bfloat16 *>(W.y);
    y[at] = __float2bfloat16_rn((epilogue & kEpilogueAdd) ? val + __bfloat162float(y[at]) : val);
  }
}
__device__ __forceinline__ void a16_store_swiglu(const A16Weight &W, size_t at, float acc_g, float acc_u, float coef) {
  const float g = acc_g * coef, u = acc_u * coef;
  static_cast<__nv_bfloat16 *>(W.y)[at] = __float2bfloat16_rn(g / (1.0f + __expf(-g)) * u);
}

// TILES: row tiles per CTA (a fused SwiGLU has two: gate rows and their up rows).
template <int TILES>
__global__ void __launch_bounds__(kA16Threads, 1) nvfp4_a16_mma_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                    const __grid_constant__ A16Maps maps,
                                                                    const __grid_constant__ A16Params p) {
  constexpr uint32_t kTileSetBytes = TILES * kABytes, kRawBytes = TILES * kRawTileBytes;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw);
  const uint32_t x_bytes = p.bn * 128u;                       // one stage of activations
  // rings: decoded weights [a_stages], activations [x_stages], packed weights [raws]; each with its full and empty barriers
  const uint32_t x_ring = base + p.a_stages * kTileSetBytes, raw_ring = x_ring + p.x_stages * x_bytes, bars = raw_ring + p.raws * kRawBytes;
  const uint32_t bar_a = bars, bar_a_empty = bar_a + 8u * p.a_stages, bar_x = bar_a_empty + 8u * p.a_stages, bar_x_empty = bar_x + 8u * p.x_stages,
                 bar_raw = bar_x_empty + 8u * p.x_stages, bar_raw_empty = bar_raw + 8u * p.raws, bar_acc = bar_raw_empty + 8u * p.raws;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base_ptr + (bar_acc - base) + 8u);
  // The groups of decoder warps at work on a tile. One skips per_tile - 1 stages between two of its own: more of them than
  // the ring has stages would let it come to a slot with two uses outstanding, which one parity cannot tell from none.
  const uint32_t per_tile = TILES == 2 || p.a_stages < static_cast<uint32_t>(kGroups) ? 2u : static_cast<uint32_t>(kGroups);
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

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < p.a_stages; ++s) {
      mbar_init(bar_a + 8 * s, 4 * TILES);      // the four decoder warps of each tile
      mbar_init(bar_a_empty + 8 * s, 1);        // the MMA warp's commit
    }
    for (uint32_t s = 0; s < p.x_stages; ++s) {
      mbar_init(bar_x + 8 * s, 1);              // the producer's expect_tx arrival
      mbar_init(bar_x_empty + 8 * s, 1);
    }
    for (uint32_t d = 0; d < p.raws; ++d) {
      mbar_init(bar_raw + 8 * d, 1);
      mbar_init(bar_raw_empty + 8 * d, 4u * TILES * per_tile);   // every decoder warp at work
    }
    mbar_init(bar_acc, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kDecoders + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);

  if (warp < kDecoders) {
    // ---- row threads: the groups of a tile decode its stages in turn ----
    const uint32_t r = threadIdx.x & 127u, group = static_cast<uint32_t>(warp) / 4u;
    const uint32_t tile = TILES == 2 ? group & 1u : 0u, g = TILES == 2 ? group >> 1 : group;
    const uint32_t row_off = tile * kABytes + (r >> 3) * 1024u + (r & 7u) * 128u, sw = r & 7u;
    const uint32_t code_off = tile * kRawTileBytes + r * 128u, scale_off = tile * kRawTileBytes + kRawCodes + (r & 31u) * 16u + (r >> 5) * 4u;
    griddep_launch_dependents();
    griddep_wait();   // the epilogue reads and writes what the previous kernels may use
    RingAt at, from;
    at.advance(g, p.a_stages);
    for (uint32_t it = g; g < per_tile && it < stages; it += per_tile, at.advance(per_tile, p.a_stages)) {
      const uint32_t j = it & 3u, raw_at = raw_ring + from.slot * kRawBytes;   // stage j of its quad
      if (!mbar_wait(bar_raw + 8 * from.slot, from.phase) || !mbar_wait(bar_a_empty + 8 * at.slot, at.phase ^ 1u)) {
        if (lane == 0) atomicOr(&g_a16_status, kDecodeTimeout);
        break;
      }
      CodeStage st;
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(st.c[4 * h]), "=r"(st.c[4 * h + 1]), "=r"(st.c[4 * h + 2]), "=r"(st.c[4 * h + 3])
                     : "r"(raw_at + code_off + (((2u * j + h) ^ sw) << 4)));
      }
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(st.sc) : "r"(raw_at + scale_off + j * 512u));
      widen_row(st, base + at.slot * kTileSetBytes + row_off, sw);
      // the tile is read by the tensor core (async proxy): order these writes before it
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      const bool quad_done = j + per_tile >= 4u;   // the group's last stage of the quad
      if (lane == 0) {
        mbar_arrive(bar_a + 8 * at.slot);
        if (quad_done) mbar_arrive(bar_raw_empty + 8 * from.slot);
      }
      if (quad_done) from.advance(1u, p.raws);
    }
  } else if (warp == kDecoders) {
    // ---- producer of the activation tiles ----
    griddep_launch_dependents();
    griddep_wait();   // the activations may come from the previous kernel
    RingAt at;
    for (uint32_t s = 0; s < stages; ++s, at.advance(1u, p.x_stages)) {
      if (!mbar_wait(bar_x_empty + 8 * at.slot, at.phase ^ 1u)) {
        if (lane == 0) atomicOr(&g_a16_status, kProducerTimeout);
        break;
      }
      if (elect_one()) {
        mbar_expect_tx(bar_x + 8 * at.slot, x_bytes);
        tma_load_2d(x_ring + at.slot * x_bytes, &map_x, bar_x + 8 * at.slot, static_cast<int32_t>((s0 + s) * 64u), static_cast<int32_t>(tok0));
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
    for (uint32_t q = q0; q < q1; ++q, at.advance(1u, p.raws)) {
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
    const uint64_t a_desc0 = smem_desc_sw128(base), x_desc0 = smem_desc_sw128(x_ring);
    bool ok = true;
    RingAt at, xat;
    for (uint32_t it = 0; it < stages; ++it, at.advance(1u, p.a_stages), xat.advance(1u, p.x_stages)) {
      if (!mbar_wait(bar_x + 8 * xat.slot, xat.phase) || !mbar_wait(bar_a + 8 * at.slot, at.phase)) {
        if (lane == 0) atomicOr(&g_a16_status, kMmaTimeout);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint64_t a_desc = a_desc0 + at.slot * (kTileSetBytes >> 4), x_desc = x_desc0 + xat.slot * (x_bytes >> 4);
#pragma unroll
        for (uint32_t kb = 0; kb < 4; ++kb) {   // 16 values along K are 32 bytes: two 16-byte units further
          const uint32_t accumulate = (it | kb) != 0u ? 1u : 0u;
          mma_f16(tmem, a_desc + 2u * kb, x_desc + 2u * kb, idesc, accumulate);
          if (TILES == 2) mma_f16(tmem + p.acc_stride, a_desc + (kABytes >> 4) + 2u * kb, x_desc + 2u * kb, idesc, accumulate);
        }
        mma_commit(bar_a_empty + 8 * at.slot);
        mma_commit(bar_x_empty + 8 * xat.slot);
      }
      __syncwarp();
    }
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
  float *part = reinterpret_cast<float *>(base_ptr);   // [tile][token][128] partial sums, over the (by then idle) rings
  bool have = false;
  if (warp < kDecoders) {
    have = mbar_wait(bar_acc, 0u);
    if (!have && lane == 0) atomicOr(&g_a16_status, kEpilogueTimeout);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  auto store = [&](uint32_t token, float va, float vb) {
    const size_t at = static_cast<size_t>(token) * W.ldy;
    if (swiglu) {
      a16_store_swiglu(W, at + row_a, va, vb, coef);
    } else {
      a16_store(W, p.epilogue, at + row_a, va, coef);
      if (TILES == 2) a16_store(W, p.epilogue, at + row_b, vb, coef);
    }
  };
  if (kc == 1u) {
    if (warp < kDecoders && have) {
      for (uint32_t c = group * 16u; c < p.bn && tok0 + c < p.tokens; c += kGroups * 16u) {
        uint32_t v[16], u[16];
        tmem_ld16(lane_base + c, v);
        if (TILES == 2) tmem_ld16(lane_base + p.acc_stride + c, u);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (tok0 + c + j < p.tokens) store(tok0 + c + j, __uint_as_float(v[j]), TILES == 2 ? __uint_as_float(u[j]) : 0.0f);
        }
      }
    }
  } else {
    __syncthreads();   // every role is done with the rings: the partial sums take their place
    float *part_b = part + static_cast<size_t>(p.bn) * 128u;
    if (warp < kDecoders) {
      for (uint32_t c = group * 16u; c < p.bn; c += kGroups * 16u) {
        uint32_t v[16], u[16];
        if (have) {
          tmem_ld16(lane_base + c, v);
          if (TILES == 2) tmem_ld16(lane_base + p.acc_stride + c, u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          part[static_cast<size_t>(c + j) * 128u + r] = have ? __uint_as_float(v[j]) : 0.0f;
          if (TILES == 2) part_b[static_cast<size_t>(c + j) * 128u + r] = have ? __uint_as_float(u[j]) : 0.0f;
        }
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp < kDecoders) {
      // tokens dealt over the cluster's CTAs and their groups of warps; partial sums added in rank order
      for (uint32_t tl = kGroups * rank + group; tl < p.bn && tok0 + tl < p.tokens; tl += kGroups * kc) {
        float pa[8], pb[8];
#pragma unroll
        for (uint32_t q = 0; q < 8u; ++q) {   // requested together
          pa[q] = q < kc ? ld_cluster_f32(part + static_cast<size_t>(tl) * 128u + r, q) : 0.0f;
          pb[q] = TILES == 2 && q < kc ? ld_cluster_f32(part_b + static_cast<size_t>(tl) * 128u + r, q) : 0.0f;
        }
        float sum_a = pa[0], sum_b = pb[0];
#pragma unroll
        for (uint32_t q = 1; q < 8u; ++q) {
          if (q < kc) sum_a += pa[q], sum_b += pb[q];
        }
        store(tok0 + tl, sum_a, sum_b);
      }
    }
    __syncwarp();
    cluster_sync_all();   // no CTA leaves while a peer may still read its partial sums
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
  uint32_t tiles, bn, kc, a_stages, x_stages, raws, acc_stride, tmem_cols;
};

size_t a16_ring_bytes(const A16Plan &pl) {
  return static_cast<size_t>(pl.a_stages) * pl.tiles * kABytes + static_cast<size_t>(pl.x_stages) * pl.bn * 128u + static_cast<size_t>(pl.raws) * pl.tiles * kRawTileBytes;
}
size_t a16_smem_bytes(const A16Plan &pl) { return a16_ring_bytes(pl) + 16u * (pl.a_stages + pl.x_stages + pl.raws) + 32u + 1024u; }

// Ring depths: two of each at least, then in turn packed weights (what is in flight there hides the
// latency of HBM), activations and decoded tiles, up to 4, 8 and 4.
bool a16_rings(A16Plan &pl) {
  pl.a_stages = pl.x_stages = pl.raws = 2u;
  if (a16_smem_bytes(pl) > kA16MaxSmem) return false;
  auto grow = [&](uint32_t &depth, uint32_t most) {
    if (depth >= most) return false;
    ++depth;
    if (a16_smem_bytes(pl) <= kA16MaxSmem) return true;
    --depth;
    return false;
  };
  for (bool grew = true; grew;) {
    grew = grow(pl.a_stages, 4u);
    grew = grow(pl.x_stages, 8u) || grew;
    grew = grow(pl.raws, 4u) || grew;
  }
  return true;
}

// The shape of a CTA for `row_tiles` tiles of 128 rows (of a SwiGLU: gate tiles): the one that costs least in
// waves of CTAs. A stage costs the slowest of the tensor core (2 bn cycles a tile), the decoder warps (about
// 220 cycles a tile), what the CTA brings from the L2 (128 bytes a token and 4.6 KB a tile at about 42 bytes a
// cycle) and some 450 cycles of barrier round trips; a CTA has a fixed part besides (fill, drain and epilogue, some
// 2 us), the epilogue's stores and, with a K split, the exchange. So few tokens take one tile, K split until the
// device is full, and many take two tiles on a shared token tile, which halves what the L2 has to bring per FLOP.
A16Plan a16_plan(const DeviceState &dev, uint32_t row_tiles, uint32_t k_stages, uint32_t tokens, bool swiglu, bool even) {
  A16Plan best = {};
  double best_cost = 1e30;
  for (uint32_t tiles = swiglu ? 2u : 1u; tiles <= (swiglu || even ? 2u : 1u); ++tiles) {
    const uint32_t nt_min = (tokens + 255u) / 256u;
    for (uint32_t nt = nt_min; nt <= nt_min + nt_min / 2u + 4u; ++nt) {
      A16Plan pl = {};
      pl.tiles = tiles;
      pl.bn = ((tokens + nt - 1u) / nt + 15u) / 16u * 16u;
      if (nt > nt_min && pl.bn < 64u) break;
      if (!a16_rings(pl)) continue;
      pl.acc_stride = 32u;
      while (pl.acc_stride < pl.bn) pl.acc_stride <<= 1;
      pl.tmem_cols = tiles * pl.acc_stride;
      const uint32_t token_tiles = (tokens + pl.bn - 1u) / pl.bn, blocks = tiles == 2u && !swiglu ? row_tiles / 2u : row_tiles;
      for (uint32_t kc = 1; kc <= 8u; ++kc) {
        if (kc > 1u && (k_stages / kc < 8u || static_cast<size_t>(tiles) * pl.bn * 512u > a16_ring_bytes(pl))) break;
        const double ctas = static_cast<double>(blocks) * token_tiles * kc, sms = dev.sm_count;
        const double waves = ceil(ctas / (kc <= 2u ? sms : sms * (kc <= 4u ? 0.95 : 0.85)));   // wide clusters leave some SMs out
        double stage = tiles * 2.0 * (pl.bn < 64u ? 64.0 : pl.bn);
        const double load = (pl.bn * 128.0 + tiles * 4608.0) / 42.0;
        for (const double limit : {load, tiles * 220.0, 450.0}) stage = stage > limit ? stage : limit;
        const double cost = waves * (ceil(static_cast<double>(k_stages) / kc) * (stage + 50.0) + 3500.0 + tiles * 4.0 * pl.bn +
                                     (kc > 1u ? 1500.0 + 60.0 * kc + tiles * 4.0 * pl.bn : 0.0));
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
  cudaError_t err = cudaFuncSetAttribute(nvfp4_a16_mma_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kA16MaxSmem));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(nvfp4_a16_mma_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kA16MaxSmem));
  if (err != cudaSuccess) return fail(slot, "nvfp4 A16 tensor-core kernel attributes: %s", cudaGetErrorString(err));
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
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
  p.a_stages = pl.a_stages;
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
  const cudaError_t err = pl.tiles == 2u ? cudaLaunchKernelEx(&config, nvfp4_a16_mma_kernel<2>, map_x, maps, p) : cudaLaunchKernelEx(&config, nvfp4_a16_mma_kernel<1>, map_x, maps, p);
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
