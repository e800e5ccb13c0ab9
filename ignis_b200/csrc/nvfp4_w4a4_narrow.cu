// NVFP4 W4A4 products of calls with few tokens - from 33 to some hundreds, by the weights' sizes: the rule and what both
// kernels measured stand at narrow_is_cheaper, nvfp4_w4a4.cu - over activations already quantized in the operand
// layout (nvfp4_w4a4.cu's quantizer): out[t][r] = bf16(alpha * sum_k E2M1(a) E4M3(sa) E2M1(w) E4M3(sw)).
// The pair GEMM's 256 x 256 tiles leave most of the device idle there - 20 tiles for a 5120-row weight
// on 74 CTA pairs, each walking all of K - while the weights still bound the call: 48 to 100 MB of them.
//
//  * The weights are the MMA's A operand: a CTA owns 128 weight rows (M) and up to 128 tokens (N, as few as the
//    call has, in steps of 16) and walks a slice of K in stages of 256 values; the CTAs of a cluster
//    split K, so that narrow weights fill the device too. Each pushes its sums (st.async) to the CTA
//    that finishes the token, which adds them in rank order: nothing waits for a remote read's round
//    trip, and no CTA waits for the others' ends. Four tokens of a row go in one store: a layer at 33 / 77 / 128
//    tokens takes 56.1 / 67.7 / 79.3 us, 58.1 / 71.0 / 83.8 where the finishing CTA reads its peers' sums, and
//    58.9 / 73.4 / 86.9 with one token a store.
//  * Warp 8 brings a stage's weight codes and token codes by TMA (128-byte swizzle) and their scale tiles by
//    bulk copies; the weights' first stages are requested before the wait for the kernel that quantizes.
//  * Warp 9 owns tensor memory, copies a stage's scale tiles there and issues its MMAs, in the pipe's order, from
//    an elected lane.
//  * Warps 0-7 pull the accumulator: a lane is a weight row, so a warp's stores are 32 neighbouring outputs.
//  * The fused SwiGLU (a gate|up parent) pairs 128 gate rows with their up rows on one token tile, two
//    accumulators; with kEpilogueQuant the tile's h goes through shared memory into the next product's operand,
//    quantized by the standalone quantizer's rule.
//  * Every mbarrier wait is bounded; one that runs out sets a bit of the workspace's status word.
#include "nvfp4_internal.cuh"
#include "nvfp4_tc.cuh"

#include <cmath>

namespace b200q {
namespace {

constexpr uint32_t kABytes = 128 * 128;    // one stage of a tile's codes: 128 rows x 256 values
constexpr uint32_t kSfBytes = 4 * 512;     // one stage of the scales of 128 rows: four K-atoms
constexpr int kEpiWarps = 8;
constexpr int kNarrowThreads = (kEpiWarps + 2) * 32;
constexpr uint32_t kProducerTimeout = 1u, kMmaTimeout = 2u, kEpilogueTimeout = 4u;   // the pair GEMM's bits

struct NarrowWeight {
  const uint8_t *scales;
  void *y;
  uint32_t n, ldy;
  float alpha;            // 1 / (d_in d_w)
  uint32_t block_begin;   // first CTA of this weight
};
struct NarrowMaps {
  CUtensorMap w[kMaxGroup];   // the weights' code planes
  CUtensorMap x;              // the tokens' codes
};
struct NarrowParams {
  NarrowWeight w[kMaxGroup];
  const uint8_t *sfx;    // the tokens' scale tiles
  uint32_t *status;
  uint32_t count, k, tokens;
  uint32_t tile;         // tokens per CTA: a multiple of 16 up to 128
  uint32_t stages, kc, tmem_cols;
  uint32_t acc_stride;   // tensor-memory columns from the first accumulator to the second
  uint32_t epilogue;     // STORE / ADD / OUT_F32, the fused SwiGLU, or the fused SwiGLU quantized
  uint8_t *q_codes;      // kEpilogueQuant: h as the next product's operand
  uint8_t *q_scales;
  float q_din;
};


// Silu(g) u as the reference's formula rounds it: both products to BF16 first.
__device__ __forceinline__ __nv_bfloat16 swiglu_bf16(float acc_g, float acc_u, float alpha) {
  const float g = __bfloat162float(__float2bfloat16_rn(__fmul_rn(acc_g, alpha)));
  const float u = __bfloat162float(__float2bfloat16_rn(__fmul_rn(acc_u, alpha)));
  return __float2bfloat16_rn(g / (1.0f + __expf(-g)) * u);
}

// TILES: row tiles per CTA (2: a SwiGLU's gate rows and up rows).
template <int TILES>
__global__ void __launch_bounds__(kNarrowThreads, 2) w4a4_narrow_kernel(const __grid_constant__ NarrowMaps maps, const __grid_constant__ NarrowParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw);
  const uint32_t x_bytes = p.tile * 128u;
  // a stage: weight codes [TILES] | token codes | weight scales [TILES] | token scales
  const uint32_t sf_off = TILES * kABytes + x_bytes;
  const uint32_t stage_bytes = sf_off + (TILES + 1) * kSfBytes, stage_pitch = (stage_bytes + 1023u) & ~1023u;
  const uint32_t bars = base + p.stages * stage_pitch;   // full[stages], empty[stages], accumulator full, sums here; then the TMEM slot
  const uint32_t bar_empty = bars + 8u * p.stages, bar_acc = bar_empty + 8u * p.stages, bar_sums = bar_acc + 8u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base_ptr + (bar_acc - base) + 16u);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), kc = p.kc;

  // Without a K split the grid is walked token tile first: the CTAs at work at one time share weight rows.
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
  const NarrowWeight &W = p.w[wi];
  const uint32_t block = (bx - W.block_begin) / kc;   // 128-row tile of the output
  const uint32_t row_a = block * 128u, row_b = W.n / 2u + row_a;
  const uint32_t k_stages = p.k / 256u, k_atoms = p.k / 64u;
  const uint32_t s0 = static_cast<uint32_t>(static_cast<uint64_t>(k_stages) * rank / kc);
  const uint32_t s1 = static_cast<uint32_t>(static_cast<uint64_t>(k_stages) * (rank + 1) / kc);
  const uint32_t tok0 = by * p.tile;
  const uint32_t live = min(p.tokens - tok0, p.tile), mma_n = (live + 15u) / 16u * 16u;   // tokens the MMA computes

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < p.stages; ++s) {
      mbar_init(bars + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_acc, 1);
    mbar_init(bar_sums, 1);
    if (kc > 1u) {   // quads of tokens are dealt over the ranks; every rank pushes its sums of this one's
      const uint32_t quads = (live + 3u) / 4u;
      mbar_expect_tx(bar_sums, (quads + kc - 1u - rank) / kc * kc * TILES * 2048u);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
  const uint32_t sf_cols0 = tmem + TILES * p.acc_stride;   // scale columns behind the accumulators

  griddep_launch_dependents();
  if (warp == kEpiWarps) {
    // ---- producer ----
    const uint64_t policy = l2_evict_first_policy();
    const bool once = gridDim.y == 1u;   // several token tiles read the same weights: leave them in the L2
    const CUtensorMap *map_w = &maps.w[wi];
    const uint8_t *sfw_a = W.scales + static_cast<size_t>(row_a / 128u) * k_atoms * 512u;
    const uint8_t *sfw_b = W.scales + static_cast<size_t>(row_b / 128u) * k_atoms * 512u;
    const uint8_t *sfx = p.sfx + static_cast<size_t>(tok0 / 128u) * k_atoms * 512u;
    auto weights = [&](uint32_t s, uint32_t slot) {
      const uint32_t full = bars + 8 * slot, stage = base + slot * stage_pitch;
      mbar_expect_tx(full, stage_bytes);
#pragma unroll
      for (int t = 0; t < TILES; ++t) {
        const int32_t row = static_cast<int32_t>(t == 0 ? row_a : row_b);
        if (once) tma_load_2d_hint(stage + t * kABytes, map_w, full, static_cast<int32_t>(s * 128u), row, policy);
        else tma_load_2d(stage + t * kABytes, map_w, full, static_cast<int32_t>(s * 128u), row);
        bulk_load(stage + sf_off + t * kSfBytes, (t == 0 ? sfw_a : sfw_b) + static_cast<size_t>(s) * kSfBytes, kSfBytes, full);
      }
    };
    auto tokens = [&](uint32_t s, uint32_t slot) {
      const uint32_t full = bars + 8 * slot, stage = base + slot * stage_pitch;
      tma_load_2d(stage + TILES * kABytes, &maps.x, full, static_cast<int32_t>(s * 128u), static_cast<int32_t>(tok0));
      bulk_load(stage + sf_off + TILES * kSfBytes, sfx + static_cast<size_t>(s) * kSfBytes, kSfBytes, full);
    };
    // the weights never depend on the previous kernel, the tokens come from it
    const uint32_t ahead = min(p.stages, s1 - s0);
    if (elect_one()) {
      for (uint32_t s = 0; s < ahead; ++s) weights(s0 + s, s);
    }
    __syncwarp();
    griddep_wait();
    if (elect_one()) {
      for (uint32_t s = 0; s < ahead; ++s) tokens(s0 + s, s);
    }
    __syncwarp();
    RingAt at;
    at.advance(ahead, p.stages);
    for (uint32_t s = s0 + ahead; s < s1; ++s, at.advance(1u, p.stages)) {
      if (!mbar_wait(bar_empty + 8 * at.slot, at.phase ^ 1u)) {
        if (lane == 0) atomicOr(p.status, kProducerTimeout);
        break;
      }
      if (elect_one()) {
        weights(s, at.slot);
        tokens(s, at.slot);
      }
      __syncwarp();
    }
  } else if (warp == kEpiWarps + 1) {
    // ---- scale copies and MMAs ----
    // E2M1 x E2M1 (format 1 at bits 7 and 10), both K-major, N >> 3 at bit 17, UE4M3 scales, M >> 4 at bit 24
    const uint32_t idesc = (1u << 7) | (1u << 10) | ((mma_n >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t desc0 = smem_desc(base, 1024u, 2u), sf_desc0 = smem_desc(base + sf_off, 128u, 0u);
    const uint32_t pitch = stage_pitch >> 4, buf_cols = (TILES + 1) * 16u;
    bool ok = true;
    RingAt at;
    for (uint32_t it = 0; it < s1 - s0; ++it, at.advance(1u, p.stages)) {
      if (!mbar_wait(bars + 8 * at.slot, at.phase)) {
        if (lane == 0) atomicOr(p.status, kMmaTimeout);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint32_t sfw_cols = sf_cols0 + (it & 1u) * buf_cols, sfx_cols = sfw_cols + TILES * 16u;
        const uint64_t sf = sf_desc0 + at.slot * pitch;
#pragma unroll
        for (uint32_t kb = 0; kb < 4; ++kb) {
#pragma unroll
          for (uint32_t t = 0; t < TILES; ++t) tmem_cp_sf(sfw_cols + t * 16u + kb * 4u, sf + t * (kSfBytes >> 4) + kb * 32u);
          tmem_cp_sf(sfx_cols + kb * 4u, sf + TILES * (kSfBytes >> 4) + kb * 32u);
        }
        const uint64_t a_desc = desc0 + at.slot * pitch, b_desc = a_desc + TILES * (kABytes >> 4);
#pragma unroll
        for (uint32_t kb = 0; kb < 4; ++kb) {   // 64 values along K are 32 bytes: two 16-byte units further
#pragma unroll
          for (uint32_t t = 0; t < TILES; ++t) {
            mma_mxf4nvf4(tmem + t * p.acc_stride, a_desc + t * (kABytes >> 4) + 2u * kb, b_desc + 2u * kb, idesc, sfw_cols + t * 16u + kb * 4u,
                         sfx_cols + kb * 4u, (it | kb) != 0u ? 1u : 0u);
          }
        }
        mma_commit(bar_empty + 8 * at.slot);
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar_acc);
    __syncwarp();
  }

  // ---- epilogue: warp w owns accumulator lanes (tile rows) 32 (w % 4) .. + 31; the two groups of four warps take the
  //      chunks of 16 tokens in turn ----
  const uint32_t quad = static_cast<uint32_t>(warp) & 3u, group = static_cast<uint32_t>(warp) >> 2;
  const uint32_t r = quad * 32u + static_cast<uint32_t>(lane), row = row_a + r;
  const uint32_t lane_base = tmem + ((quad * 32u) << 16);
  const bool quantize = TILES == 2 && (p.epilogue & kEpilogueQuant) != 0u;
  // Over the (by then idle) ring: partial sums of this rank's tokens, [source rank][turn][tile][row 128][token 4]; behind
  // them h of the quantized form, [token][row 128].
  const uint32_t turns = (p.tile / 4u + kc - 1u) / kc;
  __nv_bfloat16 *h_tile = reinterpret_cast<__nv_bfloat16 *>(base_ptr + (kc > 1u ? kc * turns * TILES * 2048u : 0u));
  constexpr uint32_t kHPitch = 136;   // values: 16-byte rows, a quarter-warp's 16-byte reads on different banks
  bool have = false;
  if (warp < kEpiWarps) {
    griddep_wait();   // what this kernel writes, an earlier one may still read
    have = mbar_wait(bar_acc, 0u);
    if (!have && lane == 0) atomicOr(p.status, kEpilogueTimeout);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  // What the residual add finds in the output, as the stored type's bits: `n` tokens from `first` on (past the last one: the
  // last), requested together before any of them is needed. One at a time, each with its own branches, they are round trips
  // one after another.
  const bool add = TILES == 1 && (p.epilogue & kEpilogueAdd) != 0u, f32 = (p.epilogue & kEpilogueF32) != 0u;
  auto request = [&](auto &bits, uint32_t first) {
    if (!add) return;
    constexpr uint32_t n = sizeof(bits) / 4u;
    if (f32) {
#pragma unroll
      for (uint32_t j = 0; j < n; ++j) bits[j] = static_cast<const uint32_t *>(W.y)[static_cast<size_t>(tok0 + min(first + j, live - 1u)) * W.ldy + row];
    } else {
#pragma unroll
      for (uint32_t j = 0; j < n; ++j) bits[j] = static_cast<const uint16_t *>(W.y)[static_cast<size_t>(tok0 + min(first + j, live - 1u)) * W.ldy + row];
    }
  };
  auto emit = [&](uint32_t tl, float va, float vb, uint32_t bits) {   // token tl of the tile
    if (quantize) {
      h_tile[tl * kHPitch + r] = swiglu_bf16(va, vb, W.alpha);
      return;
    }
    const size_t at = static_cast<size_t>(tok0 + tl) * W.ldy + row;
    if (TILES == 2) {
      static_cast<__nv_bfloat16 *>(W.y)[at] = swiglu_bf16(va, vb, W.alpha);
      return;
    }
    const float val = __fmul_rn(va, W.alpha);   // not contracted into the residual add: one value for every epilogue
    const float old = __uint_as_float(f32 ? bits : bits << 16);
    if (f32) {
      static_cast<float *>(W.y)[at] = add ? old + val : val;
    } else {
      static_cast<__nv_bfloat16 *>(W.y)[at] = __float2bfloat16_rn(add ? val + old : val);
    }
  };
  if (kc == 1u) {
    if (warp < kEpiWarps && have) {
      for (uint32_t c = group * 16u; c < live; c += 32u) {
        uint32_t v[16], u[16];
        uint32_t old[16] = {};
        tmem_ld16(lane_base + c, v);
        if (TILES == 2) tmem_ld16(lane_base + p.acc_stride + c, u);
        request(old, c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c + j < live) emit(c + j, __uint_as_float(v[j]), TILES == 2 ? __uint_as_float(u[j]) : 0.0f, old[j]);
        }
      }
    }
  } else {
    uint32_t old[4] = {};   // a quad's, requested before its sums are here
    if (warp < kEpiWarps) request(old, 4u * (group * kc + rank));
    __syncwarp();
    cluster_sync_all();   // every role of every rank is done with its ring
    if (warp < kEpiWarps) {
      for (uint32_t c = group * 16u; c < live; c += 32u) {
        uint32_t v[16], u[16];
        if (have) {
          tmem_ld16(lane_base + c, v);
          if (TILES == 2) tmem_ld16(lane_base + p.acc_stride + c, u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        uint32_t to = (c >> 2) % kc, turn = (c >> 2) / kc;
#pragma unroll
        for (uint32_t j = 0; j < 16u; j += 4u) {
          if (c + j >= live) break;
          const uint32_t at = base + ((rank * turns + turn) * TILES * 128u + r) * 16u, bar = cluster_map(bar_sums, to);
          auto sums4 = [&](const uint32_t (&w)[16]) {
            return have ? make_float4(__uint_as_float(w[j]), __uint_as_float(w[j + 1u]), __uint_as_float(w[j + 2u]), __uint_as_float(w[j + 3u]))
                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          };
          push_f32x4(cluster_map(at, to), sums4(v), bar);
          if (TILES == 2) push_f32x4(cluster_map(at + 2048u, to), sums4(u), bar);
          if (++to == kc) to = 0u, ++turn;
        }
      }
      // the rank's quads, every other one to a group of warps; partial sums added in rank order
      const float4 *sums = reinterpret_cast<const float4 *>(base_ptr) + r;
      if (mbar_wait_pushed(bar_sums)) {
        for (uint32_t turn = group; 4u * (turn * kc + rank) < live; turn += 2u) {
          if (turn != group) request(old, 4u * (turn * kc + rank));
          const float4 *from = sums + turn * TILES * 128u;
          float4 sum_a = from[0], sum_b = TILES == 2 ? from[128] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          for (uint32_t q = 1; q < kc; ++q) {
            from += turns * TILES * 128u;
            const float4 more = from[0];
            sum_a.x += more.x, sum_a.y += more.y, sum_a.z += more.z, sum_a.w += more.w;
            if (TILES == 2) {
              const float4 more_b = from[128];
              sum_b.x += more_b.x, sum_b.y += more_b.y, sum_b.z += more_b.z, sum_b.w += more_b.w;
            }
          }
          const uint32_t tl = 4u * (turn * kc + rank);
          emit(tl, sum_a.x, sum_b.x, old[0]);
          if (tl + 1u < live) emit(tl + 1u, sum_a.y, sum_b.y, old[1]);
          if (tl + 2u < live) emit(tl + 2u, sum_a.z, sum_b.z, old[2]);
          if (tl + 3u < live) emit(tl + 3u, sum_a.w, sum_b.w, old[3]);
        }
      } else if (lane == 0) {
        atomicOr(p.status, kEpilogueTimeout);
      }
    }
    __syncwarp();
  }
  if (quantize) {
    // This CTA's tokens of h, in blocks of 16 along the next product's K (this tile's 128 rows are 8 blocks), quantized as
    // the standalone quantizer would from the BF16 values. Columns past the call's tokens are never read as outputs.
    __syncthreads();
    const uint32_t inter = W.n / 2u;
    const uint32_t mine = kc == 1u ? live : turns * 4u;   // an upper bound of this CTA's tokens
    for (uint32_t i = threadIdx.x; i < mine * 8u; i += kNarrowThreads) {
      const uint32_t j = i >> 3, b = i & 7u;
      const uint32_t tl = kc == 1u ? j : ((j >> 2) * kc + rank) * 4u + (j & 3u);
      if (tl >= live) continue;
      const uint4 *src = reinterpret_cast<const uint4 *>(h_tile + tl * kHPitch + b * 16u);
      uint2 codes;
      uint8_t scale;
      quantize_block16(src[0], src[1], p.q_din, codes, scale);
      const uint32_t token = tok0 + tl, col = row_a + b * 16u, g = col / 16u;
      *reinterpret_cast<uint2 *>(p.q_codes + static_cast<size_t>(token) * (inter / 2u) + col / 2u) = codes;
      p.q_scales[(static_cast<size_t>(token >> 7) * (inter / 64u) + (g >> 2)) * 512u + (token & 31u) * 16u + ((token & 127u) >> 5) * 4u + (g & 3u)] = scale;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kEpiWarps + 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

// ---- host side --------------------------------------------------------------------------------
constexpr size_t kNarrowMaxSmem = 222 * 1024;

struct NarrowPlan {
  uint32_t tiles, tile, kc, stages, acc_stride, tmem_cols;
};

uint32_t narrow_pitch(const NarrowPlan &pl) { return (pl.tiles * (kABytes + kSfBytes) + pl.tile * 128u + kSfBytes + 1023u) & ~1023u; }
size_t narrow_smem(const NarrowPlan &pl) { return static_cast<size_t>(pl.stages) * narrow_pitch(pl) + 16u * pl.stages + 32u + 1024u; }

// One CTA per SM with as deep a ring as fits (two with half the ring each: 80 us against 72 a layer at 77 tokens), K split
// while the CTAs still run as one wave and a CTA keeps four stages.
NarrowPlan narrow_plan(const DeviceState &dev, uint32_t row_tiles, uint32_t k_stages, uint32_t tokens, bool swiglu) {
  NarrowPlan pl = {};
  pl.tiles = swiglu ? 2u : 1u;
  pl.tile = tokens <= 128u ? (tokens + 15u) / 16u * 16u : 128u;   // several token tiles start on whole scale tiles
  pl.acc_stride = (pl.tile + 31u) / 32u * 32u;
  pl.tmem_cols = 64u;
  while (pl.tmem_cols < pl.tiles * pl.acc_stride + 2u * (pl.tiles + 1u) * 16u) pl.tmem_cols <<= 1;   // two stages of scales behind the accumulators
  const uint32_t blocks = row_tiles * ((tokens + pl.tile - 1u) / pl.tile), sms = static_cast<uint32_t>(dev.sm_count);
  pl.kc = 1;
  // clusters are placed inside one GPC: wide ones leave some SMs out
  while (pl.kc < 8u && blocks * (pl.kc + 1u) <= (pl.kc + 1u <= 4u ? sms : sms * 7u / 8u) && k_stages / (pl.kc + 1u) >= 4u) ++pl.kc;
  for (pl.stages = 8u; narrow_smem(pl) > kNarrowMaxSmem;) --pl.stages;
  return pl;
}

// Bytes behind the ring's start that the epilogue needs.
size_t narrow_epilogue_bytes(const NarrowPlan &pl, bool quant) {
  return (pl.kc > 1u ? static_cast<size_t>(pl.kc) * ((pl.tile / 4u + pl.kc - 1u) / pl.kc) * pl.tiles * 2048u : 0u) + (quant ? static_cast<size_t>(pl.tile) * 272u : 0u);
}

}  // namespace

int32_t w4a4_narrow_prepare(ErrorSlot &slot) {
  cudaError_t err = cudaFuncSetAttribute(w4a4_narrow_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kNarrowMaxSmem));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(w4a4_narrow_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kNarrowMaxSmem));
  if (err != cudaSuccess) return fail(slot, "nvfp4 W4A4 narrow kernel attributes: %s", cudaGetErrorString(err));
  return 0;
}

double w4a4_narrow_cycles(const DeviceState &dev, uint32_t row_tiles, uint32_t k, uint32_t tokens, bool swiglu) {
  const uint32_t k_stages = k / 256u;
  const NarrowPlan pl = narrow_plan(dev, row_tiles, k_stages, tokens, swiglu);
  const double ctas = static_cast<double>(row_tiles) * ((tokens + pl.tile - 1u) / pl.tile) * pl.kc;
  // What an SM brings from the L2 in a cycle: 42 bytes when all of them pull, up to 64 when fewer do (5120 x 17408 at 160 and 320
  // tokens, 80 and 120 CTAs: 27.3 and 29.7 us). The waves of a gate|up parent beyond the first: 28 (20 us each at 34816 x 5120).
  const double share = 42.0 * dev.sm_count / (ctas < dev.sm_count ? ctas : dev.sm_count);
  const double stage = narrow_pitch(pl) / (swiglu && ctas > dev.sm_count ? 28.0 : share < 64.0 ? share : 64.0);
  const double walk = ceil(ctas / dev.sm_count) * (ceil(static_cast<double>(k_stages) / pl.kc) * (stage > 350.0 ? stage : 350.0) + 4000.0 + (pl.kc > 1u ? 2000.0 : 0.0));
  const double stream = row_tiles * pl.tiles * 72.0 * k / 3150.0;   // the weights at the rate of HBM, per cycle of 1.9 GHz
  return 4000.0 + (walk > stream ? walk : stream);
}

int32_t w4a4_narrow_launch(ErrorSlot &slot, const DeviceState &dev, const A4Item *items, uint32_t count, uint32_t k, uint32_t tokens,
                           uint32_t epilogue, const uint8_t *x_codes, const uint8_t *x_scales, uint32_t *status, uint8_t *q_codes,
                           uint8_t *q_scales, float q_din, cudaStream_t stream) {
  const bool swiglu = (epilogue & kEpilogueSwiglu) != 0u, quant = (epilogue & kEpilogueQuant) != 0u;
  uint32_t row_tiles = 0;
  for (uint32_t i = 0; i < count; ++i) row_tiles += items[i].n / (swiglu ? 256u : 128u);
  const NarrowPlan pl = narrow_plan(dev, row_tiles, k / 256u, tokens, swiglu);
  NarrowParams p = {};
  NarrowMaps maps = {};
  p.sfx = x_scales;
  p.status = status;
  p.count = count;
  p.k = k;
  p.tokens = tokens;
  p.tile = pl.tile;
  p.stages = pl.stages;
  p.kc = pl.kc;
  p.tmem_cols = pl.tmem_cols;
  p.acc_stride = pl.acc_stride;
  p.epilogue = epilogue;
  p.q_codes = q_codes;
  p.q_scales = q_scales;
  p.q_din = q_din;
  uint32_t ctas = 0;
  bool encoded = make_code_map(&maps.x, x_codes, (static_cast<uint64_t>(tokens) + 127u) / 128u * 128u, k / 2u, pl.tile);
  for (uint32_t i = 0; i < count; ++i) {
    NarrowWeight &g = p.w[i];
    g.scales = items[i].scales;
    g.y = items[i].y;
    g.n = items[i].n;
    g.ldy = items[i].ldy;
    g.alpha = 1.0f / (items[i].d_in * items[i].d_w);
    g.block_begin = ctas;
    ctas += items[i].n / (swiglu ? 256u : 128u) * pl.kc;
    encoded = encoded && make_code_map(&maps.w[i], items[i].codes, items[i].n, k / 2u, 128u);
  }
  if (!encoded) return fail(slot, "nvfp4 W4A4 narrow route: tensor map encoding failed");
  const size_t ring = narrow_smem(pl), need = narrow_epilogue_bytes(pl, quant) + 1024u;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(ctas, (tokens + pl.tile - 1u) / pl.tile, 1);
  config.blockDim = dim3(kNarrowThreads, 1, 1);
  config.dynamicSmemBytes = ring > need ? ring : need;
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
  const cudaError_t err = swiglu ? cudaLaunchKernelEx(&config, w4a4_narrow_kernel<2>, maps, p) : cudaLaunchKernelEx(&config, w4a4_narrow_kernel<1>, maps, p);
  if (err != cudaSuccess) return fail(slot, "nvfp4 W4A4 narrow launch: %s", cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q
