// NVFP4 W4A4 at decode and verify widths (up to 32 tokens): out[t][r] = bf16(alpha * sum_k
// E2M1(a) E4M3(sa) E2M1(w) E4M3(sw)), alpha = 1 / (d_in d_w), with the weights going from HBM to
// the tensor cores untouched. Stands where the reference, under its default AllowA4 policy, leaves
// the A16 kernels from 4 / 5 / 8 tokens and runs its FP4 MMA on quantized activations
// (kernel/vendor/src/ops/linear/nvfp4/nvfp4_dispatch.cpp:31-39, nvfp4_w4a4_mma.cuh:203-436); the
// design is not theirs.
//
//  * The weights are the MMA's A operand: a CTA owns 128 weight rows (M) and walks its slice of K
//    in stages of 256 values. A producer thread brings a stage's 16 KB of codes (TMA, 128-byte
//    swizzle, evict-first) and its four 512-byte scale tiles (a bulk copy) into a ring; nothing in
//    the SM ever decodes a weight.
//  * The tokens are the B operand (N = 16 or 32). Quantizer warps turn the stage's activations into
//    NVFP4 themselves - 16 values per item, bit for bit the rule of the prefill quantizer
//    (nvfp4_codec.cuh:81-110) - straight into the stage's swizzled B tile and its scale tile, so a
//    call needs no workspace, no second launch and no pass over global memory. Every CTA repeats
//    this for its K slice from the L2. The warps work in groups of four that take the stages in
//    turn, so a group has several stage times for its stage.
//  * The last warp owns tensor memory; per stage it copies the scale tiles of both operands to tensor memory
//    (tcgen05.cp) and issues four tcgen05.mma kind::mxf4nvf4 block_scale scale_vec::4X (M 128, N, K 64).
//  * The fused SwiGLU (a gate|up parent) pairs a tile's 128 gate rows with their up rows: per K
//    stage two ring entries, each with its own weight tile, sharing the first one's token tile,
//    into two accumulators; the epilogue writes BF16(silu(BF16(g alpha)) * BF16(u alpha)).
//  * Narrow weights split K over the CTAs of a cluster, which push their partial sums to the CTA that finishes a token,
//    where they are added in rank order (bit-reproducible, no global scratch).
//  * Every mbarrier wait is bounded; one that runs out sets a bit in the library's status word
//    (b200q_nvfp4_device_status), and the CTA falls through to the common exit and frees its
//    tensor memory.
#include "nvfp4_internal.cuh"
#include "nvfp4_tc.cuh"

namespace b200q {
namespace {

constexpr uint32_t kABytes = 128 * 128;   // one stage of weight codes: 128 rows x 256 values
constexpr uint32_t kSfBytes = 4 * 512;    // one stage of scales of a 128-row tile: four K-atoms
constexpr uint32_t kProducerTimeout = 0x100u, kMmaTimeout = 0x200u, kEpilogueTimeout = 0x400u, kQuantTimeout = 0x800u, kReduceTimeout = 0x1000u;
constexpr int kMaxQuantGroups = 2;
constexpr int kMaxItems = 4;              // 16-value items per quantizer thread and stage (32 tokens)

__device__ uint32_t g_a4_status = 0;

struct A4Weight {
  const uint8_t *scales;
  void *y;
  uint32_t n, ldy;
  float alpha;           // 1 / (d_in d_w)
  float d_in;
  uint32_t block_begin;  // first CTA of this weight
};

struct A4Maps {
  CUtensorMap m[kMaxGroup];  // the weights' code planes
};

struct A4Params {
  A4Weight w[kMaxGroup];
  const uint16_t *x;   // BF16 [tokens][k]
  uint32_t count;
  uint32_t k, tokens;
  uint32_t bn;         // token tile (MMA N): 16 or 32
  uint32_t stages;     // ring depth
  uint32_t pair;       // plain products: 1 = a CTA owns two consecutive row tiles, which share the quantized token tile
  uint32_t groups;     // quantizer groups of 128 threads; then the producer warp and the MMA warp
  uint32_t kc;         // cluster size: K slices
  uint32_t tmem_cols;  // accumulators (64) + 32 scale columns per ring entry, rounded up to a power of two
  uint32_t epilogue;   // STORE / ADD / OUT_F32, or the fused SwiGLU
};

__device__ __forceinline__ void bulk_load_hint(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr)
               : "memory");
}

struct RawItem {
  uint4 lo, hi;  // 16 BF16 activations
};

template <int ITEMS>
__global__ void __launch_bounds__(64 + 128 * kMaxQuantGroups, 2) w4a4_decode_kernel(const __grid_constant__ A4Maps maps, const __grid_constant__ A4Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - raw);
  // a stage: weight codes | token codes | weight scale tiles | token scale tiles
  const uint32_t b_bytes = p.bn * 128u;
  const uint32_t stage_bytes = kABytes + b_bytes + 2u * kSfBytes;
  const uint32_t bars = base + p.stages * stage_bytes;  // full[stages], empty[stages], accumulator full, sums landed; then the TMEM slot
  const uint32_t bar_acc = bars + 8u * 2u * p.stages, bar_sums = bar_acc + 8u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base_ptr + (bar_sums - base) + 8u);
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int producer_warp = 4 * static_cast<int>(p.groups), mma_warp = producer_warp + 1;
  const uint32_t rank = cluster_ctarank(), kc = p.kc;

  uint32_t wi = 0;
#pragma unroll
  for (uint32_t i = 1; i < kMaxGroup; ++i) {
    if (i < p.count && blockIdx.x >= p.w[i].block_begin) wi = i;
  }
  const A4Weight &W = p.w[wi];
  const bool swiglu = (p.epilogue & kEpilogueSwiglu) != 0u;
  const bool two = swiglu || p.pair != 0u;
  const uint32_t halves = two ? 2u : 1u;   // ring entries per K stage: two weight tiles share a token tile
  const uint32_t m_tile = (blockIdx.x - W.block_begin) / kc;
  // first weight rows of the CTA's tiles: gate rows and their up rows (n / 2 further down), or two
  // consecutive tiles of a plain product, or one tile
  const uint32_t row_a = swiglu ? m_tile * 128u : m_tile * 128u * halves;
  const uint32_t row_b = swiglu ? W.n / 2u + m_tile * 128u : row_a + 128u;
  const uint32_t k_stages = p.k / 256u, k_atoms = p.k / 64u;
  const uint32_t s0 = static_cast<uint32_t>(static_cast<uint64_t>(k_stages) * rank / kc);
  const uint32_t s1 = static_cast<uint32_t>(static_cast<uint64_t>(k_stages) * (rank + 1) / kc);

  // One ring entry: a weight tile of K stage s0 + it / halves (entry 2 j is the first tile, 2 j + 1
  // the second when the CTA has two) and its scale tiles.
  const uint32_t entries = (s1 - s0) * halves;
  auto produce = [&](uint32_t it, uint32_t slot, uint64_t policy) {
    const uint32_t s = s0 + (two ? it >> 1 : it);
    const uint32_t row0 = two && (it & 1u) != 0u ? row_b : row_a;
    const uint32_t full = bars + 8 * slot;
    const uint32_t stage = base + slot * stage_bytes;
    mbar_expect_tx(full, kABytes + kSfBytes);
    tma_load_2d_hint(stage, &maps.m[wi], full, static_cast<int32_t>(s * 128u), static_cast<int32_t>(row0), policy);
    bulk_load_hint(stage + kABytes + b_bytes, W.scales + (static_cast<size_t>(row0 / 128u) * k_atoms + s * 4u) * 512u, kSfBytes, full,
                   policy);
  };
  // (Requesting the first ring of weight tiles from here, before tensor memory is allocated, was
  // measured slower: the early loads take bandwidth from the previous kernel's last CTAs, which
  // this kernel's quantizers wait for.)
  if (warp == producer_warp && lane == 0) {
    for (uint32_t s = 0; s < p.stages; ++s) {
      mbar_init(bars + 8 * s, 128 + 1);          // 128 quantizer threads and the producer's expect_tx arrival
      mbar_init(bars + 8 * (p.stages + s), 1);   // the MMA thread's commit
    }
    mbar_init(bar_acc, 1);
    mbar_init(bar_sums, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // every rank of the cluster sends its sums of the tokens that this one finishes
    if (kc > 1u) mbar_expect_tx(bar_sums, kc * ((p.tokens - rank + kc - 1u) / kc) * halves * 512u);
  }
  if (warp == mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp < 4) {
    // token rows past the call's tokens are never written again: zero codes and zero scales
    for (uint32_t s = 0; s < p.stages; ++s) {
      uint8_t *stage = base_ptr + s * stage_bytes;
      for (uint32_t i = threadIdx.x; i < b_bytes / 16u; i += 128u) reinterpret_cast<uint4 *>(stage + kABytes)[i] = make_uint4(0, 0, 0, 0);
      reinterpret_cast<uint4 *>(stage + kABytes + b_bytes + kSfBytes)[threadIdx.x] = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);

  if (warp < producer_warp) {
    // ---- quantizers: item i of a stage = token i / 16, values [16 (i % 16), +16) of the stage;
    //      group g takes the CTA's stages g, g + groups, ... ----
    griddep_launch_dependents();
    griddep_wait();   // the activations may come from the previous kernel
    // A thread's values of its group's next kDepth stages are requested together (stage by stage, the trip to the L2
    // came once per stage and held up the short K slices: 1.3 us each).
    constexpr int kDepth = kMaxItems / ITEMS;
    const uint32_t items = p.tokens * 16u;
    const uint32_t group = static_cast<uint32_t>(warp) >> 2, tid = threadIdx.x & 127u;
    const uint32_t first = s0 + group;
    uint32_t tok[ITEMS], grp[ITEMS];
    const uint16_t *src[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t i = tid + 128u * j;
      tok[j] = i >> 4;
      grp[j] = i & 15u;
      src[j] = p.x + static_cast<size_t>(tok[j]) * p.k + grp[j] * 16u;
    }
    RawItem cur[kDepth][ITEMS];
    auto request = [&](RawItem (&to)[ITEMS], uint32_t s) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (tid + 128u * j < items && s < s1) {
          to[j].lo = ldg128_coherent(src[j] + static_cast<size_t>(s) * 256u);
          to[j].hi = ldg128_coherent(src[j] + static_cast<size_t>(s) * 256u + 8);
        }
      }
    };
#pragma unroll
    for (int d = 0; d < kDepth; ++d) request(cur[d], first + d * p.groups);
    bool ok = true;
    for (uint32_t sd = first; sd < s1 && ok; sd += kDepth * p.groups) {
#pragma unroll
      for (int d = 0; d < kDepth; ++d) {
        const uint32_t s = sd + d * p.groups;
        if (s >= s1 || !ok) break;
        const uint32_t it = (s - s0) * halves;   // the stage's (first) ring entry
        uint2 codes[ITEMS];
        uint8_t scale[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          if (tid + 128u * j < items) quantize_block16(cur[d][j].lo, cur[d][j].hi, W.d_in, codes[j], scale[j]);
        }
        request(cur[d], s + kDepth * p.groups);
        const uint32_t slot = it % p.stages;
        if (!mbar_wait(bars + 8 * (p.stages + slot), ((it / p.stages) & 1u) ^ 1u)) {
          if (lane == 0) atomicOr(&g_a4_status, kQuantTimeout);
          ok = false;
          break;
        }
        const uint32_t b_tile = base + slot * stage_bytes + kABytes;
        const uint32_t sf_tile = b_tile + b_bytes + kSfBytes;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          if (tid + 128u * j < items) {
            const uint32_t t = tok[j], g = grp[j];
            // 128-byte swizzle: row t of the tile, 16-byte unit g / 2 exchanged by the row's low bits
            const uint32_t at = b_tile + (t >> 3) * 1024u + (t & 7u) * 128u + (((g >> 1) ^ (t & 7u)) << 4) + (g & 1u) * 8u;
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(codes[j].x), "r"(codes[j].y) : "memory");
            // scale tile of K-atom g / 4: row t at (t % 32) * 16 + (t / 32) * 4, group g % 4 within it
            const uint32_t sat = sf_tile + (g >> 2) * 512u + (t & 31u) * 16u + (t >> 5) * 4u + (g & 3u);
            asm volatile("st.shared.u8 [%0], %1;" ::"r"(sat), "r"(static_cast<uint32_t>(scale[j])) : "memory");
          }
        }
        // the tiles are read by the tensor core (async proxy): order these writes before it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(bars + 8 * slot);
        if (two) {   // the second entry reads this token tile: nothing to write, only its turn to take
          const uint32_t it2 = it + 1u, slot2 = it2 % p.stages;
          if (!mbar_wait(bars + 8 * (p.stages + slot2), ((it2 / p.stages) & 1u) ^ 1u)) {
            if (lane == 0) atomicOr(&g_a4_status, kQuantTimeout);
            ok = false;
            break;
          }
          mbar_arrive(bars + 8 * slot2);
        }
      }
    }
  } else if (warp == producer_warp) {
    // ---- producer of the weight tiles: they never depend on the previous kernel ----
    griddep_launch_dependents();
    const uint64_t policy = l2_evict_first_policy();
    RingAt at;
    for (uint32_t it = 0; it < entries; ++it, at.advance(1u, p.stages)) {
      if (!mbar_wait(bars + 8 * (p.stages + at.slot), at.phase ^ 1u)) {
        if (lane == 0) atomicOr(&g_a4_status, kProducerTimeout);
        break;
      }
      if (elect_one()) produce(it, at.slot, policy);
      __syncwarp();
    }
  } else {
    // ---- scale copies and MMAs: the whole warp runs the loop, an elected lane issues (elect_one, nvfp4_tc.cuh), so
    //      that a stage's eight copies and four MMAs follow one another in the tensor pipe's own order ----
    griddep_launch_dependents();
    // instruction descriptor: E2M1 x E2M1 (format 1 at bits 7 and 10), both K-major, N >> 3 at bit
    // 17, UE4M3 scales (bit 23 clear), M >> 4 at bit 24
    const uint32_t idesc = (1u << 7) | (1u << 10) | ((p.bn >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t desc0 = smem_desc(base, 1024u, 2u), sf_desc0 = smem_desc(base + kABytes + b_bytes, 128u, 0u);
    const uint32_t stage_units = stage_bytes >> 4;
    bool ok = true;
    RingAt at;
    uint32_t b_slot = 0;   // the ring entry that holds the stage's token tile: the first of the stage's entries
    for (uint32_t it = 0; it < entries; ++it, at.advance(1u, p.stages)) {
      const uint32_t half = two ? it & 1u : 0u;
      if (half == 0u) b_slot = at.slot;
      if (!mbar_wait(bars + 8 * at.slot, at.phase)) {   // weights landed and tokens quantized
        if (lane == 0) atomicOr(&g_a4_status, kMmaTimeout);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint32_t sf_cols = tmem + 64u + at.slot * 32u;  // 16 columns of weight scales, 16 of token scales
        const uint32_t sfb_cols = tmem + 64u + b_slot * 32u + 16u;
        const uint64_t sfa = sf_desc0 + at.slot * stage_units, sfb = sfa + (kSfBytes >> 4);
#pragma unroll
        for (uint32_t kb = 0; kb < 4; ++kb) {
          tmem_cp_sf(sf_cols + kb * 4u, sfa + kb * 32u);
          if (half == 0u) tmem_cp_sf(sfb_cols + kb * 4u, sfb + kb * 32u);
        }
        const uint64_t a_desc = desc0 + at.slot * stage_units, b_desc = desc0 + b_slot * stage_units + (kABytes >> 4);
#pragma unroll
        for (uint32_t kb = 0; kb < 4; ++kb) {   // 64 values along K are 32 bytes: two 16-byte units further
          mma_mxf4nvf4(tmem + half * p.bn, a_desc + 2u * kb, b_desc + 2u * kb, idesc, sf_cols + kb * 4u, sfb_cols + kb * 4u,
                       (it >= halves || kb != 0u) ? 1u : 0u);
        }
        if (half + 1u == halves) {   // the stage's entries go back to their writers together
          if (two) mma_commit(bars + 8 * (p.stages + b_slot));
          mma_commit(bars + 8 * (p.stages + at.slot));
        }
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(bar_acc);
    __syncwarp();
  }

  // ---- epilogue: thread r of warps 0-3 owns accumulator lane r = weight row r of the tile ----
  const uint32_t out_elem_f32 = p.epilogue & kEpilogueF32;
  bool have = false;
  uint32_t v[32], u[32];
  if (warp < 4) {
    have = mbar_wait(bar_acc, 0u);
    if (!have && lane == 0) atomicOr(&g_a4_status, kEpilogueTimeout);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (have) {
      const uint32_t lane_base = tmem + (static_cast<uint32_t>(warp * 32) << 16);
      if (p.bn == 16u) {
        tmem_ld16(lane_base, v);
        if (two) tmem_ld16(lane_base + 16u, u);
      } else {
        tmem_ld32(lane_base, v);
        if (two) tmem_ld32(lane_base + 32u, u);
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    }
  }
  // token tl, row r of the CTA's tile(s), from the accumulator sums (the second only with two tiles)
  const bool add = (p.epilogue & kEpilogueAdd) != 0u;
  auto residual = [&](uint32_t tl, uint32_t row) {
    const size_t at = static_cast<size_t>(tl) * W.ldy + row;
    return out_elem_f32 ? static_cast<const float *>(W.y)[at] : __bfloat162float(static_cast<const __nv_bfloat16 *>(W.y)[at]);
  };
  auto store = [&](size_t at, float acc, float old) {
    const float val = __fmul_rn(acc, W.alpha);   // not contracted into the residual add: one value for every epilogue
    if (out_elem_f32) static_cast<float *>(W.y)[at] = add ? old + val : val;
    else static_cast<__nv_bfloat16 *>(W.y)[at] = __float2bfloat16_rn(add ? val + old : val);
  };
  auto emit = [&](uint32_t tl, uint32_t r, float acc, float acc_b, float old, float old_b) {
    const size_t at = static_cast<size_t>(tl) * W.ldy + r;
    if (swiglu) {
      const float gv = __bfloat162float(__float2bfloat16_rn(__fmul_rn(acc, W.alpha)));
      const float uv = __bfloat162float(__float2bfloat16_rn(__fmul_rn(acc_b, W.alpha)));
      static_cast<__nv_bfloat16 *>(W.y)[at + row_a] = __float2bfloat16_rn(gv / (1.0f + __expf(-gv)) * uv);
    } else {
      store(at + row_a, acc, old);
      if (two) store(at + row_b, acc_b, old_b);
    }
  };
  if (kc == 1u) {
    if (warp < 4 && have) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (static_cast<uint32_t>(j) >= p.tokens) break;
        const uint32_t tl = static_cast<uint32_t>(j);
        emit(tl, threadIdx.x, __uint_as_float(v[j]), two ? __uint_as_float(u[j]) : 0.0f, add ? residual(tl, row_a + threadIdx.x) : 0.0f,
             add && two ? residual(tl, row_b + threadIdx.x) : 0.0f);
      }
    }
  } else {
    // Token tl is finished by rank tl % kc: once every ring of the cluster is idle, every CTA pushes its sums of it over
    // that rank's ring, [sender][turn][half][128 rows], and the bytes count at the receiver's barrier. Nobody reads
    // another CTA's memory, so nobody waits for a reader before it leaves. (Pulled between two meetings of the cluster, a
    // launch took 2.8 us from the last MMA to its end; with room for the sums beside the ring, and so without this
    // meeting, a layer at 8 tokens was no faster: 42.8 us against 42.3.)
    const uint32_t r = threadIdx.x & 127u;
    // the residual of a thread's next token is requested before it is needed
    float old = 0.0f, old_b = 0.0f;
    auto request_residual = [&](uint32_t i) {
      if (!add || i * kc + rank >= p.tokens) return;
      old = residual(i * kc + rank, row_a + r);
      if (two) old_b = residual(i * kc + rank, row_b + r);
    };
    if (warp < producer_warp) request_residual(static_cast<uint32_t>(warp) >> 2);
    cluster_sync_all();
    const uint32_t turns = (p.tokens + kc - 1u) / kc;
    if (warp < 4) {
      uint32_t at = base + (rank * turns * halves * 128u + threadIdx.x) * 4u, to = 0;
#pragma unroll
      for (uint32_t j = 0; j < 32u; ++j) {
        if (j >= p.tokens) break;
        const uint32_t bar = cluster_map(bar_sums, to);
        push_f32(cluster_map(at, to), have ? __uint_as_float(v[j]) : 0.0f, bar);
        if (two) push_f32(cluster_map(at + 512u, to), have ? __uint_as_float(u[j]) : 0.0f, bar);
        if (++to == kc) to = 0, at += halves * 512u;
      }
    }
    if (warp < producer_warp) {
      const float *sums = reinterpret_cast<const float *>(base_ptr) + r;
      if (mbar_wait_pushed(bar_sums)) {
        for (uint32_t i = static_cast<uint32_t>(warp) >> 2; i * kc + rank < p.tokens; i += p.groups) {
          float sum = 0.0f, sum_up = 0.0f;
          for (uint32_t q = 0; q < kc; ++q) {   // in rank order
            const float *from = sums + (q * turns + i) * halves * 128u;
            sum = q == 0u ? from[0] : sum + from[0];
            if (two) sum_up = q == 0u ? from[128] : sum_up + from[128];
          }
          emit(i * kc + rank, r, sum, sum_up, old, old_b);
          request_residual(i + p.groups);
        }
      } else if (lane == 0) {
        atomicOr(&g_a4_status, kReduceTimeout);
      }
    }
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == mma_warp) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
  }
}

constexpr size_t kA4MaxSmem = 220 * 1024;

// Ring depth: what fits beside the other CTAs of the SM, at most 8 stages and no more than the K slice has.
uint32_t a4_ring_depth(uint32_t ctas_per_sm, uint32_t bn, uint32_t k_stages) {
  const uint32_t stage_bytes = kABytes + bn * 128u + 2u * kSfBytes;
  uint32_t stages = (static_cast<uint32_t>(kA4MaxSmem / ctas_per_sm) - 2048u) / stage_bytes;
  if (stages > 8u) stages = 8u;
  return stages < k_stages ? stages : k_stages;
}

// The ring, barriers and the tensor-memory slot behind it, alignment slack.
size_t a4_smem_bytes(uint32_t bn, uint32_t stages) {
  return static_cast<size_t>(stages) * (kABytes + bn * 128u + 2u * kSfBytes) + 8u * (2u * stages + 2u) + 16u + 1024u;
}

}  // namespace

int32_t w4a4_decode_prepare(ErrorSlot &slot) {
  cudaError_t err = cudaFuncSetAttribute(w4a4_decode_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kA4MaxSmem));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(w4a4_decode_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kA4MaxSmem));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(w4a4_decode_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kA4MaxSmem));
  if (err != cudaSuccess) return fail(slot, "nvfp4 W4A4 decode kernel attributes: %s", cudaGetErrorString(err));
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
  // How many clusters of each size the device places at one CTA per SM (clusters stay inside one
  // GPC, so sizes 7 and 8 leave many SMs out). The occupancy query counts one CTA per SM for this
  // kernel whatever its shared memory; the plan scales the count by the CTAs that do share an SM.
  DeviceState *dev = device_state(slot);
  if (dev == nullptr) return -1;
  for (int kc = 1; kc <= 8 && !dev->counted; ++kc) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(kc) * 1024u, 1, 1);
    config.blockDim = dim3(64 + 128 * 2, 1, 1);
    config.dynamicSmemBytes = a4_smem_bytes(16, a4_ring_depth(1, 16, 64));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(kc);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, w4a4_decode_kernel<1>, &config) == cudaSuccess && clusters > 0) {
      dev->a4_slots[kc] = clusters * kc;
    } else {
      dev->a4_slots[kc] = 0;
      (void)cudaGetLastError();
    }
  }
  return 0;
}

bool w4a4_decode_takes(uint32_t n, uint32_t k, uint32_t tokens, uint32_t epilogue) {
  if ((epilogue & kEpilogueSwiglu) != 0u && ((n % 256u) != 0 || (epilogue & (kEpilogueAdd | kEpilogueF32)) != 0u)) return false;
  return tokens >= 1u && tokens <= kA4DecodeMaxTokens && (k % 256u) == 0 && (n % 128u) == 0;
}

int32_t w4a4_decode_launch(ErrorSlot &slot, const DeviceState &dev, const A4Item *items, uint32_t count, const uint16_t *x,
                           uint32_t k, uint32_t tokens, uint32_t epilogue, cudaStream_t stream) {
  A4Params p = {};
  A4Maps maps = {};
  p.x = x;
  p.count = count;
  p.k = k;
  p.tokens = tokens;
  p.bn = tokens <= 16u ? 16u : 32u;
  p.epilogue = epilogue;
  const uint32_t ctas_per_sm = dev.a4_decode_ctas == 1 ? 1u : 2u;
  const bool swiglu = (epilogue & kEpilogueSwiglu) != 0u;
  const uint32_t k_stages = k / 256u;
  // cluster size for `tiles` CTA rows: the largest K split that still runs as one wave (clusters are
  // placed inside one GPC: sizes 7 and 8 leave many slots empty)
  auto plan_kc = [&](uint32_t tiles) {
    uint32_t best = 1;
    for (uint32_t c = 2; c <= 8u && k_stages / c >= 2u; ++c) {
      const int known = dev.a4_slots[c];
      const uint32_t resident = (known > 0 ? static_cast<uint32_t>(known) : static_cast<uint32_t>(dev.sm_count) * 3u / 4u) * ctas_per_sm;
      if (tiles * c <= resident) best = c;
    }
    return best;
  };
  uint32_t row_tiles = 0;
  bool even = true;
  for (uint32_t i = 0; i < count; ++i) {
    row_tiles += (swiglu ? items[i].n / 2u : items[i].n) / 128u;
    even = even && (items[i].n % 256u) == 0;
  }
  uint32_t kc = plan_kc(row_tiles);
  // Two row tiles per CTA halve the quantizers' work per weight byte, K being split twice as often to
  // keep the CTA count. Worth it where the quantizers bound the kernel and K is hardly split yet:
  // wide weights at more than 8 tokens.
  const bool pair = !swiglu && even && k_stages >= 4u && (dev.a4_decode_pair >= 0 ? dev.a4_decode_pair != 0 : tokens > 8u && kc <= 2u);
  if (pair) {
    row_tiles /= 2u;
    kc = plan_kc(row_tiles);
  }
  p.pair = pair ? 1u : 0u;
  const bool two = swiglu || pair;
  uint32_t stages = a4_ring_depth(ctas_per_sm, p.bn, two ? 2u * k_stages : k_stages);
  if (two) stages &= ~1u;   // a K stage takes two ring entries
  p.stages = stages;
  // quantizer groups: two, so that two CTAs still share an SM's registers
  p.groups = dev.a4_decode_groups > 0 ? static_cast<uint32_t>(dev.a4_decode_groups) : 2u;
  if (p.groups > static_cast<uint32_t>(kMaxQuantGroups)) p.groups = kMaxQuantGroups;
  const uint32_t cols = 64u + 32u * stages;
  p.tmem_cols = cols <= 128u ? 128u : (cols <= 256u ? 256u : 512u);
  if (dev.a4_decode_kc > 0 && static_cast<uint32_t>(dev.a4_decode_kc) <= 8u && k_stages / dev.a4_decode_kc >= 1u) kc = dev.a4_decode_kc;
  p.kc = kc;
  uint32_t ctas = 0;
  for (uint32_t i = 0; i < count; ++i) {
    A4Weight &g = p.w[i];
    g.scales = items[i].scales;
    g.y = items[i].y;
    g.n = items[i].n;
    g.ldy = items[i].ldy;
    g.alpha = 1.0f / (items[i].d_in * items[i].d_w);
    g.d_in = items[i].d_in;
    g.block_begin = ctas;
    ctas += (two ? items[i].n / 2u : items[i].n) / 128u * kc;
    if (!make_code_map(&maps.m[i], items[i].codes, items[i].n, k / 2u, 128u)) {
      return fail(slot, "nvfp4 W4A4 decode route: tensor map encoding failed");
    }
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(ctas, 1, 1);
  config.blockDim = dim3(64 + 128 * p.groups, 1, 1);
  // the cluster's sums land over the ring: at least four stages of it where K is split, 32 tokens of two tiles at most
  if (kc > 1u && stages * (kABytes + p.bn * 128u + 2u * kSfBytes) < (tokens + kc - 1u) / kc * kc * (two ? 2u : 1u) * 512u) {
    return fail(slot, "nvfp4 W4A4 decode route: the ring is too short for a cluster of %u", kc);
  }
  config.dynamicSmemBytes = a4_smem_bytes(p.bn, stages);
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = dev.pdl ? 2 : 1;
  const cudaError_t err = tokens <= 8u    ? cudaLaunchKernelEx(&config, w4a4_decode_kernel<1>, maps, p)
                          : tokens <= 16u ? cudaLaunchKernelEx(&config, w4a4_decode_kernel<2>, maps, p)
                                          : cudaLaunchKernelEx(&config, w4a4_decode_kernel<4>, maps, p);
  if (err != cudaSuccess) return fail(slot, "nvfp4 W4A4 decode launch: %s", cudaGetErrorString(err));
  return 0;
}

int32_t w4a4_decode_status(ErrorSlot &slot, cudaStream_t stream, uint32_t *status) {
  cudaError_t err = cudaMemcpyFromSymbolAsync(status, g_a4_status, sizeof(uint32_t), 0, cudaMemcpyDeviceToHost, stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
  if (err != cudaSuccess) return fail(slot, "b200q_nvfp4_device_status: %s", cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q
