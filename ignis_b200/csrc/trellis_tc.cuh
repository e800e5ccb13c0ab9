// The trellis products on the 5th-generation tensor cores: the part shared by the dense prefill
// route (trellis_prefill.cu) and the MoE expert GEMMs (moe_tc.cu).
//
// Stands where the reference runs its prefill kernels on warp-level MMAs - trellis tiles decoded
// from shared memory into mma.sync fragments, fp16 accumulation folded every 32 inputs
// (kernel/src/trellis_linear_prefill.cu:162-279, kernel/src/moe_prefill.cu:252-421). The design
// here is not theirs:
//
//  * The activations are rotated once by a kernel of their own (x o suh, the 128-wide Hadamard in
//    fp32) and stored as plain fp16 rows [row][in] with ONE power-of-two scale per row (largest
//    magnitude in [2^13, 2^14)), so the whole sum over `in` accumulates in tensor memory and the
//    inverse scale is applied once, in the epilogue. fp16 keeps 11 significant bits of every value
//    down to 2^-28 of the row's largest; what lies below contributes less than that to any sum.
//  * A CTA owns up to 256 rows (two MMA tiles of M = 128: the rows are the accumulator's lanes) and
//    256 output columns (two 128-column Hadamard blocks: the MMA's N), and walks `in` in stages of
//    64. Sixteen decoder warps (four per scheduler: the decode is a chain of dependent integer
//    operations, and two warps per scheduler left it idle most cycles) turn the stage's 64
//    trellis tiles into fp16 in registers (the decode of
//    trellis_device.cuh: funnel shifts, IMAD, DP4A, half an HFMA2 per weight) and store them into
//    the stage's B tile in the K-major 128-byte-swizzle layout the tensor core reads: a lane's
//    eight values are four 4-byte stores that hit 32 different banks across the warp. A producer
//    thread brings the rows' fp16 activations by TMA (the same swizzle); one thread issues
//    tcgen05.mma kind::f16 (M 128, N 256, K 16; fp16 x fp16, fp32 accumulation in tensor memory).
//    Every decoded tile serves both row tiles: 512 accumulator columns, all of tensor memory.
//  * The epilogue: a thread owns one row of one 128-column block (of half a block when the job has
//    one row tile, so that all sixteen warps take part). It reads 64 accumulator columns, applies
//    the row's inverse scale and six Hadamard stages in registers and parks the 64 values in the
//    (by then idle) stage ring, where the seventh stage combines the two halves; the results are
//    parked once more and written out row-wise - half a warp per row, four columns a lane - with svh
//    and the caller's epilogue. All of it moves 16 bytes per lane and access.
//  * Every mbarrier wait is bounded; a wait that runs out sets a bit of a status word and the CTA
//    falls through to the common exit and frees its tensor memory.
#ifndef B200Q_TRELLIS_TC_CUH
#define B200Q_TRELLIS_TC_CUH

#include "nvfp4_tc.cuh"
#include "trellis_device.cuh"

namespace b200q {
namespace trellis_tc {

using namespace trellis_dev;

constexpr uint32_t kABytes = 128 * 128;     // one row tile of a stage: 128 rows x 64 fp16

// Two shapes of the CTA. DW = 16 decoder warps: 256 output columns (two Hadamard blocks), three
// stages, all 512 tensor-memory columns, one CTA per SM - every decoded tile serves up to 256 rows
// once. DW = 8: 128 output columns (one block), two stages, 256 tensor-memory columns, so that TWO
// CTAs share an SM (the same sixteen decoder warps in all) and one's setup, pipeline fill, drain and
// epilogue run under the other's decoding: for jobs too short to amortise those (the MoE items).
template <int DW>
struct Shape {
  static constexpr int kDecoderWarps = DW;
  static constexpr int kThreads = (DW + 2) * 32;   // the decoder / epilogue warps, the producer warp, the MMA warp
  static constexpr uint32_t kBlocks = DW / 8;       // 128-column blocks per CTA
  static constexpr uint32_t kCols = DW * 16;        // output columns per CTA = accumulator columns per row tile
  static constexpr uint32_t kStages = DW == 16 ? 3 : 2;
  static constexpr uint32_t kBBytes = kCols * 128;  // one stage of decoded weights: kCols columns x 64 fp16
  static constexpr uint32_t kStageBytes = 2 * kABytes + kBBytes;
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + 256 + 1024;   // + barriers and the tensor-memory slot + alignment slack
  static constexpr uint32_t kTmemCols = 2 * kCols;
};
constexpr uint32_t kStatusProducer = 1u, kStatusMma = 2u, kStatusEpilogue = 4u, kStatusDecoder = 8u;

// What one CTA multiplies: rows [row0, row0 + rows) of the rotated activations (rows <= 256) with
// two 128-column blocks of one trellis plane.
struct Job {
  const uint32_t *trellis;  // the plane: tile (tk, tn) at word (tk * tile_stride + tn) * 4 k2
  uint32_t k2;
  uint32_t tile_stride;     // tiles per stored row of the plane
  uint32_t blk0, blk1;      // the 128-column blocks behind accumulator columns 0..127 and 128..255
  uint32_t nblk;            // 1: blk1 does not exist (the MMA's N is 128)
  uint32_t row0, rows;      // row0 is also the TMA row coordinate
  uint32_t stage0, stage1;  // the K stages of 64 inputs it walks: all of `in`, or the CTA's share of a cluster's
};

// The raw words of the 4 tiles a decoder warp owns in one stage (1 tile column x 4 tile rows), one
// word per lane and tile (two for the widths whose tiles have more than 32 words): lane l holds
// word l of the tile, and the three words a lane's window needs come from its neighbours by shuffle.
// A 16 x 16 tile is 4 k2 words, so one coalesced load of up to 128 bytes fetches a whole tile.
template <int K2>
struct StageWords {
  static constexpr int kPerTile = (4 * K2 + 31) / 32;
  uint32_t w[4][kPerTile];
};

constexpr int kWordRing = 4;   // stages of raw words a decoder warp keeps in flight in registers

// Six stages of the in-register Sylvester Hadamard (natural order) on 64 values: one half of a
// 128-wide transform, whose seventh stage pairs value i of one half with value i of the other.
__device__ __forceinline__ void hadamard64_regs(float (&v)[64]) {
#pragma unroll
  for (int h = 1; h < 64; h <<= 1) {
#pragma unroll
    for (int i = 0; i < 64; ++i) {
      if ((i & h) == 0) {
        const float a = v[i], b = v[i + h];
        v[i] = a + b;
        v[i + h] = a - b;
      }
    }
  }
}

template <int K2>
__device__ __forceinline__ void load_stage_words(StageWords<K2> &sw, const uint32_t *col0, int lane, uint64_t row_words, uint32_t ks) {
  // tile rows 4 ks .. 4 ks + 3 of the warp's tile column
  const uint32_t *base = col0 + static_cast<uint64_t>(ks) * 4u * row_words + lane;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t *t = base + static_cast<uint64_t>(r) * row_words;
#pragma unroll
    for (int h = 0; h < StageWords<K2>::kPerTile; ++h) {
      sw.w[r][h] = (32 * h + lane < 4 * K2) ? __ldg(t + 32 * h) : 0u;
    }
  }
}

// Word `index` of a tile whose words lie one per lane (and, beyond 32, in the second register).
template <int K2>
__device__ __forceinline__ uint32_t tile_word(const uint32_t (&w)[(4 * K2 + 31) / 32], uint32_t index) {
  if ((4 * K2 + 31) / 32 == 1) return __shfl_sync(0xFFFFFFFFu, w[0], static_cast<int>(index));
  const uint32_t lo = __shfl_sync(0xFFFFFFFFu, w[0], static_cast<int>(index & 31u));
  const uint32_t hi = __shfl_sync(0xFFFFFFFFu, w[(4 * K2 + 31) / 32 - 1], static_cast<int>(index & 31u));
  return index < 32u ? lo : hi;
}

// The decoder warps' loop over the job's K stages. `stages_base` is the shared-memory address of
// stage 0; `bars`: full[kStages], empty[kStages].
template <int K2, int DW>
__device__ __forceinline__ bool decode_stages(const Job &job, uint32_t stages_base, uint32_t bars, int warp, int lane, uint32_t *status) {
  constexpr uint32_t kStages = Shape<DW>::kStages, kStageBytes = Shape<DW>::kStageBytes;
  const LaneWindow win = lane_window(K2, lane);
  const uint32_t k_stages = job.stage1 - job.stage0;
  const uint32_t cb = static_cast<uint32_t>(warp) >> 3;                    // which of the job's two column blocks
  const uint32_t blk = cb == 0u ? job.blk0 : job.blk1;
  const uint32_t tn = blk * 8u + (static_cast<uint32_t>(warp) & 7u);        // the warp's tile column in the plane
  const uint64_t row_words = static_cast<uint64_t>(job.tile_stride) * 4u * K2;
  const uint32_t *col0 = job.trellis + static_cast<uint64_t>(tn) * 4u * K2 + static_cast<uint64_t>(job.stage0) * 4u * row_words;
  const bool live = cb < job.nblk;
  const uint32_t c0 = static_cast<uint32_t>(lane) >> 2, t = static_cast<uint32_t>(lane) & 3u;
  // row n = 16 warp + c0 (+ 8) of the B tile: 8-row group 2 warp (+ 1)
  const uint32_t lane_off = kABytes * 2u + (2u * static_cast<uint32_t>(warp)) * 1024u + c0 * 128u + 4u * t;
  // The words of the next kWordRing stages are in flight in registers: a load issued when its
  // stage's slot of the ring was last decoded has several stage times to arrive (one stage ahead is
  // not enough: a stage is shorter than the latency of HBM).
  StageWords<K2> ring[kWordRing];
#pragma unroll
  for (int d = 0; d < kWordRing; ++d) {   // the weights never depend on the previous kernel
    if (live && static_cast<uint32_t>(d) < k_stages) load_stage_words<K2>(ring[d], col0, lane, row_words, static_cast<uint32_t>(d));
  }
  griddep_launch_dependents();
  griddep_wait();   // from here on the warp may also touch what an earlier kernel wrote
  for (uint32_t it0 = 0; it0 < k_stages; it0 += kWordRing) {
#pragma unroll
    for (int d = 0; d < kWordRing; ++d) {
      const uint32_t it = it0 + static_cast<uint32_t>(d);
      if (it >= k_stages) break;
      const uint32_t slot = it % kStages;
      if (!mbar_wait(bars + 8u * (kStages + slot), ((it / kStages) & 1u) ^ 1u)) {
        if (lane == 0) atomicOr(status, kStatusDecoder);
        return false;
      }
      if (live) {
        const uint32_t tile = stages_base + slot * kStageBytes + lane_off;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t w0 = tile_word<K2>(ring[d].w[r], win.w0), w1 = tile_word<K2>(ring[d].w[r], win.w1),
                         w2 = tile_word<K2>(ring[d].w[r], win.w2);
          uint32_t frag[4];
          decode8<K2>(w0, w1, w2, win.off, frag);
          const uint32_t lo = ((2u * r) ^ c0) << 4, hi = ((2u * r + 1u) ^ c0) << 4;
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + lo), "r"(frag[0]) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + hi), "r"(frag[1]) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + 1024u + lo), "r"(frag[2]) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + 1024u + hi), "r"(frag[3]) : "memory");
        }
        // the tile is read by the tensor core (async proxy): order these writes before it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      mbar_arrive(bars + 8u * slot);
      if (live && it + kWordRing < k_stages) load_stage_words<K2>(ring[d], col0, lane, row_words, it + kWordRing);
    }
  }
  return true;
}

template <int DW>
__device__ __forceinline__ bool decode_stages_any(const Job &job, uint32_t stages_base, uint32_t bars, int warp, int lane, uint32_t *status) {
  switch (job.k2) {
    case 4: return decode_stages<4, DW>(job, stages_base, bars, warp, lane, status);
    case 5: return decode_stages<5, DW>(job, stages_base, bars, warp, lane, status);
    case 6: return decode_stages<6, DW>(job, stages_base, bars, warp, lane, status);
    case 8: return decode_stages<8, DW>(job, stages_base, bars, warp, lane, status);
    case 10: return decode_stages<10, DW>(job, stages_base, bars, warp, lane, status);
    default: return decode_stages<12, DW>(job, stages_base, bars, warp, lane, status);
  }
}

// Shared-memory carve-up and the three roles up to the finished accumulator. On return with true,
// the calling decoder warp may read the accumulators: tensor-memory columns [256 tt, 256 tt + 256)
// hold row tile tt, lanes = rows, the job's block 0 in the first 128 columns of a tile. The caller
// ends with core_finish().
struct Core {
  uint32_t base, bars, bar_acc, tmem;
  uint32_t *tmem_slot;
  int warp, lane;
};

template <int DW>
__device__ __forceinline__ Core core_setup(uint8_t *smem_raw) {
  constexpr uint32_t kStages = Shape<DW>::kStages, kStageBytes = Shape<DW>::kStageBytes, kTmemCols = Shape<DW>::kTmemCols;
  constexpr int kDecoderWarps = DW;
  Core c;
  const uint32_t raw = smem_u32(smem_raw);
  c.base = (raw + 1023u) & ~1023u;   // the 128-byte swizzle wants 1024-byte aligned tiles
  c.bars = c.base + kStages * kStageBytes;       // full[kStages], empty[kStages], accumulator full
  c.bar_acc = c.bars + 8u * 2u * kStages;
  c.tmem_slot = reinterpret_cast<uint32_t *>(smem_raw + (c.base - raw) + kStages * kStageBytes + 128);
  c.warp = threadIdx.x >> 5;   // not uniform_warp(): a uniform index moved the decoders' addressing to the uniform datapath and cost 27 %
  c.lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; ++s) {
      mbar_init(c.bars + 8u * s, kDecoderWarps * 32 + 1);   // every decoder thread and the producer's expect_tx arrival
      mbar_init(c.bars + 8u * (kStages + s), 1);            // the MMA thread's commit
    }
    mbar_init(c.bar_acc, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (c.warp == kDecoderWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(c.tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  c.tmem = __shfl_sync(0xFFFFFFFFu, *c.tmem_slot, 0);
  return c;
}

// The decoder warps' second step: waits for the accumulator. Returns true in the decoder warps when
// all of them have the complete accumulator (the epilogue may read tensor memory and use barrier 1).
// Every decoder warp calls it, with what core_roles returned to it.
template <int DW>
__device__ __forceinline__ bool core_accumulator(const Core &c, bool decoded, uint32_t *status) {
  constexpr int kDecoderWarps = DW;
  bool have = false;
  if (decoded) {
    have = mbar_wait(c.bar_acc, 0u);
    if (!have && c.lane == 0) atomicOr(status, kStatusEpilogue);
  }
  // The epilogue's warps meet at barriers of their own: either every decoder warp has its
  // accumulator or none goes on (a warp whose wait ran out must not leave the others waiting).
  uint32_t all;
  asm volatile("{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.and.pred q, 1, %2, p; selp.u32 %0, 1, 0, q; }"
               : "=r"(all) : "r"(static_cast<uint32_t>(have)), "n"(kDecoderWarps * 32) : "memory");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return all != 0u;
}

// Runs the CTA's roles: the producer and the MMA thread to their end, the decoder warps through
// their K stages. Returns true in a decoder warp that decoded all of them; such a warp has time for
// loads of its own (what its epilogue will need) before it calls core_accumulator, while the last
// MMAs retire.
template <int DW>
__device__ __forceinline__ bool core_roles(const Core &c, const Job &job, const CUtensorMap *map_a, uint32_t *status) {
  constexpr uint32_t kStages = Shape<DW>::kStages, kStageBytes = Shape<DW>::kStageBytes;
  constexpr int kDecoderWarps = DW;
  const uint32_t k_stages = job.stage1 - job.stage0;
  const uint32_t row_tiles = job.rows > 128u ? 2u : 1u;
  if (c.warp < kDecoderWarps) return decode_stages_any<DW>(job, c.base, c.bars, c.warp, c.lane, status);
  if (c.warp == kDecoderWarps) {
    // ---- producer of the activation tiles ----
    griddep_launch_dependents();
    griddep_wait();   // the rotated activations come from the kernel before
    RingAt at;
    for (uint32_t it = 0; it < k_stages; ++it, at.advance(1u, kStages)) {
      if (!mbar_wait(c.bars + 8u * (kStages + at.slot), at.phase ^ 1u)) {
        if (c.lane == 0) atomicOr(status, kStatusProducer);
        break;
      }
      if (elect_one()) {
        const uint32_t full = c.bars + 8u * at.slot, stage = c.base + at.slot * kStageBytes;
        const int32_t x = static_cast<int32_t>((job.stage0 + it) * 64u);
        mbar_expect_tx(full, row_tiles * kABytes);
        tma_load_2d(stage, map_a, full, x, static_cast<int32_t>(job.row0));
        if (row_tiles == 2u) tma_load_2d(stage + kABytes, map_a, full, x, static_cast<int32_t>(job.row0 + 128u));
      }
      __syncwarp();
    }
    return false;
  }
  // ---- MMA issuer: the whole warp runs the loop, an elected lane issues (elect_one, nvfp4_tc.cuh) ----
  griddep_launch_dependents();
  griddep_wait();
  // instruction descriptor: FP32 accumulator (bit 4), A and B FP16 (format 0), both K-major,
  // N >> 3 at bit 17, M >> 4 at bit 24
  const uint32_t mma_n = job.nblk * 128u;
  const uint32_t idesc = (1u << 4) | ((mma_n >> 3) << 17) | ((128u >> 4) << 24);
  const uint64_t desc0 = smem_desc_sw128(c.base);
  bool ok = true;
  RingAt at;
  for (uint32_t it = 0; it < k_stages; ++it, at.advance(1u, kStages)) {
    if (!mbar_wait(c.bars + 8u * at.slot, at.phase)) {
      if (c.lane == 0) atomicOr(status, kStatusMma);
      ok = false;
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (elect_one()) {
      const uint64_t a0 = desc0 + at.slot * (kStageBytes >> 4), a1 = a0 + (kABytes >> 4), b = a1 + (kABytes >> 4);
#pragma unroll
      for (uint32_t kb = 0; kb < 4; ++kb) {   // 16 values along K are 32 bytes: two 16-byte units further
        mma_f16(c.tmem, a0 + 2u * kb, b + 2u * kb, idesc, (it | kb) != 0u ? 1u : 0u);
        if (row_tiles == 2u) mma_f16(c.tmem + Shape<DW>::kCols, a1 + 2u * kb, b + 2u * kb, idesc, (it | kb) != 0u ? 1u : 0u);
      }
      mma_commit(c.bars + 8u * (kStages + at.slot));
    }
    __syncwarp();
  }
  if (ok && elect_one()) mma_commit(c.bar_acc);
  __syncwarp();
  return false;
}

// ---- epilogue ------------------------------------------------------------------------------------
// A warp group (warp / 4: four warps, 128 threads = the 128 rows of a row tile, a warp's lanes the
// rows 32 (warp % 4) .. + 31) owns an area of the idle stage ring: 128 rows of 64 floats, 68 apart, so
// that 16-byte accesses are free of bank conflicts both when a warp's lanes are 32 rows (a thread
// parking its row) and when they are one row's values (the warp writing rows out).
constexpr uint32_t kPitch = 68;
constexpr uint32_t kArea = 128 * kPitch;   // floats
static_assert(2 * kArea * 4 <= Shape<8>::kStages * Shape<8>::kStageBytes && 4 * kArea * 4 <= Shape<16>::kStages * Shape<16>::kStageBytes,
              "the areas of all warp groups fit into the stage ring");

// A cluster that shares a job's K stages parks every CTA's share of the sums (the transform is linear);
// the rows are dealt over the ranks, and a row's owner adds what the ranks parked for it, its own first.
struct Split {
  uint32_t ranks, rank;
};
constexpr Split kWhole = {1u, 0u};

// The cluster meetings of one job's epilogue, for the threads that do not run it.
__device__ __forceinline__ void split_meetings(const Split split, uint32_t row_tiles) {
  if (split.ranks == 1u) return;
  for (uint32_t i = 0; i < 2u * row_tiles; ++i) cluster_sync_all();
}

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

// Hands the calling warp's first `rows` rows of 64 parked values to `emit(r, there, v)`, two rows at a
// time: a half-warp per row, lane l its values 4 (l % 16) .. + 3, so what the caller stores per row is
// contiguous. (A thread storing its own row touches 32 different lines per instruction, and the memory
// pipe takes them one per cycle: the row-wise form is what makes the epilogue short.) All lanes call
// `emit` together; `there` is false in the half whose row does not exist.
//
// With a cluster the row pairs are dealt over the ranks between two meetings: everything is parked, and
// nothing is parked over it before every rank has read it.
template <class RowEmit>
__device__ __forceinline__ void emit_rows(const float *area, uint32_t quad, uint32_t lane, uint32_t rows, const Split split, RowEmit emit) {
  const uint32_t up = lane >> 4, pairs = (rows + 1u) / 2u;
  const float *base = area + (quad * 32u + up) * kPitch + 4u * (lane & 15u);
  if (split.ranks == 1u) {
    for (uint32_t i = 0; i < pairs; ++i) emit(2u * i + up, 2u * i + up < rows, *reinterpret_cast<const float4 *>(base + 2u * i * kPitch));
    return;
  }
  cluster_sync_all();
  const uint32_t mine = smem_u32(base);
  for (uint32_t i0 = split.rank; i0 < pairs; i0 += 4u * split.ranks) {   // four pairs at a time: their loads travel together
    float4 sum[4];
    for (uint32_t k = 0, q = split.rank; k < split.ranks; ++k, q = q + 1u == split.ranks ? 0u : q + 1u) {   // no rank is read by all at once
      float4 v[4];
#pragma unroll
      for (uint32_t j = 0; j < 4u; ++j) {
        const uint32_t i = i0 + j * split.ranks;
        v[j] = i < pairs ? ld_cluster_f32x4(mine + 8u * kPitch * i, q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
#pragma unroll
      for (uint32_t j = 0; j < 4u; ++j) {
        if (k == 0u) sum[j] = v[j];
        else sum[j].x += v[j].x, sum[j].y += v[j].y, sum[j].z += v[j].z, sum[j].w += v[j].w;
      }
    }
#pragma unroll
    for (uint32_t j = 0; j < 4u; ++j) {
      const uint32_t i = i0 + j * split.ranks;
      if (i < pairs) emit(2u * i + up, 2u * i + up < rows, sum[j]);
    }
  }
  cluster_sync_all();
}

__device__ __forceinline__ void load_half_row(uint32_t taddr, float inv, float (&v)[64]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t r[32];
    tmem_ld32(taddr + 32u * q, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[32 * q + i] = __uint_as_float(r[i]) * inv;
  }
}

__device__ __forceinline__ float4 four_halves(const uint16_t *p) {
  const uint2 raw = __ldg(reinterpret_cast<const uint2 *>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void park_row(float *row, const float (&v)[64]) {
#pragma unroll
  for (int i = 0; i < 64; i += 4) *reinterpret_cast<float4 *>(row + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// The epilogue of one (row tile, block) item for the calling warp: a thread owns one row (lane =
// row 32 quad + lane of the row tile; `rows` of the warp's 32 exist, `valid` = lane < rows) and
// `taddr` is the tensor-memory address of the block's first column in those lanes. The thread
// applies `inv` and six Hadamard stages to each half of its 128 columns in registers, the seventh
// stage combines the halves through `area`, and `emit(pass, r, there, v)` receives, two rows at a
// time, columns 64 pass + 4 (lane % 16) .. + 3 of row r, 1 / sqrt(128) included.
template <class RowEmit>
__device__ __forceinline__ void block_epilogue(uint32_t taddr, float inv, bool valid, float *area, uint32_t quad, uint32_t lane,
                                               uint32_t rows, const Split split, RowEmit emit) {
  float *row = area + (quad * 32u + lane) * kPitch;
  float v[64];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    load_half_row(taddr + 64u * half, inv, v);
    if (valid) {
      hadamard64_regs(v);
      if (half == 0) park_row(row, v);
    }
  }
  const float c = 0.08838834764831845f;   // 1 / sqrt(128)
  if (valid) {   // the seventh stage: columns i (sum, parked) and 64 + i (difference, kept)
#pragma unroll
    for (int i = 0; i < 64; i += 4) {
      float4 a = *reinterpret_cast<const float4 *>(row + i);
      const float b0 = v[i], b1 = v[i + 1], b2 = v[i + 2], b3 = v[i + 3];
      *reinterpret_cast<float4 *>(row + i) = make_float4((a.x + b0) * c, (a.y + b1) * c, (a.z + b2) * c, (a.w + b3) * c);
      v[i] = (a.x - b0) * c;
      v[i + 1] = (a.y - b1) * c;
      v[i + 2] = (a.z - b2) * c;
      v[i + 3] = (a.w - b3) * c;
    }
  }
  __syncwarp();
  emit_rows(area, quad, lane, rows, split, [&](uint32_t r, bool there, const float4 &o) { emit(0u, r, there, o); });
  __syncwarp();
  if (valid) park_row(row, v);
  __syncwarp();
  emit_rows(area, quad, lane, rows, split, [&](uint32_t r, bool there, const float4 &o) { emit(1u, r, there, o); });
}

// The same for a job of one row tile, where only two of the four warp groups would have a block:
// groups g and g ^ 2 share block g & 1, a thread owning 64 columns of its row (half = g >> 1). Each
// transforms its half and parks it in its group's area (`mine`); all decoder warps meet at barrier 1;
// the seventh stage gives the first half's owner columns 0..63 (sums) and the other's columns
// 64..127 (differences), parked again after a second meeting and written out row-wise:
// `emit(half, r, there, v)` as above. Every decoder warp calls this exactly once (`live`: the group's
// block exists - warp-uniform).
template <int DW, class RowEmit>
__device__ __forceinline__ void half_epilogue(uint32_t taddr_block, uint32_t half, bool live, float inv, bool valid, float *mine,
                                              const float *other, uint32_t quad, uint32_t lane, uint32_t rows, const Split split, RowEmit emit) {
  const uint32_t at = (quad * 32u + lane) * kPitch;
  float v[64];
  if (live) {
    load_half_row(taddr_block + 64u * half, inv, v);
    if (valid) {
      hadamard64_regs(v);
      park_row(mine + at, v);
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
  const float c = 0.08838834764831845f;   // 1 / sqrt(128)
  if (live && valid) {
#pragma unroll
    for (int i = 0; i < 64; i += 4) {
      const float4 o = *reinterpret_cast<const float4 *>(other + at + i);
      v[i] = half == 0u ? (v[i] + o.x) * c : (o.x - v[i]) * c;
      v[i + 1] = half == 0u ? (v[i + 1] + o.y) * c : (o.y - v[i + 1]) * c;
      v[i + 2] = half == 0u ? (v[i + 2] + o.z) * c : (o.z - v[i + 2]) * c;
      v[i + 3] = half == 0u ? (v[i + 3] + o.w) * c : (o.w - v[i + 3]) * c;
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
  if (!live) return;
  if (valid) park_row(mine + at, v);
  __syncwarp();
  emit_rows(mine, quad, lane, rows, split, [&](uint32_t r, bool there, const float4 &o) { emit(half, r, there, o); });
}

template <int DW>
__device__ __forceinline__ void core_finish(const Core &c) {
  constexpr int kDecoderWarps = DW;
  constexpr uint32_t kTmemCols = Shape<DW>::kTmemCols;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (c.warp == kDecoderWarps + 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(kTmemCols) : "memory");
  }
}

// The rotated activations [rows][in] fp16 as a 2-D tensor with boxes of 128 rows x 64 values, 128-byte swizzle.
inline bool make_rows_map(CUtensorMap *map, const void *rows_f16, uint64_t rows, uint64_t in) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {in, rows};
  const cuuint64_t strides[1] = {in * 2u};
  const cuuint32_t box[2] = {64u, 128u};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(rows_f16), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace trellis_tc
}  // namespace b200q

#endif
