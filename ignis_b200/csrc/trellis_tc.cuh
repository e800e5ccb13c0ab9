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
//    parked once more and written out row-wise - a warp per row, a lane per column - with svh and
//    the caller's epilogue, so that a warp's stores (or atomics) are contiguous.
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
  static constexpr uint32_t kRawBytes = kBlocks * 15360;          // ring of packed words
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + kRawBytes + 256 + 1024;   // + barriers and the tensor-memory slot + alignment slack
  static constexpr uint32_t kTmemCols = 2 * kCols;
};
constexpr uint32_t kStatusProducer = 1u, kStatusMma = 2u, kStatusEpilogue = 4u, kStatusDecoder = 8u;

// What one CTA multiplies: rows [row0, row0 + rows) of the rotated activations (rows <= 256) with
// two 128-column blocks of one trellis plane.
struct Job {
  const uint32_t *trellis;  // the plane: tile (tk, tn) at word (tk * tile_stride + tn) * 4 k2
  uint32_t k2;
  uint32_t tile_stride;     // tiles per stored row of the plane
  uint32_t in;              // a multiple of 128
  uint32_t blk0, blk1;      // the 128-column blocks behind accumulator columns 0..127 and 128..255
  uint32_t nblk;            // 1: blk1 does not exist (the MMA's N is 128)
  uint32_t row0, rows;      // row0 is also the TMA row coordinate
  uint32_t stage0, stage1;  // the K stages of 64 inputs it walks
};

// The ring of packed words: a slot is one K stage of the CTA's tile columns, four tile rows of a contiguous 128 k2 bytes per
// column block. Three to seven stages fit, by the width (of DW = 16 as many: twice the columns, twice the bytes).
__host__ __device__ constexpr uint32_t raw_slot_bytes(uint32_t k2, uint32_t blocks) { return 512u * k2 * blocks; }
constexpr uint32_t kMaxRaw = 7;
template <int DW>
__device__ __forceinline__ uint32_t raw_slots(uint32_t k2) {
  const uint32_t fit = Shape<DW>::kRawBytes / raw_slot_bytes(k2, Shape<DW>::kBlocks);
  return fit < kMaxRaw ? fit : kMaxRaw;
}
__device__ __forceinline__ uint32_t lds32(uint32_t address) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(address));
  return v;
}

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

// The decoder warps' loop over the job's K stages. `stages_base` is the shared-memory address of
// stage 0; `bars`: full[kStages], empty[kStages]; `raw_base`, `raw_bars`: the packed words' ring and its full barriers. (Words
// requested ahead into registers have to arrive before the proxy fence that hands a stage to the tensor core lets a thread go
// on, whichever stage they belong to; from shared memory the fence finds nothing in flight.)
template <int K2, int DW>
__device__ __forceinline__ bool decode_stages(const Job &job, uint32_t stages_base, uint32_t bars, uint32_t raw_base, uint32_t raw_bars, int warp,
                                              int lane, uint32_t *status) {
  constexpr uint32_t kStages = Shape<DW>::kStages, kStageBytes = Shape<DW>::kStageBytes, kSlot = raw_slot_bytes(K2, Shape<DW>::kBlocks);
  const LaneWindow win = lane_window(K2, lane);
  const uint32_t cb = static_cast<uint32_t>(warp) >> 3;                    // which of the job's two column blocks
  const bool live = cb < job.nblk;
  const uint32_t c0 = static_cast<uint32_t>(lane) >> 2, t = static_cast<uint32_t>(lane) & 3u;
  // row n = 16 warp + c0 (+ 8) of the B tile: 8-row group 2 warp (+ 1)
  const uint32_t lane_off = kABytes * 2u + (2u * static_cast<uint32_t>(warp)) * 1024u + c0 * 128u + 4u * t;
  // the lane's words of the warp's tile column in a slot: tile row r is 128 K2 bytes further
  const uint32_t col = raw_base + cb * 512u * K2 + (static_cast<uint32_t>(warp) & 7u) * 16u * K2;
  const uint32_t at0 = col + 4u * win.w0, at1 = col + 4u * win.w1, at2 = col + 4u * win.w2;
  const uint32_t raws = raw_slots<DW>(K2);
  griddep_launch_dependents();
  griddep_wait();   // the epilogue touches what an earlier kernel wrote
  RingAt at, from;
  // A stage's twelve words are read while the stage before is handed over: their latency, and the wait for the copies behind
  // them, run under the fence.
  uint32_t w[4][3];
  auto read_words = [&]() {
    const uint32_t raw = from.slot * kSlot;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      w[r][0] = lds32(at0 + raw + r * 128u * K2);
      w[r][1] = lds32(at1 + raw + r * 128u * K2);
      w[r][2] = lds32(at2 + raw + r * 128u * K2);
    }
  };
  if (!mbar_wait(raw_bars, 0u)) {
    if (lane == 0) atomicOr(status, kStatusDecoder);
    return false;
  }
  if (live) read_words();
  for (uint32_t it = job.stage0; it < job.stage1; ++it, at.advance(1u, kStages)) {
    if (!mbar_wait(bars + 8u * (kStages + at.slot), at.phase ^ 1u)) {
      if (lane == 0) atomicOr(status, kStatusDecoder);
      return false;
    }
    if (live) {
      const uint32_t tile = stages_base + at.slot * kStageBytes + lane_off;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        uint32_t frag[4];
        decode8<K2>(w[r][0], w[r][1], w[r][2], win.off, frag);
        const uint32_t lo = ((2u * r) ^ c0) << 4, hi = ((2u * r + 1u) ^ c0) << 4;
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + lo), "r"(frag[0]) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + hi), "r"(frag[1]) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + 1024u + lo), "r"(frag[2]) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + 1024u + hi), "r"(frag[3]) : "memory");
      }
    }
    from.advance(1u, raws);
    if (it + 1u < job.stage1) {
      if (!mbar_wait(raw_bars + 8u * from.slot, from.phase)) {
        if (lane == 0) atomicOr(status, kStatusDecoder);
        return false;
      }
      if (live) read_words();
    }
    // the tile is read by the tensor core (async proxy): order these writes before it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bars + 8u * at.slot);
  }
  return true;
}

template <int DW>
__device__ __forceinline__ bool decode_stages_any(const Job &job, uint32_t stages_base, uint32_t bars, uint32_t raw_base, uint32_t raw_bars, int warp, int lane,
                                                  uint32_t *status) {
  switch (job.k2) {
    case 4: return decode_stages<4, DW>(job, stages_base, bars, raw_base, raw_bars, warp, lane, status);
    case 5: return decode_stages<5, DW>(job, stages_base, bars, raw_base, raw_bars, warp, lane, status);
    case 6: return decode_stages<6, DW>(job, stages_base, bars, raw_base, raw_bars, warp, lane, status);
    case 8: return decode_stages<8, DW>(job, stages_base, bars, raw_base, raw_bars, warp, lane, status);
    case 10: return decode_stages<10, DW>(job, stages_base, bars, raw_base, raw_bars, warp, lane, status);
    default: return decode_stages<12, DW>(job, stages_base, bars, raw_base, raw_bars, warp, lane, status);
  }
}

// Shared-memory carve-up and the three roles up to the finished accumulator. On return with true,
// the calling decoder warp may read the accumulators: tensor-memory columns [256 tt, 256 tt + 256)
// hold row tile tt, lanes = rows, the job's block 0 in the first 128 columns of a tile. The caller
// ends with core_finish().
struct Core {
  uint32_t base, bars, bar_acc, raw, raw_bars, tmem;
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
  c.raw = c.base + kStages * kStageBytes;        // the packed words' ring
  c.bars = c.raw + Shape<DW>::kRawBytes;         // full[kStages], empty[kStages], accumulator full, words full[kMaxRaw]
  c.bar_acc = c.bars + 8u * 2u * kStages;
  c.raw_bars = c.bar_acc + 8u;
  c.tmem_slot = reinterpret_cast<uint32_t *>(smem_raw + (c.bars - raw) + 128);
  c.warp = threadIdx.x >> 5;   // not uniform_warp(): a uniform index moved the decoders' addressing to the uniform datapath and cost 27 %
  c.lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; ++s) {
      mbar_init(c.bars + 8u * s, kDecoderWarps + 1);        // every decoder warp and the producer's expect_tx arrival
      mbar_init(c.bars + 8u * (kStages + s), 1);            // the MMA thread's commit
    }
    mbar_init(c.bar_acc, 1);
    for (uint32_t s = 0; s < kMaxRaw; ++s) mbar_init(c.raw_bars + 8u * s, 1);
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
  if (c.warp < kDecoderWarps) return decode_stages_any<DW>(job, c.base, c.bars, c.raw, c.raw_bars, c.warp, c.lane, status);
  if (c.warp == kDecoderWarps) {
    // ---- producer: the packed words (they never depend on the previous kernel) and the activation tiles ----
    const uint32_t raws = raw_slots<DW>(job.k2), slot_bytes = raw_slot_bytes(job.k2, Shape<DW>::kBlocks), row_bytes = 128u * job.k2;
    const uint64_t row_pitch = static_cast<uint64_t>(job.tile_stride) * 16u * job.k2;   // bytes from a tile row to the next
    const uint8_t *plane = reinterpret_cast<const uint8_t *>(job.trellis) + static_cast<uint64_t>(job.stage0) * 4u * row_pitch;
    auto words = [&](uint32_t it, uint32_t slot) {   // stage `it` of the job into `slot`: four tile rows per column block
      const uint32_t full = c.raw_bars + 8u * slot, dst = c.raw + slot * slot_bytes;
      mbar_expect_tx(full, 4u * row_bytes * job.nblk);
      const uint8_t *src = plane + static_cast<uint64_t>(it) * 4u * row_pitch;
      for (uint32_t b = 0; b < job.nblk; ++b) {
        const uint8_t *block = src + static_cast<uint64_t>(b == 0u ? job.blk0 : job.blk1) * row_bytes;
#pragma unroll
        for (uint32_t r = 0; r < 4u; ++r) bulk_load(dst + b * 512u * job.k2 + r * row_bytes, block + r * row_pitch, row_bytes, full);
      }
    };
    const uint32_t ahead = raws < k_stages ? raws : k_stages;
    if (elect_one()) {
      for (uint32_t it = 0; it < ahead; ++it) words(it, it);
    }
    __syncwarp();
    griddep_launch_dependents();
    griddep_wait();   // the rotated activations come from the kernel before
    RingAt at, next;
    for (uint32_t it = 0; it < k_stages; ++it, at.advance(1u, kStages)) {
      if (!mbar_wait(c.bars + 8u * (kStages + at.slot), at.phase ^ 1u)) {
        if (c.lane == 0) atomicOr(status, kStatusProducer);
        break;
      }
      // The MMAs of stage it - kStages have retired, so its words were decoded: their slot takes the stage `raws` further on.
      const bool refill = it >= kStages && it - kStages + raws < k_stages;
      if (elect_one()) {
        const uint32_t full = c.bars + 8u * at.slot, stage = c.base + at.slot * kStageBytes;
        const int32_t x = static_cast<int32_t>((job.stage0 + it) * 64u);
        mbar_expect_tx(full, row_tiles * kABytes);
        tma_load_2d(stage, map_a, full, x, static_cast<int32_t>(job.row0));
        if (row_tiles == 2u) tma_load_2d(stage + kABytes, map_a, full, x, static_cast<int32_t>(job.row0 + 128u));
        if (refill) words(it - kStages + raws, next.slot);
      }
      __syncwarp();
      if (refill) next.advance(1u, raws);
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

// Both steps back to back.
template <int DW>
__device__ __forceinline__ bool core_run(const Core &c, const Job &job, const CUtensorMap *map_a, uint32_t *status) {
  const bool decoded = core_roles<DW>(c, job, map_a, status);
  return c.warp < DW ? core_accumulator<DW>(c, decoded, status) : false;
}

// ---- epilogue ------------------------------------------------------------------------------------
// A warp group (warp / 4: four warps, 128 threads = the 128 rows of a row tile, a warp's lanes the
// rows 32 (warp % 4) .. + 31) owns 32 KB of the idle stage ring as [value 64][row 128] floats. The
// row's low five bits are XORed with the value index, so a warp's accesses are free of bank
// conflicts both when its lanes are 32 rows of one value (a thread parking its row) and when they
// are 32 values of one row (the warp writing a row out).
__device__ __forceinline__ uint32_t stash_at(uint32_t i, uint32_t t) { return i * 128u + (t & 96u) + ((t ^ i) & 31u); }

// Hands the calling warp's first `rows` rows of 64 parked values to `emit(r, lo, hi)`: lane l gets
// values l and l + 32 of row r, so what the caller stores per row is contiguous across the warp.
// (A thread storing its own row touches 32 different lines per instruction, and the memory pipe
// takes them one per cycle: the row-wise form is what makes the epilogue short.)
template <class RowEmit>
__device__ __forceinline__ void emit_rows(const float *area, uint32_t quad, uint32_t lane, uint32_t rows, RowEmit emit) {
  for (uint32_t r = 0; r < rows; ++r) {
    const uint32_t t = quad * 32u + r;
    emit(r, area[stash_at(lane, t)], area[stash_at(lane + 32u, t)]);
  }
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

// The epilogue of one (row tile, block) item for the calling warp: a thread owns one row (lane =
// row 32 quad + lane of the row tile; `rows` of the warp's 32 exist, `valid` = lane < rows) and
// `taddr` is the tensor-memory address of the block's first column in those lanes. The thread
// applies `inv` and six Hadamard stages to each half of its 128 columns in registers, the seventh
// stage combines the halves through `area`, and `emit(pass, r, lo, hi)` receives, a row at a
// time, columns 64 pass + lane (lo) and 64 pass + 32 + lane (hi), 1 / sqrt(128) included.
template <class RowEmit>
__device__ __forceinline__ void block_epilogue(uint32_t taddr, float inv, bool valid, float *area, uint32_t quad, uint32_t lane,
                                               uint32_t rows, RowEmit emit) {
  const uint32_t t = quad * 32u + lane;
  float v[64];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    load_half_row(taddr + 64u * half, inv, v);
    if (valid) {
      hadamard64_regs(v);
      if (half == 0) {
#pragma unroll
        for (int i = 0; i < 64; ++i) area[stash_at(i, t)] = v[i];
      }
    }
  }
  const float c = 0.08838834764831845f;   // 1 / sqrt(128)
  if (valid) {   // the seventh stage: columns i (sum, parked) and 64 + i (difference, kept)
#pragma unroll
    for (int i = 0; i < 64; ++i) {
      const float a = area[stash_at(i, t)], b = v[i];
      area[stash_at(i, t)] = (a + b) * c;
      v[i] = (a - b) * c;
    }
  }
  __syncwarp();
  emit_rows(area, quad, lane, rows, [&](uint32_t r, float lo, float hi) { emit(0u, r, lo, hi); });
  __syncwarp();
  if (valid) {
#pragma unroll
    for (int i = 0; i < 64; ++i) area[stash_at(i, t)] = v[i];
  }
  __syncwarp();
  emit_rows(area, quad, lane, rows, [&](uint32_t r, float lo, float hi) { emit(1u, r, lo, hi); });
}

// The same for a job of one row tile, where only two of the four warp groups would have a block:
// groups g and g ^ 2 share block g & 1, a thread owning 64 columns of its row (half = g >> 1). Each
// transforms its half and parks it in its group's area (`mine`); all decoder warps meet at barrier 1;
// the seventh stage gives the first half's owner columns 0..63 (sums) and the other's columns
// 64..127 (differences), parked again after a second meeting and written out row-wise:
// `emit(half, r, lo, hi)` as above. Every decoder warp calls this exactly once (`live`: the group's
// block exists - warp-uniform).
template <int DW, class RowEmit>
__device__ __forceinline__ void half_epilogue(uint32_t taddr_block, uint32_t half, bool live, float inv, bool valid, float *mine,
                                              const float *other, uint32_t quad, uint32_t lane, uint32_t rows, RowEmit emit) {
  const uint32_t t = quad * 32u + lane;
  float v[64];
  if (live) {
    load_half_row(taddr_block + 64u * half, inv, v);
    if (valid) {
      hadamard64_regs(v);
#pragma unroll
      for (int i = 0; i < 64; ++i) mine[stash_at(i, t)] = v[i];
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
  const float c = 0.08838834764831845f;   // 1 / sqrt(128)
  if (live && valid) {
#pragma unroll
    for (int i = 0; i < 64; ++i) {
      const float o = other[stash_at(i, t)];
      v[i] = half == 0u ? (v[i] + o) * c : (o - v[i]) * c;
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
  if (!live) return;
  if (valid) {
#pragma unroll
    for (int i = 0; i < 64; ++i) mine[stash_at(i, t)] = v[i];
  }
  __syncwarp();
  emit_rows(mine, quad, lane, rows, [&](uint32_t r, float lo, float hi) { emit(half, r, lo, hi); });
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
