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
//  * A CTA owns one block of 128 output columns (the MMA's M: a column is a lane of the accumulator) and up to 192 or 384 rows
//    (its N, as few as there are in steps of 16), and walks `in` in stages of 64: two shapes, below.
//  * The decoded weights are the MMA's A operand and go to TENSOR MEMORY: groups of four decoder warps take the stages in
//    turn; a warp decodes two tile columns of four tiles each (trellis_device.cuh: funnel shifts, IMAD, DP4A, half an HFMA2
//    per weight) and stores a column with one tcgen05.st 16x128b - the eight values of a lane are that shape's fragment as
//    they are. (Decoded to shared memory, with the rows as A, a stage moved 56 KB through the 128-byte port for 512 cycles of
//    MMAs: writes of the tile, its reads by two row tiles and theirs, and the rows' arrival.)
//  * One warp brings the packed words through a ring in shared memory by bulk copies, ahead of the previous kernel's end; one
//    the rows' fp16 activations by TMA (128-byte swizzle); one issues tcgen05.mma kind::f16 (M 128, K 16; fp16 x fp16, fp32
//    accumulation in tensor memory) from an elected lane.
//  * The epilogue turns the accumulator round through the (by then idle) rings: a thread stores its column's sums there, a
//    warp then reads eight rows, four lanes a row, in 16-byte pieces, and applies the Hadamard transform, the row's inverse
//    scale, svh and the caller's epilogue. The CTAs of a cluster that shares K push their sums to the rank that finishes a row.
//  * Every mbarrier wait is bounded; a wait that runs out sets a bit of a status word and the CTA
//    falls through to the common exit and frees its tensor memory.
#ifndef B200Q_TRELLIS_TC_CUH
#define B200Q_TRELLIS_TC_CUH

#include "nvfp4_tc.cuh"
#include "trellis_device.cuh"

namespace b200q {
namespace trellis_tc {

using namespace trellis_dev;

constexpr uint32_t kStageCols = 32;                // tensor-memory columns of a decoded stage: 128 lanes x 64 fp16
constexpr uint32_t kMaxStages = 8;
constexpr uint32_t kMaxRanks = 8;                  // the CTAs of a cluster that share the K stages of an item

// Two shapes of the CTA, by its groups of four decoder warps (which run the epilogue too). Two groups: up to 192 rows, half of
// an SM, so that one CTA's setup, fill and epilogue run under the other's decoding. Four: up to 384 rows, so that a decoded
// stage serves twice as many, a CTA per SM.
template <int GROUPS>
struct Shape {
  static constexpr int kDecoderWarps = 4 * GROUPS;
  static constexpr int kThreads = (kDecoderWarps + 3) * 32;               // and a warp each for the rows, the MMAs and the packed words
  static constexpr uint32_t kMaxRows = GROUPS == 2 ? 192 : 384;
  static constexpr uint32_t kTmemCols = GROUPS == 2 ? 256 : 512;          // the accumulator and the decoded stages
  static constexpr uint32_t kRingBytes = (GROUPS == 2 ? 110 : 212) * 1024;
  static constexpr uint32_t kWordBytes = (GROUPS == 2 ? 36 : 48) * 1024;  // of them for packed words, at most
  static constexpr uint32_t kSmemBytes = kRingBytes + 8u * (2u * (2u * kMaxStages + 4u) + 2u) + 16u + 1024u;   // + barriers, the tensor-memory slot, alignment slack
  static_assert((kMaxRows + kMaxRanks - 1u) * 512u <= kRingBytes, "the epilogue's sums fit into the rings, in whole turns of a cluster");
};
constexpr uint32_t kStatusProducer = 1u, kStatusMma = 2u, kStatusEpilogue = 4u, kStatusDecoder = 8u;

// What one CTA multiplies: rows [row0, row0 + rows) of the rotated activations (as many as its shape takes) with
// one 128-column block of one trellis plane.
struct Job {
  const uint32_t *trellis;  // the plane: tile (tk, tn) at word (tk * tile_stride + tn) * 4 k2
  uint32_t k2;
  uint32_t tile_stride;     // tiles per stored row of the plane
  uint32_t blk;             // the 128-column block
  uint32_t row0, rows;      // row0 is also the TMA row coordinate
  uint32_t box;             // rows of one TMA load (a multiple of 8)
  uint32_t stage0, stage1;  // the K stages of 64 inputs it walks: all of `in`, or the CTA's share of a cluster's
};

// A cluster that shares a job's K stages: rank r finishes the rows r, r + ranks, ...
struct Split {
  uint32_t ranks, rank;
};
constexpr Split kWhole = {1u, 0u};

struct Core {
  uint32_t base, words, bars, tmem, tmem_a;
  uint32_t n, x_bytes, x_stages, word_bytes, w_stages, a_slots;
  uint8_t *base_ptr;
  int warp, lane;
  __device__ __forceinline__ uint32_t x_full() const { return bars; }
  __device__ __forceinline__ uint32_t x_empty() const { return bars + 8u * kMaxStages; }
  __device__ __forceinline__ uint32_t w_full() const { return bars + 16u * kMaxStages; }
  __device__ __forceinline__ uint32_t w_empty() const { return bars + 24u * kMaxStages; }
  __device__ __forceinline__ uint32_t a_full() const { return bars + 32u * kMaxStages; }
  __device__ __forceinline__ uint32_t a_empty() const { return bars + 32u * kMaxStages + 32u; }
  __device__ __forceinline__ uint32_t acc() const { return bars + 32u * kMaxStages + 64u; }
  __device__ __forceinline__ uint32_t sums() const { return bars + 32u * kMaxStages + 72u; }
};

template <int GROUPS>
__device__ __forceinline__ Core core_setup(uint8_t *smem_raw, const Job &job, const Split split) {
  constexpr uint32_t kRingBytes = Shape<GROUPS>::kRingBytes, kWordBytes = Shape<GROUPS>::kWordBytes, kTmemCols = Shape<GROUPS>::kTmemCols;
  constexpr int kDecoderWarps = Shape<GROUPS>::kDecoderWarps;
  Core c;
  const uint32_t raw = smem_u32(smem_raw);
  c.base = (raw + 1023u) & ~1023u;   // the 128-byte swizzle wants 1024-byte aligned tiles
  c.base_ptr = smem_raw + (c.base - raw);
  c.bars = c.base + kRingBytes;
  c.warp = uniform_warp();
  c.lane = threadIdx.x & 31;
  c.n = (job.rows + 15u) / 16u * 16u;
  c.x_bytes = (job.rows + job.box - 1u) / job.box * job.box * 128u;
  c.word_bytes = 512u * job.k2;
  c.w_stages = min(kMaxStages, kWordBytes / c.word_bytes);
  c.x_stages = min(kMaxStages, (kRingBytes - c.w_stages * c.word_bytes) / c.x_bytes);
  c.words = c.base + c.x_stages * c.x_bytes;
  const uint32_t acc_cols = (c.n + 31u) / 32u * 32u;
  c.a_slots = min(4u, (kTmemCols - acc_cols) / kStageCols);
  uint32_t *slot = reinterpret_cast<uint32_t *>(c.base_ptr + kRingBytes + 32u * kMaxStages + 80u);
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kMaxStages; ++s) {
      mbar_init(c.x_full() + 8u * s, 1);    // the producers' expect_tx arrivals, the MMA warp's commits
      mbar_init(c.x_empty() + 8u * s, 1);
      mbar_init(c.w_full() + 8u * s, 1);
      mbar_init(c.w_empty() + 8u * s, 4);   // the four warps of the group that decodes the stage
    }
    for (uint32_t s = 0; s < 4u; ++s) {
      mbar_init(c.a_full() + 8u * s, 4);
      mbar_init(c.a_empty() + 8u * s, 1);
    }
    mbar_init(c.acc(), 1);
    mbar_init(c.sums(), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // every rank of the cluster sends its sums of the rows that this one finishes
    if (split.ranks > 1u) mbar_expect_tx(c.sums(), split.ranks * ((job.rows + split.ranks - 1u - split.rank) / split.ranks) * 512u);
  }
  if (c.warp == kDecoderWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  c.tmem = __shfl_sync(0xFFFFFFFFu, *slot, 0);
  c.tmem_a = c.tmem + acc_cols;
  return c;
}

__device__ __forceinline__ uint32_t lds_word(uint32_t address) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(address));
  return v;
}
// 16 lanes x 32 columns: register 2 i (+ 1) of lane 4 g + t is row g (+ 8), column 4 i + t.
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t addr, const uint32_t *r) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t addr, const uint32_t *r) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// The decoder warps' loop: group g (warp / 4) takes the job's stages g, g + GROUPS, ...; warp w of it the tile columns 2 w and
// 2 w + 1 of the block, whose values are lanes 32 w .. + 31 of the MMA's A operand.
template <int K2, int GROUPS>
__device__ __forceinline__ bool decode_stages(const Core &c, const Job &job, uint32_t *status) {
  const LaneWindow win = lane_window(K2, c.lane);
  const uint32_t quad = static_cast<uint32_t>(c.warp) & 3u, group = static_cast<uint32_t>(c.warp) >> 2;
  const uint32_t k_stages = job.stage1 - job.stage0;
  // the lane's words of the warp's first tile column inside a stage of the ring, as byte addresses
  const uint32_t column = c.words + quad * 32u * K2;
  const uint32_t at0 = column + 4u * win.w0, at1 = column + 4u * win.w1, at2 = column + 4u * win.w2;
  const uint32_t lanes = c.tmem_a + (quad << 21);
  RingAt from, to;
  from.step(group, c.w_stages);
  to.step(group, c.a_slots);
  for (uint32_t it = group; it < k_stages; it += GROUPS, from.step(GROUPS, c.w_stages), to.step(GROUPS, c.a_slots)) {
    if (!mbar_wait(c.w_full() + 8u * from.slot, from.phase)) {
      if (c.lane == 0) atomicOr(status, kStatusDecoder);
      return false;
    }
    const uint32_t stage = from.slot * (512u * K2), cols = lanes + to.slot * kStageCols;
    // Tiles in one body of code: all eight of the warp's stage where decoding is the bound (two at a time: 213 us against 192
    // for 5120 -> 17408 at 1000 tokens), two where the MMAs are and the long body only misses the instruction cache (17408 ->
    // 5120 at 1000 tokens in the shape of four groups: 186 us with eight, 168 with two).
    constexpr uint32_t kTiles = GROUPS == 2 ? 8u : 2u;
    bool ok = true;
#pragma unroll 1
    for (uint32_t first = 0; first < 8u; first += kTiles) {
      uint32_t frag[4 * kTiles];
#pragma unroll
      for (uint32_t r = 0; r < kTiles; ++r) {   // tile (first + r) / 4 of a row, (first + r) % 4 of the stage's four rows (16 inputs each, eight tile columns apart)
        const uint32_t off = stage + ((first + r) >> 2) * 16u * K2 + ((first + r) & 3u) * 128u * K2;
        uint32_t f[4];
        decode8<K2>(lds_word(at0 + off), lds_word(at1 + off), lds_word(at2 + off), win.off, f);
        frag[4 * r] = f[0];       // inputs 2 t, 2 t + 1, column g
        frag[4 * r + 1] = f[2];   // column g + 8
        frag[4 * r + 2] = f[1];   // inputs 2 t + 8, 2 t + 9
        frag[4 * r + 3] = f[3];
      }
      if (first == 0u) {
        ok = mbar_wait(c.a_empty() + 8u * to.slot, to.phase ^ 1u);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      if constexpr (kTiles == 8u) {
        tmem_st_16x128b_x8(cols, frag);
        tmem_st_16x128b_x8(cols + (16u << 16), frag + 16);
      } else {
        tmem_st_16x128b_x4(cols + ((first >> 2) << 20) + (first & 3u) * 8u, frag);
      }
    }
    if (!ok) {
      if (c.lane == 0) atomicOr(status, kStatusDecoder);
      return false;
    }
    __syncwarp();
    if (c.lane == 0) mbar_arrive(c.w_empty() + 8u * from.slot);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (c.lane == 0) mbar_arrive(c.a_full() + 8u * to.slot);
  }
  return true;
}

// Runs the CTA's roles: the producers and the MMA warp to their end, the decoder warps through
// their K stages. Returns true in a decoder warp that decoded all of them; such a warp has time for
// loads of its own (what its epilogue will need) before it calls core_accumulator, while the last
// MMAs retire.
template <int GROUPS>
__device__ __forceinline__ bool core_roles(const Core &c, const Job &job, const CUtensorMap *map_rows, uint32_t *status) {
  constexpr int kDecoderWarps = Shape<GROUPS>::kDecoderWarps;
  const uint32_t k_stages = job.stage1 - job.stage0;
  griddep_launch_dependents();
  if (c.warp < kDecoderWarps) {
    bool decoded;
    switch (job.k2) {
      case 4: decoded = decode_stages<4, GROUPS>(c, job, status); break;
      case 5: decoded = decode_stages<5, GROUPS>(c, job, status); break;
      case 6: decoded = decode_stages<6, GROUPS>(c, job, status); break;
      case 8: decoded = decode_stages<8, GROUPS>(c, job, status); break;
      case 10: decoded = decode_stages<10, GROUPS>(c, job, status); break;
      default: decoded = decode_stages<12, GROUPS>(c, job, status); break;
    }
    griddep_wait();   // the epilogue touches what an earlier kernel wrote
    return decoded;
  }
  if (c.warp == kDecoderWarps) {
    // ---- producer of the rows ----
    griddep_wait();   // the rotated activations come from the kernel before
    const uint32_t boxes = c.x_bytes / (job.box * 128u);
    RingAt at;
    for (uint32_t it = 0; it < k_stages; ++it, at.step(1u, c.x_stages)) {
      if (!mbar_wait(c.x_empty() + 8u * at.slot, at.phase ^ 1u)) {
        if (c.lane == 0) atomicOr(status, kStatusProducer);
        break;
      }
      if (elect_one()) {
        const uint32_t full = c.x_full() + 8u * at.slot, stage = c.base + at.slot * c.x_bytes;
        const int32_t x = static_cast<int32_t>((job.stage0 + it) * 64u);
        mbar_expect_tx(full, c.x_bytes);
        for (uint32_t b = 0; b < boxes; ++b) tma_load_2d(stage + b * job.box * 128u, map_rows, full, x, static_cast<int32_t>(job.row0 + b * job.box));
      }
      __syncwarp();
    }
  } else if (c.warp == kDecoderWarps + 2) {
    // ---- producer of the packed words: lane r copies the eight tiles of tile row r; they never depend on the previous kernel ----
    const uint64_t row_pitch = static_cast<uint64_t>(job.tile_stride) * 16u * job.k2;   // bytes from a tile row to the next
    const uint8_t *src = reinterpret_cast<const uint8_t *>(job.trellis) + static_cast<uint64_t>(job.blk) * 128u * job.k2 +
                         (static_cast<uint64_t>(job.stage0) * 4u + static_cast<uint32_t>(c.lane)) * row_pitch;
    RingAt at;
    for (uint32_t it = 0; it < k_stages; ++it, at.step(1u, c.w_stages), src += 4u * row_pitch) {
      if (!mbar_wait(c.w_empty() + 8u * at.slot, at.phase ^ 1u)) {
        if (c.lane == 0) atomicOr(status, kStatusProducer);
        break;
      }
      const uint32_t full = c.w_full() + 8u * at.slot;
      if (c.lane == 0) mbar_expect_tx(full, c.word_bytes);
      __syncwarp();
      if (c.lane < 4) bulk_load(c.words + at.slot * c.word_bytes + static_cast<uint32_t>(c.lane) * 128u * job.k2, src, 128u * job.k2, full);
    }
  } else {
    // ---- MMA issuer: the whole warp runs the loop, an elected lane issues (elect_one, nvfp4_tc.cuh) ----
    // instruction descriptor: FP32 accumulator (bit 4), A and B FP16 (format 0), both K-major,
    // N >> 3 at bit 17, M >> 4 at bit 24; more than 256 rows are two MMAs
    const uint32_t n0 = c.n > 256u ? (c.n / 2u + 31u) / 32u * 32u : c.n, n1 = c.n - n0;
    const uint32_t idesc = (1u << 4) | ((128u >> 4) << 24);
    const uint64_t desc0 = smem_desc_sw128(c.base);
    bool ok = true;
    RingAt at, from;
    for (uint32_t it = 0; it < k_stages; ++it, at.step(1u, c.a_slots), from.step(1u, c.x_stages)) {
      if (!mbar_wait(c.x_full() + 8u * from.slot, from.phase) || !mbar_wait(c.a_full() + 8u * at.slot, at.phase)) {
        if (c.lane == 0) atomicOr(status, kStatusMma);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint32_t a = c.tmem_a + at.slot * kStageCols;
        const uint64_t b = desc0 + from.slot * (c.x_bytes >> 4);
#pragma unroll
        for (uint32_t kb = 0; kb < 4; ++kb) {   // 16 values along K: 8 columns of A, two 16-byte units of the rows further
          mma_f16_ts(c.tmem, a + 8u * kb, b + 2u * kb, idesc | ((n0 >> 3) << 17), (it | kb) != 0u ? 1u : 0u);
          if (GROUPS == 4 && n1 != 0u) mma_f16_ts(c.tmem + n0, a + 8u * kb, b + n0 * 8u + 2u * kb, idesc | ((n1 >> 3) << 17), (it | kb) != 0u ? 1u : 0u);
        }
        mma_commit(c.a_empty() + 8u * at.slot);
        mma_commit(c.x_empty() + 8u * from.slot);
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(c.acc());
    __syncwarp();
  }
  return false;
}

// ---- epilogue ------------------------------------------------------------------------------------

__device__ __forceinline__ float4 four_halves(const uint2 raw) {
  const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// Waits for the accumulator and hands the job's finished rows to the decoder warps: `ask(r)` gives what the epilogue needs of
// row r, `old(asked, col)` requests what it reads at columns col .. + 3, `emit(asked, col, old, v)` takes those columns, the
// Hadamard transform with 1 / sqrt(128) and the row's inverse scale (`inv(r)`) included. With four groups, whose jobs have many
// rows, a warp takes eight rows, lane l eight times four columns of row l % 8; with two a warp takes a row, four columns a lane
// (jobs of some dozens of rows leave warps without any in eights: the experts of 4096 tokens 1214 us a block against 1188).
// All threads of the CTA call it; `decoded` is what core_roles returned to them.
//
// A row's sums lie in 512 bytes of the rings, the 16-byte pieces exchanged by the low bits of the row's place, so that the
// eight lanes of a phase of the 16-byte reads (eight rows, one piece) meet eight different bank groups.
//
// Without a cluster the sums go through this CTA's own rings. With one, every CTA pushes its share of row r's sums (the
// transform is linear) to rank r % ranks once the rings of all are idle, and nobody reads another CTA's memory.
__device__ __forceinline__ uint32_t sums_at(uint32_t place, uint32_t piece) { return place * 512u + ((piece ^ (place & 7u)) << 4); }

template <int GROUPS, class Inv, class Ask, class Old, class Emit>
__device__ __forceinline__ void core_finish_rows(const Core &c, const Job &job, const Split split, bool decoded, uint32_t *status, Inv inv, Ask ask, Old old, Emit emit) {
  constexpr int kDecoderWarps = Shape<GROUPS>::kDecoderWarps;
  const uint32_t quad = static_cast<uint32_t>(c.warp) & 3u, group = static_cast<uint32_t>(c.warp) >> 2, lane = static_cast<uint32_t>(c.lane);
  const bool works = c.warp < kDecoderWarps;
  bool have = false;
  if (works) {
    if (decoded) {
      have = mbar_wait(c.acc(), 0u);
      if (!have && lane == 0u) atomicOr(status, kStatusEpilogue);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (split.ranks > 1u) cluster_sync_all();   // the rings of every CTA are idle
  if (works) {
    const uint32_t turns = (job.rows + split.ranks - 1u) / split.ranks;
    const uint32_t piece = quad * 8u + (lane >> 2), in_piece = (lane & 3u) * 4u;   // the thread's column in a row's 512 bytes
    for (uint32_t r0 = group * 32u; r0 < job.rows; r0 += GROUPS * 32u) {
      uint32_t v[32];
      if (have) {
        tmem_ld32(c.tmem + ((quad * 32u) << 16) + r0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
      if (split.ranks == 1u) {
        uint8_t *dst = c.base_ptr + in_piece;
#pragma unroll
        for (uint32_t j = 0; j < 32u; ++j) *reinterpret_cast<float *>(dst + r0 * 512u + sums_at(j, piece)) = have ? __uint_as_float(v[j]) : 0.0f;
      } else {   // place [sender][turn]
        uint32_t to = r0 % split.ranks, place = split.rank * turns + r0 / split.ranks;
#pragma unroll
        for (uint32_t j = 0; j < 32u; ++j) {
          if (r0 + j >= job.rows) break;
          push_f32(cluster_map(c.base + sums_at(place, piece) + in_piece, to), have ? __uint_as_float(v[j]) : 0.0f, cluster_map(c.sums(), to));
          if (++to == split.ranks) to = 0u, ++place;
        }
      }
    }
    if (split.ranks == 1u) {
      // either every decoder warp has its accumulator or none goes on
      uint32_t all;
      asm volatile("{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.and.pred q, 1, %2, p; selp.u32 %0, 1, 0, q; }"
                   : "=r"(all) : "r"(static_cast<uint32_t>(have)), "n"(kDecoderWarps * 32) : "memory");
      have = all != 0u;
    } else {
      have = mbar_wait_pushed(c.sums());
      if (!have && lane == 0u) atomicOr(status, kStatusEpilogue);
    }
    const uint32_t mine = (job.rows + split.ranks - 1u - split.rank) / split.ranks;   // rows this CTA finishes: rank, rank + ranks, ...
    auto sum_of = [&](uint32_t i, uint32_t unit) {
      float4 sum = *reinterpret_cast<const float4 *>(c.base_ptr + sums_at(i, unit));
      for (uint32_t q = 1; q < split.ranks; ++q) {   // in rank order
        const float4 more = *reinterpret_cast<const float4 *>(c.base_ptr + sums_at(q * turns + i, unit));
        sum.x += more.x, sum.y += more.y, sum.z += more.z, sum.w += more.w;
      }
      return sum;
    };
    if constexpr (GROUPS == 4) {
      for (uint32_t i0 = static_cast<uint32_t>(c.warp) * 8u; have && i0 < mine; i0 += 8u * kDecoderWarps) {
        const uint32_t i = i0 + (lane & 7u), at = min(i, mine - 1u), r = at * split.ranks + split.rank, q = lane >> 3;
        const auto asked = ask(r);
        decltype(old(asked, 0u)) was[8];
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u) was[u] = old(asked, 16u * u + 4u * q);
        const float scale = inv(r) * kHadamardNorm;
        float2 v[8][2];
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u) {
          const float4 sum = sum_of(at, 4u * u + q);
          v[u][0] = make_float2(sum.x, sum.y);
          v[u][1] = make_float2(sum.z, sum.w);
        }
        hadamard_quad<8, 2>(v, c.lane, 8, 16);
        if (i < mine) {
#pragma unroll
          for (uint32_t u = 0; u < 8u; ++u)
            emit(asked, 16u * u + 4u * q, was[u], make_float4(v[u][0].x * scale, v[u][0].y * scale, v[u][1].x * scale, v[u][1].y * scale));
        }
      }
    } else {
      constexpr int kBatch = 4;   // rows in work at a time
      for (uint32_t i0 = static_cast<uint32_t>(c.warp); have && i0 < mine; i0 += kBatch * kDecoderWarps) {
        float v[kBatch][4], scale[kBatch];
        decltype(ask(0u)) asked[kBatch];
        decltype(old(asked[0], 0u)) was[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const uint32_t i = min(i0 + b * kDecoderWarps, mine - 1u), r = i * split.ranks + split.rank;
          asked[b] = ask(r);
          was[b] = old(asked[b], 4u * lane);
          scale[b] = inv(r);
          const float4 sum = sum_of(i, lane);
          v[b][0] = sum.x, v[b][1] = sum.y, v[b][2] = sum.z, v[b][3] = sum.w;
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) hadamard128(v[b], c.lane);
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          if (i0 + b * kDecoderWarps >= mine) break;
          emit(asked[b], 4u * lane, was[b], make_float4(v[b][0] * scale[b], v[b][1] * scale[b], v[b][2] * scale[b], v[b][3] * scale[b]));
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (c.warp == kDecoderWarps + 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(Shape<GROUPS>::kTmemCols) : "memory");
  }
}

// The rotated activations [rows][in] fp16 as a 2-D tensor with boxes of `box` rows x 64 values, 128-byte swizzle.
inline bool make_rows_map(CUtensorMap *map, const void *rows_f16, uint64_t rows, uint64_t in, uint32_t box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {in, rows};
  const cuuint64_t strides[1] = {in * 2u};
  const cuuint32_t box[2] = {64u, box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(rows_f16), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace trellis_tc
}  // namespace b200q

#endif
