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
//  * A CTA owns one block of 128 output columns (the MMA's M: a column is a lane of the accumulator) and up to 192 rows (its
//    N, as few as there are in steps of 16), and walks `in` in stages of 64. Two CTAs share an SM, so that one's setup, fill
//    and epilogue run under the other's decoding.
//  * The decoded weights are the MMA's A operand and go to TENSOR MEMORY: two groups of four decoder warps take the stages in
//    turn; a warp decodes two tile columns of four tiles each (trellis_device.cuh: funnel shifts, IMAD, DP4A, half an HFMA2
//    per weight) and stores a column with one tcgen05.st 16x128b - the eight values of a lane are that shape's fragment as
//    they are. (Decoded to shared memory, with the rows as A, a stage moved 56 KB through the 128-byte port for 512 cycles of
//    MMAs: writes of the tile, its reads by two row tiles and theirs, and the rows' arrival.)
//  * One warp brings the packed words through a ring in shared memory by bulk copies, ahead of the previous kernel's end; one
//    the rows' fp16 activations by TMA (128-byte swizzle); one issues tcgen05.mma kind::f16 (M 128, K 16; fp16 x fp16, fp32
//    accumulation in tensor memory) from an elected lane.
//  * The epilogue turns the accumulator round through the (by then idle) rings: a thread stores its column's sums there, a
//    warp then reads a row, 128 columns in 16-byte pieces, and applies the Hadamard transform, the row's inverse scale, svh
//    and the caller's epilogue. The CTAs of a cluster that shares K push their sums to the rank that finishes a row.
//  * Every mbarrier wait is bounded; a wait that runs out sets a bit of a status word and the CTA
//    falls through to the common exit and frees its tensor memory.
#ifndef B200Q_TRELLIS_TC_CUH
#define B200Q_TRELLIS_TC_CUH

#include "nvfp4_tc.cuh"
#include "trellis_device.cuh"

namespace b200q {
namespace trellis_tc {

using namespace trellis_dev;

constexpr uint32_t kMaxRows = 192;                 // rows of a CTA
constexpr int kDecoderWarps = 8;                   // two groups of four; they run the epilogue too
constexpr int kThreads = (kDecoderWarps + 3) * 32; // and a warp each for the rows, the MMAs and the packed words
constexpr uint32_t kTmemCols = 256;                // per CTA: the accumulator and the decoded stages
constexpr uint32_t kStageCols = 32;                // a decoded stage: 128 lanes x 64 fp16
constexpr uint32_t kRingBytes = 110 * 1024;        // the rings of one CTA
constexpr uint32_t kWordBytes = 36 * 1024;         // of them for packed words, at most
constexpr uint32_t kMaxStages = 8;
constexpr uint32_t kSmemBytes = kRingBytes + 8u * (2u * (2u * kMaxStages + 4u) + 2u) + 16u + 1024u;   // + barriers, the tensor-memory slot, alignment slack
static_assert(kMaxRows * 512u <= kRingBytes, "the epilogue's sums fit into the rings");
constexpr uint32_t kStatusProducer = 1u, kStatusMma = 2u, kStatusEpilogue = 4u, kStatusDecoder = 8u;

// What one CTA multiplies: rows [row0, row0 + rows) of the rotated activations (rows <= 192) with
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

__device__ __forceinline__ Core core_setup(uint8_t *smem_raw, const Job &job, const Split split) {
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
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
// kind::f16 with A in tensor memory: row r in lane r, two values of K a column.
__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{ .reg .pred p; setp.ne.u32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
               : "memory");
}

// The decoder warps' loop: group g (warp / 4) takes the job's stages g, g + 2, ...; warp w of it the tile columns 2 w and
// 2 w + 1 of the block, whose values are lanes 32 w .. + 31 of the MMA's A operand.
template <int K2>
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
  for (uint32_t it = group; it < k_stages; it += 2u, from.step(2u, c.w_stages), to.step(2u, c.a_slots)) {
    if (!mbar_wait(c.w_full() + 8u * from.slot, from.phase)) {
      if (c.lane == 0) atomicOr(status, kStatusDecoder);
      return false;
    }
    const uint32_t stage = from.slot * (512u * K2);
    uint32_t frag[2][16];
#pragma unroll
    for (int col = 0; col < 2; ++col) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {   // tile rows of the stage: 16 inputs each, eight tile columns apart
        const uint32_t off = stage + r * 128u * K2 + col * 16u * K2;
        uint32_t f[4];
        decode8<K2>(lds_word(at0 + off), lds_word(at1 + off), lds_word(at2 + off), win.off, f);
        frag[col][4 * r] = f[0];       // inputs 2 t, 2 t + 1, column g
        frag[col][4 * r + 1] = f[2];   // column g + 8
        frag[col][4 * r + 2] = f[1];   // inputs 2 t + 8, 2 t + 9
        frag[col][4 * r + 3] = f[3];
      }
    }
    __syncwarp();
    if (c.lane == 0) mbar_arrive(c.w_empty() + 8u * from.slot);
    if (!mbar_wait(c.a_empty() + 8u * to.slot, to.phase ^ 1u)) {
      if (c.lane == 0) atomicOr(status, kStatusDecoder);
      return false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem_st_16x128b_x8(lanes + to.slot * kStageCols, frag[0]);
    tmem_st_16x128b_x8(lanes + (16u << 16) + to.slot * kStageCols, frag[1]);
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
__device__ __forceinline__ bool core_roles(const Core &c, const Job &job, const CUtensorMap *map_rows, uint32_t *status) {
  const uint32_t k_stages = job.stage1 - job.stage0;
  griddep_launch_dependents();
  if (c.warp < kDecoderWarps) {
    bool decoded;
    switch (job.k2) {
      case 4: decoded = decode_stages<4>(c, job, status); break;
      case 5: decoded = decode_stages<5>(c, job, status); break;
      case 6: decoded = decode_stages<6>(c, job, status); break;
      case 8: decoded = decode_stages<8>(c, job, status); break;
      case 10: decoded = decode_stages<10>(c, job, status); break;
      default: decoded = decode_stages<12>(c, job, status); break;
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
    // N >> 3 at bit 17, M >> 4 at bit 24
    const uint32_t idesc = (1u << 4) | ((c.n >> 3) << 17) | ((128u >> 4) << 24);
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
          mma_f16_ts(c.tmem, a + 8u * kb, b + 2u * kb, idesc, (it | kb) != 0u ? 1u : 0u);
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

__device__ __forceinline__ float4 four_halves(const uint16_t *p) {
  const uint2 raw = __ldg(reinterpret_cast<const uint2 *>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// Waits for the accumulator and hands the job's finished rows to the decoder warps, a warp per row: `ask(r)` requests what the
// epilogue of row r reads (several rows' requests and transforms travel together), `emit(r, asked, v)` takes columns 4 lane ..
// + 3 of row r, the Hadamard transform with 1 / sqrt(128) and the row's inverse scale (`inv(r)`) included. All threads of the
// CTA call it; `decoded` is what core_roles returned to them.
//
// Without a cluster the sums go through this CTA's own rings. With one, every CTA pushes its share of row r's sums (the
// transform is linear) to rank r % ranks once the rings of all are idle, and nobody reads another CTA's memory.
template <class Inv, class Ask, class Emit>
__device__ __forceinline__ void core_finish_rows(const Core &c, const Job &job, const Split split, bool decoded, uint32_t *status, Inv inv, Ask ask, Emit emit) {
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
    const uint32_t column = (quad * 32u + lane) * 4u;   // the thread's column of a row's 512 bytes
    for (uint32_t r0 = group * 32u; r0 < job.rows; r0 += 64u) {
      uint32_t v[32];
      if (have) {
        tmem_ld32(c.tmem + ((quad * 32u) << 16) + r0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
      if (split.ranks == 1u) {
        float *dst = reinterpret_cast<float *>(c.base_ptr + r0 * 512u + column);
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[j * 128] = have ? __uint_as_float(v[j]) : 0.0f;
      } else {   // [sender][turn][128 columns]
        uint32_t to = r0 % split.ranks, at = c.base + (split.rank * turns + r0 / split.ranks) * 512u + column;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (r0 + j >= job.rows) break;
          push_f32(cluster_map(at, to), have ? __uint_as_float(v[j]) : 0.0f, cluster_map(c.sums(), to));
          if (++to == split.ranks) to = 0u, at += 512u;
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
    constexpr int kBatch = 4;
    const uint32_t mine = (job.rows + split.ranks - 1u - split.rank) / split.ranks;   // rows this CTA finishes: rank, rank + ranks, ...
    for (uint32_t i0 = static_cast<uint32_t>(c.warp); have && i0 < mine; i0 += kBatch * kDecoderWarps) {
      float v[kBatch][4];
      decltype(ask(0u)) asked[kBatch];
      float scale[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const uint32_t i = min(i0 + b * kDecoderWarps, mine - 1u), r = i * split.ranks + split.rank;
        asked[b] = ask(r);
        scale[b] = inv(r);
        float4 sum = *reinterpret_cast<const float4 *>(c.base_ptr + i * 512u + lane * 16u);
        for (uint32_t q = 1; q < split.ranks; ++q) {   // in rank order
          const float4 more = *reinterpret_cast<const float4 *>(c.base_ptr + (q * turns + i) * 512u + lane * 16u);
          sum.x += more.x, sum.y += more.y, sum.z += more.z, sum.w += more.w;
        }
        v[b][0] = sum.x, v[b][1] = sum.y, v[b][2] = sum.z, v[b][3] = sum.w;
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) hadamard128(v[b], c.lane);
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        if (i0 + b * kDecoderWarps >= mine) break;
        emit((i0 + b * kDecoderWarps) * split.ranks + split.rank, asked[b],
             make_float4(v[b][0] * scale[b], v[b][1] * scale[b], v[b][2] * scale[b], v[b][3] * scale[b]));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (c.warp == kDecoderWarps + 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(kTmemCols) : "memory");
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
