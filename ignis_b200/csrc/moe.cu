// Flash-Next mixture-of-experts ops: the entry points of include/ignis_moe.h and their kernels.
//
// Routed experts (the reference's ignis_moe_experts_prefill / _decode, kernel/src/moe_prefill.cu:
// 41-492 and moe_decode.cu:325-399): the (token, rank) assignments are grouped by expert on the
// device (count, scan, scatter) and cut into work items of at most 192 rows of one expert, which
// moe_tc.cu multiplies with the expert's records on the tensor cores at every size, the decode
// entry's included. (Warp-level kernels with the decoded tiles in registers stood here for up to 64
// tokens: 75.8 us against 66.4 at one token, 107.8 against 88 at eight, 258 against 210 at 64, 2048
// x 768 with 512 experts, ten of them a token.) Products are added to `acc` in 64-bit fixed point
// (2^-32), so the sum does not depend on arrival order. No CTA waits for another; a row's
// arithmetic does not depend on the item it is in, so the decode and prefill entries give the same
// bits.
//
// Nothing here traps or spins: a bad expert id, an absent record or an out-of-range contribution
// is skipped and recorded in the workspace's status word.
#include "../../include/ignis_moe.h"

#include "moe_internal.cuh"

#include <mutex>

namespace b200q {
namespace {

using Geometry = b200q_moe_geometry;
// The geometry the reference's own entry points (no geometry argument) work at: the reference
// compiles it in; here it starts at the reference's and b200q_moe_set_geometry replaces it.
Geometry g_default = {IGNIS_MOE_HIDDEN, IGNIS_MOE_INTERMEDIATE, IGNIS_MOE_EXPERTS, IGNIS_MOE_TOP_K};

constexpr uint32_t kMaxExperts = 4096;

int32_t check_geometry(ErrorSlot &slot, const Geometry *g, const char *what) {
  if (g == nullptr) return fail(slot, "%s: geometry is NULL", what);
  if (g->hidden == 0 || (g->hidden % 128u) != 0 || g->inter == 0 || (g->inter % 128u) != 0) {
    return fail(slot, "%s: hidden and inter must be positive multiples of 128", what);
  }
  if (g->experts == 0 || g->experts > kMaxExperts || g->top_k == 0 || g->top_k > 32u || g->top_k > g->experts) {
    return fail(slot, "%s: experts must lie in 1..4096 and top_k in 1..min(32, experts)", what);
  }
  if (g->hidden / 128u > 8u * 40u || g->inter / 128u > 8u * 40u) return fail(slot, "%s: dimension too long", what);
  return 0;
}

// Workspace regions for `tokens_max` tokens.
struct Layout {
  uint64_t status, counts, cursor, offsets, n_items, sorted, items, x_rows, x_scale, gu, h_rows, h_scale, down_rows, total;
  uint32_t rows_max, items_max;
};

uint64_t align256(uint64_t v) { return (v + 255u) & ~static_cast<uint64_t>(255u); }

uint32_t items_bound(const Geometry &g, uint32_t rows, uint32_t item_rows) {
  return rows / item_rows + (g.experts < rows ? g.experts : rows);
}

Layout layout_for(const Geometry &g, uint32_t tokens_max) {
  Layout l = {};
  l.rows_max = tokens_max * g.top_k;
  l.items_max = items_bound(g, l.rows_max, kMoeTcItemRows);
  const uint64_t rows = l.rows_max;
  uint64_t at = 0;
  l.status = at; at += 256;
  l.counts = at; at = align256(at + 4ull * g.experts);
  l.cursor = at; at = align256(at + 4ull * g.experts);
  l.offsets = at; at = align256(at + 4ull * (g.experts + 1));
  l.n_items = at; at += 256;
  l.sorted = at; at = align256(at + 4ull * rows);
  l.items = at; at = align256(at + 16ull * l.items_max);
  l.x_rows = at; at = align256(at + 2ull * rows * g.hidden);      // rotated x: fp16 [rows][hidden]
  l.x_scale = at; at = align256(at + 4ull * rows);                // inverse scale per row
  l.gu = at; at = align256(at + 8ull * rows * g.inter);           // fp32 [rows][2 inter]
  l.h_rows = at; at = align256(at + 2ull * rows * g.inter);       // rotated silu(g) u: fp16 [rows][inter]
  l.h_scale = at; at = align256(at + 4ull * rows);
  l.down_rows = at; at = align256(at + 4ull * rows * g.hidden);   // weighted down products: fp32 [tokens][top_k][hidden]
  l.total = at;
  return l;
}

// ---- grouping ------------------------------------------------------------------------------
// A CTA counts in shared memory and adds its counts to the experts' once: added one by one, a popular expert's rows queue at
// one address (13 us for 40 960 rows under Zipf routing).
constexpr uint32_t kSmallRows = 4096;

__global__ void __launch_bounds__(256) moe_count_kernel(const int32_t *ids, uint32_t rows, uint32_t experts,
                                                        uint32_t *counts, uint32_t *status) {
  __shared__ uint32_t mine[kMaxExperts];
  for (uint32_t e = threadIdx.x; e < experts; e += blockDim.x) mine[e] = 0u;
  __syncthreads();
  griddep_launch_dependents();
  griddep_wait();
  for (uint32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < rows; a += gridDim.x * blockDim.x) {
    const int32_t e = ids[a];
    if (e < 0 || static_cast<uint32_t>(e) >= experts) {
      if (e != IGNIS_MOE_NO_EXPERT) atomicOr(status, kStatusBadExpert);  // -1 is "no expert for this choice": skipped, not an error
    } else {
      atomicAdd(&mine[e], 1u);
    }
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < experts; e += blockDim.x) {
    if (mine[e] != 0u) atomicAdd(&counts[e], mine[e]);
  }
}

// One CTA: exclusive scans of the per-expert row and item counts, then the item list.
__global__ void __launch_bounds__(1024) moe_scan_kernel(const uint32_t *counts, uint32_t experts, uint32_t item_rows,
                                                        uint32_t *offsets, uint32_t *n_items, Item *items) {
  griddep_launch_dependents();
  griddep_wait();
  __shared__ uint32_t row_sum[1024], item_sum[1024];
  const uint32_t per = (experts + 1023u) / 1024u;  // experts per thread, consecutive
  const uint32_t e0 = threadIdx.x * per;
  uint32_t rows = 0, its = 0;
  for (uint32_t e = e0; e < e0 + per && e < experts; ++e) {
    rows += counts[e];
    its += (counts[e] + item_rows - 1u) / item_rows;
  }
  row_sum[threadIdx.x] = rows;
  item_sum[threadIdx.x] = its;
  __syncthreads();
  for (uint32_t d = 1; d < 1024; d <<= 1) {  // Hillis-Steele inclusive scan
    const uint32_t r = threadIdx.x >= d ? row_sum[threadIdx.x - d] : 0u;
    const uint32_t i = threadIdx.x >= d ? item_sum[threadIdx.x - d] : 0u;
    __syncthreads();
    row_sum[threadIdx.x] += r;
    item_sum[threadIdx.x] += i;
    __syncthreads();
  }
  uint32_t row_at = row_sum[threadIdx.x] - rows, item_at = item_sum[threadIdx.x] - its;
  for (uint32_t e = e0; e < e0 + per && e < experts; ++e) {
    offsets[e] = row_at;
    const uint32_t c = counts[e];
    for (uint32_t j = 0; j < c; j += item_rows) {
      items[item_at++] = Item{e, row_at + j, c - j < item_rows ? c - j : item_rows, 0u};
    }
    row_at += c;
  }
  if (threadIdx.x == 1023) {
    offsets[experts] = row_sum[1023];
    n_items[0] = item_sum[1023];
  }
}

// The rows of one expert are independent of each other, so their order inside the group does not change any output bit. A
// CTA's rows of an expert take their places together, as they were counted.
__global__ void __launch_bounds__(256) moe_scatter_kernel(const int32_t *ids, uint32_t rows, uint32_t experts,
                                                          const uint32_t *offsets, uint32_t *cursor, uint32_t *sorted) {
  __shared__ uint32_t mine[kMaxExperts];   // rows of the CTA, then their first place
  for (uint32_t e = threadIdx.x; e < experts; e += blockDim.x) mine[e] = 0u;
  __syncthreads();
  griddep_launch_dependents();
  griddep_wait();
  for (uint32_t a0 = blockIdx.x * blockDim.x; a0 < rows; a0 += gridDim.x * blockDim.x) {
    const uint32_t a = a0 + threadIdx.x;
    const int32_t e = a < rows ? ids[a] : -1;
    const bool there = e >= 0 && static_cast<uint32_t>(e) < experts;
    const uint32_t rank = there ? atomicAdd(&mine[e], 1u) : 0u;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < experts; i += blockDim.x) {
      if (mine[i] != 0u) mine[i] = offsets[i] + atomicAdd(&cursor[i], mine[i]);
    }
    __syncthreads();
    if (there) sorted[mine[e] + rank] = a;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < experts; i += blockDim.x) mine[i] = 0u;
    __syncthreads();
  }
}

// Count, scan and scatter in one CTA for calls of a few rows (the decode widths): the three launches
// above cost more than their work there. Counts and cursors live in shared memory.
__global__ void __launch_bounds__(1024) moe_group_small_kernel(const int32_t *ids, uint32_t rows, uint32_t experts, uint32_t item_rows,
                                                               uint32_t *offsets, uint32_t *n_items, Item *items,
                                                               uint32_t *sorted, uint32_t *status) {
  griddep_launch_dependents();
  griddep_wait();
  __shared__ uint32_t counts[kMaxExperts], start[kMaxExperts];
  __shared__ uint32_t row_sum[1024], item_sum[1024];
  for (uint32_t e = threadIdx.x; e < experts; e += 1024) counts[e] = 0u;
  __syncthreads();
  for (uint32_t a = threadIdx.x; a < rows; a += 1024) {
    const int32_t e = ids[a];
    if (e < 0 || static_cast<uint32_t>(e) >= experts) {
      if (e != IGNIS_MOE_NO_EXPERT) atomicOr(status, kStatusBadExpert);  // -1 is "no expert for this choice": skipped, not an error
    } else {
      atomicAdd(&counts[e], 1u);
    }
  }
  __syncthreads();
  const uint32_t per = (experts + 1023u) / 1024u;
  const uint32_t e0 = threadIdx.x * per;
  uint32_t nrows = 0, its = 0;
  for (uint32_t e = e0; e < e0 + per && e < experts; ++e) {
    nrows += counts[e];
    its += (counts[e] + item_rows - 1u) / item_rows;
  }
  row_sum[threadIdx.x] = nrows;
  item_sum[threadIdx.x] = its;
  __syncthreads();
  for (uint32_t d = 1; d < 1024; d <<= 1) {
    const uint32_t r = threadIdx.x >= d ? row_sum[threadIdx.x - d] : 0u;
    const uint32_t i = threadIdx.x >= d ? item_sum[threadIdx.x - d] : 0u;
    __syncthreads();
    row_sum[threadIdx.x] += r;
    item_sum[threadIdx.x] += i;
    __syncthreads();
  }
  uint32_t row_at = row_sum[threadIdx.x] - nrows, item_at = item_sum[threadIdx.x] - its;
  for (uint32_t e = e0; e < e0 + per && e < experts; ++e) {
    offsets[e] = row_at;
    start[e] = row_at;
    const uint32_t c = counts[e];
    for (uint32_t j = 0; j < c; j += item_rows) {
      items[item_at++] = Item{e, row_at + j, c - j < item_rows ? c - j : item_rows, 0u};
    }
    row_at += c;
  }
  if (threadIdx.x == 1023) {
    offsets[experts] = row_sum[1023];
    n_items[0] = item_sum[1023];
  }
  __syncthreads();
  for (uint32_t a = threadIdx.x; a < rows; a += 1024) {
    const int32_t e = ids[a];
    if (e < 0 || static_cast<uint32_t>(e) >= experts) continue;
    sorted[atomicAdd(&start[e], 1u)] = a;  // rows of one expert are independent: their order changes no output bit
  }
}

// ---- combine ----------------------------------------------------------------------------------
// One CTA per token: out = BF16(acc * 2^-32 + sigmoid(x . w_gate) * shared), acc zeroed behind it. Bound by
// memory at many tokens (22 bytes per value, most of it the accumulator read and cleared) and by
// latency at few: a thread takes eight neighbouring columns per trip in 16-byte pieces and asks for its
// first trip's accumulators and shared values before the gate's sum is known. VEC: every pointer is
// 16-byte aligned (the accumulator promises 8, the rest less).
struct CombineLoad {
  long long a[8];
  float s[8];
};
template <bool VEC>
__device__ __forceinline__ void combine_load(CombineLoad &v, const long long *acc, const float *shared) {
  if (VEC) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 q = ldg128_coherent(acc + 2 * i);
      v.a[2 * i] = static_cast<long long>((static_cast<unsigned long long>(q.y) << 32) | q.x);
      v.a[2 * i + 1] = static_cast<long long>((static_cast<unsigned long long>(q.w) << 32) | q.z);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint4 q = ldg128_coherent(shared + 4 * i);
      v.s[4 * i] = __uint_as_float(q.x), v.s[4 * i + 1] = __uint_as_float(q.y), v.s[4 * i + 2] = __uint_as_float(q.z), v.s[4 * i + 3] = __uint_as_float(q.w);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v.a[i] = acc[i], v.s[i] = shared[i];
  }
}

template <bool VEC>
__global__ void __launch_bounds__(256) moe_combine_kernel(long long *acc, const float *shared, const uint16_t *x,
                                                          const uint16_t *w_gate, uint32_t hidden, uint16_t *out) {
  griddep_launch_dependents();
  griddep_wait();
  __shared__ float partial[8];
  const size_t row = static_cast<size_t>(blockIdx.x) * hidden;
  CombineLoad v;
  const uint32_t k_first = threadIdx.x * 8u;
  if (k_first < hidden) combine_load<VEC>(v, acc + row + k_first, shared + row + k_first);
  float dot = 0.0f;
  for (uint32_t k = k_first; k < hidden; k += 2048u) {   // hidden is a multiple of 128
    alignas(16) uint16_t xv[8], wv[8];
    if (VEC) {
      *reinterpret_cast<uint4 *>(xv) = ldg128_coherent(x + row + k);
      *reinterpret_cast<uint4 *>(wv) = __ldg(reinterpret_cast<const uint4 *>(w_gate + k));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) xv[i] = x[row + k + i], wv[i] = w_gate[k + i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) dot = fmaf(bf16_bits_to_f32(xv[i]), bf16_bits_to_f32(wv[i]), dot);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xFFFFFFFFu, dot, o);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = dot;
  __syncthreads();
  float total = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) total += partial[i];
  const float gate = 1.0f / (1.0f + __expf(-total));
  for (uint32_t k = k_first; k < hidden; k += 2048u) {
    if (k != k_first) combine_load<VEC>(v, acc + row + k, shared + row + k);
    alignas(16) uint16_t o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float routed = static_cast<float>(static_cast<double>(v.a[i]) * (1.0 / 4294967296.0));
      o[i] = __bfloat16_as_ushort(__float2bfloat16_rn(routed + gate * v.s[i]));
    }
    if (VEC) {
      *reinterpret_cast<uint4 *>(out + row + k) = *reinterpret_cast<const uint4 *>(o);
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4 *>(acc + row + k + 2 * i) = make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) out[row + k + i] = o[i], acc[row + k + i] = 0;
    }
  }
}

bool aligned(const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

const DeviceState *prepared(ErrorSlot &slot, const char *what) {
  const DeviceState *dev = device_state(slot);
  if (dev == nullptr) return nullptr;
  if (!dev->prepared) {
    fail(slot, "%s: the device was not prepared (call ignis_moe_prepare at load)", what);
    return nullptr;
  }
  return dev;
}

int32_t run_experts(const Geometry &g, const void *x, uint32_t tokens, const int32_t *ids, const float *weights, const ignis_moe_slot *slots,
                    const ignis_moe_workspace *workspace, int64_t *acc, void *stream_v, uint32_t limit, const char *what) {
  ErrorSlot &slot = moe_error();
  if (x == nullptr || ids == nullptr || weights == nullptr || slots == nullptr || workspace == nullptr || acc == nullptr ||
      workspace->base == nullptr) {
    return fail(slot, "%s: NULL argument", what);
  }
  if (tokens == 0 || tokens > limit) return fail(slot, "%s: %u tokens are outside 1..%u", what, tokens, limit);
  if (!aligned(x, 16) || !aligned(workspace->base, 256)) return fail(slot, "%s: x must be 16-byte and the workspace 256-byte aligned", what);
  const DeviceState *dev = prepared(slot, what);
  if (dev == nullptr) return -1;
  const uint32_t tokens_max = workspace->decode_tokens > workspace->prefill_tokens ? workspace->decode_tokens : workspace->prefill_tokens;
  const Layout l = layout_for(g, tokens_max);
  uint8_t *base = static_cast<uint8_t *>(workspace->base);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  const uint32_t rows = tokens * g.top_k;
  uint32_t *counts = reinterpret_cast<uint32_t *>(base + l.counts);
  uint32_t *cursor = reinterpret_cast<uint32_t *>(base + l.cursor);
  uint32_t *offsets = reinterpret_cast<uint32_t *>(base + l.offsets);
  uint32_t *n_items = reinterpret_cast<uint32_t *>(base + l.n_items);
  uint32_t *sorted = reinterpret_cast<uint32_t *>(base + l.sorted);
  Item *items = reinterpret_cast<Item *>(base + l.items);
  uint32_t *status = reinterpret_cast<uint32_t *>(base + l.status);
  const bool pdl = dev->pdl != 0;
  cudaError_t err = cudaSuccess;
  if (rows <= kSmallRows) {
    err = launch(moe_group_small_kernel, dim3(1), dim3(1024), 0, stream, pdl, ids, rows, g.experts, kMoeTcItemRows, offsets, n_items, items,
                 sorted, status);
    if (err != cudaSuccess) return fail(slot, "%s: grouping launch failed: %s", what, cudaGetErrorString(err));
  } else {
  err = cudaMemsetAsync(counts, 0, l.offsets - l.counts, stream);  // counts and cursor
  if (err != cudaSuccess) return fail(slot, "%s: %s", what, cudaGetErrorString(err));
  const uint32_t grid_rows = (rows + 255u) / 256u < 1184u ? (rows + 255u) / 256u : 1184u;
  err = launch(moe_count_kernel, dim3(grid_rows), dim3(256), 0, stream, false, ids, rows, g.experts, counts, status);
  if (err == cudaSuccess) err = launch(moe_scan_kernel, dim3(1), dim3(1024), 0, stream, pdl, static_cast<const uint32_t *>(counts), g.experts, kMoeTcItemRows, offsets, n_items, items);
  if (err == cudaSuccess) err = launch(moe_scatter_kernel, dim3(grid_rows), dim3(256), 0, stream, pdl, ids, rows, g.experts, static_cast<const uint32_t *>(offsets), cursor, sorted);
  if (err != cudaSuccess) return fail(slot, "%s: grouping launch failed: %s", what, cudaGetErrorString(err));
  }

  ExpertParams p = {};
  p.ids = ids;
  p.slots = slots;
  p.items = items;
  p.n_items = n_items;
  p.sorted = sorted;
  p.x = static_cast<const uint16_t *>(x);
  p.weights = weights;
  p.x_rows = reinterpret_cast<uint16_t *>(base + l.x_rows);
  p.x_scale = reinterpret_cast<float *>(base + l.x_scale);
  p.gu = reinterpret_cast<float *>(base + l.gu);
  p.h_rows = reinterpret_cast<uint16_t *>(base + l.h_rows);
  p.h_scale = reinterpret_cast<float *>(base + l.h_scale);
  p.down_rows = reinterpret_cast<float *>(base + l.down_rows);
  p.acc = reinterpret_cast<long long *>(acc);
  p.status = status;
  p.hidden = g.hidden;
  p.inter = g.inter;
  p.top_k = g.top_k;
  p.experts = g.experts;
  // The grid is sized for the worst case the host can know (the grouping happened on the device);
  // CTAs beyond the item count return at once.
  return moe_tc_experts(slot, *dev, p, rows, items_bound(g, rows, kMoeTcItemRows), offsets, stream, what);
}

}  // namespace

int32_t prepare_moe_kernels(ErrorSlot &slot) {
  if (moe_rows_prepare(slot) != 0) return -1;
  if (moe_tc_prepare(slot) != 0) return -1;
  return moe_fp8_tc_prepare(slot);
}
}  // namespace b200q

using namespace b200q;

extern "C" {

int32_t b200q_moe_set_geometry(uint32_t hidden, uint32_t inter, uint32_t experts, uint32_t top_k) {
  const Geometry g = {hidden, inter, experts, top_k};
  if (check_geometry(moe_error(), &g, "b200q_moe_set_geometry") != 0) return -1;
  g_default = g;
  return 0;
}

int32_t b200q_moe_record_bytes(const b200q_moe_geometry *geometry, uint32_t projection, uint32_t k2, uint64_t *bytes) {
  ErrorSlot &slot = moe_error();
  if (check_geometry(slot, geometry, "ignis_moe_record_bytes") != 0) return -1;
  const Geometry &g_geo = *geometry;
  if (bytes == nullptr) return fail(slot, "ignis_moe_record_bytes: bytes is NULL");
  if (projection > IGNIS_MOE_PROJ_DOWN) return fail(slot, "ignis_moe_record_bytes: unknown projection %u", projection);
  if (!(k2 == 4 || k2 == 5 || k2 == 6 || k2 == 8)) return fail(slot, "ignis_moe_record_bytes: k2 = %u is not one of 4, 5, 6, 8", k2);
  const uint64_t in = projection == IGNIS_MOE_PROJ_GATE_UP ? g_geo.hidden : g_geo.inter;
  const uint64_t out = projection == IGNIS_MOE_PROJ_GATE_UP ? 2ull * g_geo.inter : g_geo.hidden;
  const uint64_t data = in * out * k2 / 16u + 2u * in + 2u * out;
  *bytes = (data + 4095u) & ~static_cast<uint64_t>(4095u);
  return 0;
}

int32_t ignis_moe_trellis_reconstruct(const void *trellis, uint32_t k2, uint32_t in, uint32_t out, void *w_f16, void *stream) {
  return trellis_reconstruct_raw(moe_error(), "ignis_moe_trellis_reconstruct", trellis, k2, in, out, 0, w_f16, stream);
}

int32_t ignis_moe_prepare(void) { return prepare_all(moe_error()); }

uint64_t b200q_moe_workspace_bytes(const b200q_moe_geometry *geometry, uint32_t decode_tokens, uint32_t prefill_tokens) {
  if (check_geometry(moe_error(), geometry, "ignis_moe_workspace_bytes") != 0) return 0;
  const Geometry &g_geo = *geometry;
  const uint32_t tokens_max = decode_tokens > prefill_tokens ? decode_tokens : prefill_tokens;
  if (tokens_max == 0 || decode_tokens > IGNIS_MOE_DECODE_MAX_TOKENS) return 0;
  return layout_for(g_geo, tokens_max).total;
}

int32_t b200q_moe_workspace_init(const b200q_moe_geometry *geometry, const struct ignis_moe_workspace *workspace, int64_t *acc, void *stream) {
  ErrorSlot &slot = moe_error();
  if (check_geometry(slot, geometry, "ignis_moe_workspace_init") != 0) return -1;
  const Geometry &g_geo = *geometry;
  if (workspace == nullptr || workspace->base == nullptr || acc == nullptr) return fail(slot, "ignis_moe_workspace_init: NULL argument");
  if (!aligned(workspace->base, 256)) return fail(slot, "ignis_moe_workspace_init: base is not 256-byte aligned");
  if (ignis_moe_prepare() != 0) return -1;
  const uint32_t tokens_max = workspace->decode_tokens > workspace->prefill_tokens ? workspace->decode_tokens : workspace->prefill_tokens;
  if (tokens_max == 0) return fail(slot, "ignis_moe_workspace_init: the workspace describes no tokens");
  const Layout l = layout_for(g_geo, tokens_max);
  cudaError_t err = cudaMemsetAsync(workspace->base, 0, l.sorted, static_cast<cudaStream_t>(stream));  // status, counters
  if (err == cudaSuccess) err = cudaMemsetAsync(acc, 0, sizeof(int64_t) * tokens_max * g_geo.hidden, static_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(slot, "ignis_moe_workspace_init: %s", cudaGetErrorString(err));
  return 0;
}

int32_t b200q_moe_plan_bytes(const b200q_moe_geometry *geometry, uint32_t decode_tokens, uint32_t prefill_tokens, struct ignis_moe_plan *plan) {
  ErrorSlot &slot = moe_error();
  if (plan == nullptr) return fail(slot, "ignis_moe_plan_bytes: plan is NULL");
  if (check_geometry(slot, geometry, "ignis_moe_plan_bytes") != 0) return -1;
  const Geometry &g_geo = *geometry;
  const uint64_t ws = b200q_moe_workspace_bytes(geometry, decode_tokens, prefill_tokens);
  if (ws == 0) return fail(slot, "ignis_moe_plan_bytes: no tokens, or more than %d decode tokens", IGNIS_MOE_DECODE_MAX_TOKENS);
  const uint64_t mx = decode_tokens > prefill_tokens ? decode_tokens : prefill_tokens;
  plan->workspace = ws;
  plan->acc = mx * g_geo.hidden * 8u;
  plan->router = mx * g_geo.top_k * 4u + mx * g_geo.top_k * 4u + mx * g_geo.experts * 4u;
  plan->shared = mx * g_geo.inter * 2u + mx * g_geo.hidden * 4u;
  plan->total = align256(plan->workspace) + align256(plan->acc) + align256(plan->router) + align256(plan->shared);
  return 0;
}

int32_t b200q_moe_router_logits(const b200q_moe_geometry *geometry, const void *x, uint32_t tokens, const void *w_router, float *logits,
                                void *stream) {
  ErrorSlot &slot = moe_error();
  if (check_geometry(slot, geometry, "ignis_moe_router_logits") != 0) return -1;
  const Geometry &g_geo = *geometry;
  if (x == nullptr || w_router == nullptr || logits == nullptr) return fail(slot, "ignis_moe_router_logits: NULL argument");
  if (tokens == 0) return fail(slot, "ignis_moe_router_logits: tokens must be positive");
  if (!aligned(x, 16) || !aligned(w_router, 16)) return fail(slot, "ignis_moe_router_logits: x and w_router must be 16-byte aligned");
  const DeviceState *dev = prepared(slot, "ignis_moe_router_logits");
  if (dev == nullptr) return -1;
  const cudaError_t err = moe_router_logits_launch(*dev, static_cast<const uint16_t *>(x), static_cast<const uint16_t *>(w_router), tokens,
                                                   g_geo.hidden, g_geo.experts, logits, static_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(slot, "ignis_moe_router_logits: launch failed: %s", cudaGetErrorString(err));
  return 0;
}

int32_t b200q_moe_router(const b200q_moe_geometry *geometry, const void *x, uint32_t tokens, const void *w_router, int32_t *ids,
                         float *weights, float *logits, void *stream) {
  ErrorSlot &slot = moe_error();
  if (ids == nullptr || weights == nullptr) return fail(slot, "ignis_moe_router: NULL argument");
  if (b200q_moe_router_logits(geometry, x, tokens, w_router, logits, stream) != 0) return -1;
  const Geometry &g_geo = *geometry;
  const DeviceState *dev = prepared(slot, "ignis_moe_router");
  if (dev == nullptr) return -1;
  const cudaError_t err = moe_router_select_launch(*dev, logits, tokens, g_geo.experts, g_geo.top_k, ids, weights, static_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(slot, "ignis_moe_router: launch failed: %s", cudaGetErrorString(err));
  return 0;
}

int32_t b200q_moe_experts_decode(const b200q_moe_geometry *geometry, const void *x, uint32_t tokens, const int32_t *ids,
                                 const float *weights, const struct ignis_moe_slot *slots,
                                 const struct ignis_moe_workspace *workspace, int64_t *acc, void *stream) {
  if (check_geometry(moe_error(), geometry, "ignis_moe_experts_decode") != 0) return -1;
  const uint32_t limit = workspace != nullptr ? workspace->decode_tokens : 0u;
  return run_experts(*geometry, x, tokens, ids, weights, slots, workspace, acc, stream, limit, "ignis_moe_experts_decode");
}

int32_t b200q_moe_experts_prefill(const b200q_moe_geometry *geometry, const void *x, uint32_t tokens, const int32_t *ids,
                                  const float *weights, const struct ignis_moe_slot *slots,
                                  const struct ignis_moe_workspace *workspace, int64_t *acc, void *stream) {
  if (check_geometry(moe_error(), geometry, "ignis_moe_experts_prefill") != 0) return -1;
  const uint32_t limit = workspace != nullptr ? workspace->prefill_tokens : 0u;
  return run_experts(*geometry, x, tokens, ids, weights, slots, workspace, acc, stream, limit, "ignis_moe_experts_prefill");
}

int32_t ignis_moe_decode_cluster_size(void) { return 0; }

int32_t b200q_moe_shared_expert(const b200q_moe_geometry *geometry, const void *gate, const void *up, const void *down, const void *x,
                                uint32_t tokens, void *h, float *shared, void *stream) {
  ErrorSlot &slot = moe_error();
  if (check_geometry(slot, geometry, "ignis_moe_shared_expert") != 0) return -1;
  const Geometry &g_geo = *geometry;
  if (gate == nullptr || up == nullptr || down == nullptr || x == nullptr || h == nullptr || shared == nullptr) {
    return fail(slot, "ignis_moe_shared_expert: NULL argument");
  }
  if (tokens == 0) return fail(slot, "ignis_moe_shared_expert: tokens must be positive");
  if (!aligned(gate, 16) || !aligned(up, 16) || !aligned(down, 16) || !aligned(x, 16) || !aligned(h, 8)) {
    return fail(slot, "ignis_moe_shared_expert: weights and x must be 16-byte aligned, h 8-byte aligned");
  }
  const DeviceState *dev = prepared(slot, "ignis_moe_shared_expert");
  if (dev == nullptr) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t err;
  if (moe_fp8_tc_takes(*dev, g_geo.hidden, g_geo.inter, tokens, x, h)) {  // wide calls: tcgen05
    err = moe_fp8_tc_shared_expert(*dev, static_cast<const uint8_t *>(gate), static_cast<const uint8_t *>(up),
                                   static_cast<const uint8_t *>(down), static_cast<const uint16_t *>(x), tokens, g_geo.hidden, g_geo.inter, h,
                                   shared, s);
  } else {
    err = moe_rows_shared_expert(*dev, static_cast<const uint8_t *>(gate), static_cast<const uint8_t *>(up), static_cast<const uint8_t *>(down),
                                 static_cast<const uint16_t *>(x), tokens, g_geo.hidden, g_geo.inter, h, shared, s);
  }
  if (err != cudaSuccess) return fail(slot, "ignis_moe_shared_expert: launch failed: %s", cudaGetErrorString(err));
  return 0;
}

int32_t b200q_moe_combine(const b200q_moe_geometry *geometry, int64_t *acc, const float *shared, const void *x, const void *w_gate,
                          uint32_t tokens, void *out, void *stream) {
  ErrorSlot &slot = moe_error();
  if (check_geometry(slot, geometry, "ignis_moe_combine") != 0) return -1;
  const Geometry &g_geo = *geometry;
  if (acc == nullptr || shared == nullptr || x == nullptr || w_gate == nullptr || out == nullptr) {
    return fail(slot, "ignis_moe_combine: NULL argument");
  }
  if (tokens == 0) return fail(slot, "ignis_moe_combine: tokens must be positive");
  const DeviceState *dev = prepared(slot, "ignis_moe_combine");
  if (dev == nullptr) return -1;
  const bool vec = aligned(acc, 16) && aligned(shared, 16) && aligned(x, 16) && aligned(w_gate, 16) && aligned(out, 16);
  const cudaError_t err = launch(vec ? moe_combine_kernel<true> : moe_combine_kernel<false>, dim3(tokens), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                 dev->pdl != 0, reinterpret_cast<long long *>(acc), shared, static_cast<const uint16_t *>(x),
                                 static_cast<const uint16_t *>(w_gate), g_geo.hidden, static_cast<uint16_t *>(out));
  if (err != cudaSuccess) return fail(slot, "ignis_moe_combine: launch failed: %s", cudaGetErrorString(err));
  return 0;
}

// ---- the reference's own entry points: the same calls at the default geometry -----------------------
int32_t ignis_moe_record_bytes(uint32_t projection, uint32_t k2, uint64_t *bytes) {
  return b200q_moe_record_bytes(&g_default, projection, k2, bytes);
}
uint64_t ignis_moe_workspace_bytes(uint32_t decode_tokens, uint32_t prefill_tokens) {
  return b200q_moe_workspace_bytes(&g_default, decode_tokens, prefill_tokens);
}
int32_t ignis_moe_workspace_init(const struct ignis_moe_workspace *workspace, int64_t *acc, void *stream) {
  return b200q_moe_workspace_init(&g_default, workspace, acc, stream);
}
int32_t ignis_moe_plan_bytes(uint32_t decode_tokens, uint32_t prefill_tokens, struct ignis_moe_plan *plan) {
  return b200q_moe_plan_bytes(&g_default, decode_tokens, prefill_tokens, plan);
}
int32_t ignis_moe_router_logits(const void *x, uint32_t tokens, const void *w_router, float *logits, void *stream) {
  return b200q_moe_router_logits(&g_default, x, tokens, w_router, logits, stream);
}
int32_t ignis_moe_router(const void *x, uint32_t tokens, const void *w_router, int32_t *ids, float *weights, float *logits,
                         void *stream) {
  return b200q_moe_router(&g_default, x, tokens, w_router, ids, weights, logits, stream);
}
int32_t ignis_moe_experts_decode(const void *x, uint32_t tokens, const int32_t *ids, const float *weights,
                                 const struct ignis_moe_slot *slots, const struct ignis_moe_workspace *workspace,
                                 int64_t *acc, void *stream) {
  return b200q_moe_experts_decode(&g_default, x, tokens, ids, weights, slots, workspace, acc, stream);
}
int32_t ignis_moe_experts_prefill(const void *x, uint32_t tokens, const int32_t *ids, const float *weights,
                                  const struct ignis_moe_slot *slots, const struct ignis_moe_workspace *workspace,
                                  int64_t *acc, void *stream) {
  return b200q_moe_experts_prefill(&g_default, x, tokens, ids, weights, slots, workspace, acc, stream);
}
int32_t ignis_moe_shared_expert(const void *gate, const void *up, const void *down, const void *x, uint32_t tokens, void *h,
                                float *shared, void *stream) {
  return b200q_moe_shared_expert(&g_default, gate, up, down, x, tokens, h, shared, stream);
}
int32_t ignis_moe_combine(int64_t *acc, const float *shared, const void *x, const void *w_gate, uint32_t tokens, void *out,
                          void *stream) {
  return b200q_moe_combine(&g_default, acc, shared, x, w_gate, tokens, out, stream);
}

int32_t ignis_moe_stream_sync(void *stream) {
  const cudaError_t err = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(moe_error(), "ignis_moe_stream_sync: %s", cudaGetErrorString(err));
  return 0;
}

int32_t ignis_moe_workspace_status(const struct ignis_moe_workspace *workspace, void *stream, uint32_t *status) {
  ErrorSlot &slot = moe_error();
  if (workspace == nullptr || workspace->base == nullptr || status == nullptr) return fail(slot, "ignis_moe_workspace_status: NULL argument");
  uint32_t words[2] = {0u, 0u};   // [0] the expert kernels' bits, [1] bounded waits of the tensor-core kernels that ran out
  uint32_t shared_expert = 0u;    // the same for the shared expert's tensor-core kernels (no workspace of their own)
  cudaError_t err = cudaMemcpyAsync(words, workspace->base, sizeof(words), cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream));
  if (err == cudaSuccess) err = moe_fp8_tc_status(&shared_expert, static_cast<cudaStream_t>(stream));
  if (err == cudaSuccess) err = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(slot, "ignis_moe_workspace_status: %s", cudaGetErrorString(err));
  *status = words[0] | ((words[1] | shared_expert) != 0u ? kStatusTcWait : 0u);
  return 0;
}

const char *ignis_moe_last_error(void) { return moe_error().text; }

}  // extern "C"
