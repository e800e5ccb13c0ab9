// Dense trellis linear beyond 64 tokens: the prefill route on the tensor cores.
//
// Stands where the reference switches from its decode kernel to its prefill kernel
// (kernel/src/trellis_linear.cu: rotate_kernel + prefill_kernel, trellis_linear_prefill.cu:162-279;
// the route needs the workspace, as theirs does). Two launches: `trellis_rotate_rows_kernel` writes
// the rotated activations as fp16 rows with one scale per token into the workspace, and
// `trellis_tc_dense_kernel` multiplies them with the trellis plane on tcgen05 (trellis_tc.cuh).
// SwiGLU runs the gate product first (BF16 into h, as the reference's prefill route stores the gate
// between its passes: ignis_trellis_linear.h:43-44) and the up product with an epilogue that
// multiplies by silu of what it finds there.
#include "../../include/ignis_trellis_linear.h"

#include "trellis_internal.cuh"
#include "trellis_tc.cuh"

#include <cmath>

namespace b200q {
namespace {

using namespace trellis_tc;

__device__ uint32_t g_trellis_tc_status = 0;

// ---- rotation: one CTA per token (rotate_row, trellis_device.cuh) --------------------------------------------------
// THREADS: the most a launch has (fewer leave a thread more registers for loads in flight).
template <int THREADS>
__global__ void __launch_bounds__(THREADS) trellis_rotate_rows_kernel(const uint16_t *x, const uint16_t *suh, uint32_t in, uint16_t *rows_f16, float *inv) {
  __shared__ float warp_max[32];
  griddep_launch_dependents();
  const size_t token = blockIdx.x;
  griddep_wait();
  rotate_row(in, rows_f16 + token * in, inv + token, warp_max, [&](uint32_t k, float2 (&v)[4]) {
    const uint2 lo = __ldg(reinterpret_cast<const uint2 *>(suh + k)), hi = __ldg(reinterpret_cast<const uint2 *>(suh + k + 4));   // 8-byte aligned
    scaled_inputs(ldg128_coherent(x + token * in + k), make_uint4(lo.x, lo.y, hi.x, hi.y), v);
  });
}

// ---- the product -----------------------------------------------------------------------------------
constexpr uint32_t kEpiStore = 0, kEpiAdd = 1, kEpiSiluMul = 2;   // kEpiSiluMul: y = BF16(silu(float(y)) * v)

struct DenseParams {
  const uint32_t *trellis;
  const uint16_t *svh;
  const float *inv;      // the tokens' inverse scales
  uint16_t *y;           // BF16 [tokens][ldy]
  uint32_t k2, tile_stride, in, out, tokens, ldy, epilogue;
  uint32_t tile;         // tokens per CTA
  uint32_t ranks;        // the CTAs of a cluster share an item's K stages (1: no cluster)
};

template <int GROUPS>
__global__ void __launch_bounds__(Shape<GROUPS>::kThreads, GROUPS == 2 ? 2 : 1) trellis_tc_dense_kernel(const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ DenseParams p) {
  extern __shared__ uint8_t smem_raw[];
  // Token tiles run fastest over the grid, so the CTAs at work at one time decode the same columns
  // of the plane (read from HBM once, then from the L2).
  const uint32_t row_tiles = (p.tokens + p.tile - 1u) / p.tile;
  const Split split = {p.ranks, p.ranks == 1u ? 0u : cluster_ctarank()};
  const uint32_t item = blockIdx.x / p.ranks;
  Job job;
  job.trellis = p.trellis;
  job.k2 = p.k2;
  job.tile_stride = p.tile_stride;
  const uint32_t stages = p.in / 64u;
  job.stage0 = stages * split.rank / p.ranks;
  job.stage1 = stages * (split.rank + 1u) / p.ranks;
  job.blk = item / row_tiles;
  job.row0 = item % row_tiles * p.tile;
  job.rows = min(p.tokens - job.row0, p.tile);
  job.box = p.tile > 256u ? p.tile / 2u : p.tile;
  const Core c = core_setup<GROUPS>(smem_raw, job, split);
  const bool decoded = core_roles<GROUPS>(c, job, &map_rows, &g_trellis_tc_status);
  const uint16_t *svh = p.svh + job.blk * 128u;
  uint16_t *out = p.y + static_cast<size_t>(job.row0) * p.ldy + job.blk * 128u;
  core_finish_rows<GROUPS>(
      c, job, split, decoded, &g_trellis_tc_status, [&](uint32_t r) { return p.inv[job.row0 + r]; },
      [&](uint32_t r) { return out + static_cast<size_t>(r) * p.ldy; },
      [&](const uint16_t *y, uint32_t col) { return p.epilogue != kEpiStore ? *reinterpret_cast<const uint2 *>(y + col) : make_uint2(0u, 0u); },
      [&](uint16_t *y, uint32_t col, const uint2 &old, const float4 &o) {
        const float4 sv = four_halves(__ldg(reinterpret_cast<const uint2 *>(svh + col)));
        float v[4] = {o.x * sv.x, o.y * sv.y, o.z * sv.z, o.w * sv.w};
        if (p.epilogue != kEpiStore) {
          const float was[4] = {bf16_bits_to_f32(old.x & 0xFFFFu), __uint_as_float(old.x & 0xFFFF0000u), bf16_bits_to_f32(old.y & 0xFFFFu),
                                __uint_as_float(old.y & 0xFFFF0000u)};
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = p.epilogue == kEpiAdd ? v[e] + was[e] : was[e] / (1.0f + __expf(-was[e])) * v[e];
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
        *reinterpret_cast<uint2 *>(y + col) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
      });
}

uint64_t align256(uint64_t v) { return (v + 255u) & ~static_cast<uint64_t>(255u); }

constexpr uint32_t kRotateMaxIn = 51200;   // inputs of a row the route takes

bool aligned_to(const void *p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

}  // namespace

uint64_t trellis_tc_workspace_bytes(uint32_t in, uint32_t weights, uint32_t tokens) {
  // a status line, then per weight the rotated rows (fp16) and the tokens' inverse scales
  return 256u + static_cast<uint64_t>(weights) * (align256(static_cast<uint64_t>(tokens) * in * 2u) + align256(static_cast<uint64_t>(tokens) * 4u));
}

namespace {
cudaLaunchConfig_t dense_config(bool wide, uint32_t items, uint32_t ranks, cudaStream_t stream, bool pdl, cudaLaunchAttribute (&attr)[2]) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(items * ranks);
  config.blockDim = dim3(wide ? Shape<4>::kThreads : Shape<2>::kThreads);
  config.dynamicSmemBytes = wide ? Shape<4>::kSmemBytes : Shape<2>::kSmemBytes;
  config.stream = stream;
  unsigned n = 0;
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (ranks > 1u) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = ranks;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  config.attrs = attr;
  config.numAttrs = n;
  return config;
}

// The CTA's shape, the tokens per CTA and the CTAs per item: those for which a model of the launch gives the least time. In
// microseconds, fitted to every choice for five shapes (5120 -> 1024, 6144 and 17408, 6144 and 17408 -> 5120) at 70 to 4096 tokens
// and 3 and 5 bits; what it picks is within 1 % of the fastest measured on average, 20 % at worst (a 1024-column weight at 300
// tokens). The two-group shape takes 0.62 a stage with two CTAs on the SM and 0.41 alone while the decoder warps bound it, 4 ns
// a token where the rows do; the four-group shape, one CTA an SM, 0.46 and 1.4 ns a token, but nothing runs under its fill and
// epilogue. Then the epilogue and a cluster's exchange. Few items leave SMs idle and walk all of K alone (17408 -> 5120 at 200
// tokens: 80 items, 174 us; 40 of the other shape, three ranks each: 57). At least four stages per rank.
struct DensePlan {
  uint32_t tile, ranks;
  bool wide;   // four decoder groups
};
DensePlan dense_plan(const DeviceState &dev, uint32_t blocks, uint32_t stages, uint32_t tokens) {
  DensePlan best = {0u, 1u, false};
  float least = 0.0f;
  for (const bool wide : {false, true}) {
    if (dev.trellis_dw == (wide ? 8 : 16)) continue;   // B200Q_TRELLIS_TC_SHAPE asks for the other
    const uint32_t most = wide ? Shape<4>::kMaxRows : Shape<2>::kMaxRows, fewest = (tokens + most - 1u) / most;
    for (uint32_t nt = fewest; nt <= fewest + 2u; ++nt) {
      const uint32_t tile = ((tokens + nt - 1u) / nt + 15u) / 16u * 16u;
      if (nt > fewest && tile < 48u) break;
      const uint32_t items = blocks * ((tokens + tile - 1u) / tile);
      const float rows = static_cast<float>(tile);
      for (uint32_t ranks = 1; ranks <= kMaxRanks && (ranks == 1u || stages / ranks >= 4u); ++ranks) {
        // clusters (CTAs) the device places with one CTA per SM: what the occupancy query counts
        const uint32_t one_each = ranks == 1u ? static_cast<uint32_t>(dev.sm_count) : static_cast<uint32_t>(dev.trellis_clusters[ranks]);
        if (one_each == 0u) continue;
        const float walked = static_cast<float>((stages + ranks - 1u) / ranks), r = static_cast<float>(ranks);
        float t;
        if (wide) {
          const float cta = walked * fmaxf(0.46f, 0.0014f * rows) + 0.45f + 0.022f * rows / r + (ranks > 1u ? 1.0f + 0.022f * rows : 0.0f);
          t = static_cast<float>((items + one_each - 1u) / one_each) * cta;
        } else {
          const float pair = fmaxf(0.62f, 0.004f * rows), alone = fmaxf(0.41f, 0.0005f * rows);
          const float rest = 0.34f + 0.012f * rows / r + (ranks > 1u ? 1.6f + 0.023f * rows : 0.0f);
          const uint32_t left = items % (2u * one_each);
          t = static_cast<float>(items / (2u * one_each)) * (walked * pair + rest) + (left == 0u ? 0.0f : walked * (left > one_each ? pair : alone) + rest);
        }
        if (best.tile == 0u || t < least) least = t, best = {tile, ranks, wide};
      }
    }
  }
  return best;
}
}  // namespace

int32_t trellis_tc_prepare(ErrorSlot &slot) {
  DeviceState *dev = device_state(slot);
  if (dev == nullptr) return -1;
  cudaError_t err = cudaFuncSetAttribute(trellis_tc_dense_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<2>::kSmemBytes));
  if (err == cudaSuccess) err = cudaFuncSetAttribute(trellis_tc_dense_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<4>::kSmemBytes));
  if (err != cudaSuccess) return fail(slot, "trellis prefill kernel attributes: %s", cudaGetErrorString(err));
  for (uint32_t ranks = 2; ranks <= kMaxRanks && !dev->counted; ++ranks) {
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t config = dense_config(false, 1u, ranks, nullptr, false, attr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, trellis_tc_dense_kernel<2>, &config) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    dev->trellis_clusters[ranks] = clusters;
  }
  if (encode_tiled_fn() == nullptr) return fail(slot, "cuTensorMapEncodeTiled is not available from this driver");
  return 0;
}

bool trellis_tc_takes(const DeviceState &dev, uint32_t in, uint32_t tokens, uint32_t weights, const ignis_trellis_workspace *workspace) {
  if (dev.trellis_tc == 0 || tokens <= IGNIS_TRELLIS_DECODE_MAX_TOKENS) return false;
  if (in > kRotateMaxIn) return false;
  if (workspace == nullptr || workspace->base == nullptr || !aligned_to(workspace->base, 256)) return false;
  return workspace->bytes >= trellis_tc_workspace_bytes(in, weights, tokens);
}

namespace {
int32_t one_product(ErrorSlot &slot, const DeviceState &dev, const ignis_trellis_weight *w, const uint16_t *x, uint32_t tokens, uint16_t *y,
                    uint32_t ldy, uint32_t epilogue, uint8_t *region, cudaStream_t stream, const char *what) {
  uint16_t *rows = reinterpret_cast<uint16_t *>(region);
  float *inv = reinterpret_cast<float *>(region + align256(static_cast<uint64_t>(tokens) * w->in * 2u));
  const uint32_t threads = 32u * rotate_warps(w->in);
  cudaError_t err = launch(threads <= 256u ? trellis_rotate_rows_kernel<256> : threads <= 640u ? trellis_rotate_rows_kernel<640> : trellis_rotate_rows_kernel<1024>,
                           dim3(tokens), dim3(threads), 0, stream, dev.pdl != 0, x, static_cast<const uint16_t *>(w->suh), w->in, rows, inv);
  if (err != cudaSuccess) return fail(slot, "%s: rotation launch failed: %s", what, cudaGetErrorString(err));
  const DensePlan plan = dense_plan(dev, w->out / 128u, w->in / 64u, tokens);
  CUtensorMap map_rows;
  if (!make_rows_map(&map_rows, rows, tokens, w->in, plan.tile > 256u ? plan.tile / 2u : plan.tile)) return fail(slot, "%s: tensor map encoding failed", what);
  DenseParams p = {};
  p.trellis = static_cast<const uint32_t *>(w->trellis);
  p.svh = static_cast<const uint16_t *>(w->svh);
  p.inv = inv;
  p.y = y;
  p.k2 = w->k2;
  p.tile_stride = w->tile_stride ? w->tile_stride : w->out / 16u;
  p.in = w->in;
  p.out = w->out;
  p.tokens = tokens;
  p.ldy = ldy;
  p.epilogue = epilogue;
  p.tile = plan.tile;
  p.ranks = plan.ranks;
  const uint32_t items = w->out / 128u * ((tokens + p.tile - 1u) / p.tile);
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t config = dense_config(plan.wide, items, p.ranks, stream, dev.pdl != 0, attr);
  err = cudaLaunchKernelEx(&config, plan.wide ? trellis_tc_dense_kernel<4> : trellis_tc_dense_kernel<2>, map_rows, p);
  if (err != cudaSuccess) return fail(slot, "%s: launch failed: %s", what, cudaGetErrorString(err));
  return 0;
}
}  // namespace

int32_t trellis_tc_linear(ErrorSlot &slot, const DeviceState &dev, const ignis_trellis_weight *w, const ignis_trellis_weight *up,
                          const void *x, uint32_t tokens, void *y, uint32_t ldy, uint32_t epilogue,
                          const ignis_trellis_workspace *workspace, cudaStream_t stream, const char *what) {
  uint8_t *base = static_cast<uint8_t *>(workspace->base) + 256;
  const uint16_t *xs = static_cast<const uint16_t *>(x);
  uint16_t *ys = static_cast<uint16_t *>(y);
  if (up == nullptr) return one_product(slot, dev, w, xs, tokens, ys, ldy, epilogue == 1u ? kEpiAdd : kEpiStore, base, stream, what);
  // SwiGLU: the gate product into h, then the up product times silu of what it finds there
  if (one_product(slot, dev, w, xs, tokens, ys, ldy, kEpiStore, base, stream, what) != 0) return -1;
  uint8_t *second = base + align256(static_cast<uint64_t>(tokens) * w->in * 2u) + align256(static_cast<uint64_t>(tokens) * 4u);
  return one_product(slot, dev, up, xs, tokens, ys, ldy, kEpiSiluMul, second, stream, what);
}

int32_t trellis_tc_status(ErrorSlot &slot, cudaStream_t stream, uint32_t *status) {
  cudaError_t err = cudaMemcpyFromSymbolAsync(status, g_trellis_tc_status, sizeof(uint32_t), 0, cudaMemcpyDeviceToHost, stream);
  if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
  if (err != cudaSuccess) return fail(slot, "b200q_trellis_device_status: %s", cudaGetErrorString(err));
  return 0;
}

}  // namespace b200q
