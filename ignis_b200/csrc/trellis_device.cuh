// Device-side pieces shared by the dense trellis linear and the MoE expert kernels: the tile
// decode (format: kernel/src/trellis_decode.cuh:6-24 of the reference), the warp Hadamard and the
// cluster helpers.
#ifndef B200Q_TRELLIS_DEVICE_CUH
#define B200Q_TRELLIS_DEVICE_CUH

#include "common.cuh"

namespace b200q {
namespace trellis_dev {

constexpr uint32_t kMul1 = 0x83DCD12Du;

// Exclusive end bit of step p in a tile of class k2 = 2 K.
__host__ __device__ constexpr int step_end(int k2, int p) {
  return k2 == 5 ? 3 * ((p + 1) / 2) + 2 * (p / 2 + 1) : (k2 / 2) * (p + 1);
}

struct LaneWindow {
  uint32_t w0, w1, w2;  // word indices inside the tile
  uint32_t off;         // bit offset of the lane's first window bit inside word w0
};

__device__ __forceinline__ LaneWindow lane_window(uint32_t k2, int lane) {
  const int words = 4 * static_cast<int>(k2), bits = 128 * static_cast<int>(k2);
  int first = 4 * static_cast<int>(k2) * lane + static_cast<int>(k2 >> 1) - 16;  // end of step 8 lane, minus 16
  if (first < 0) first += bits;
  LaneWindow w;
  w.w0 = static_cast<uint32_t>(first >> 5);
  w.off = static_cast<uint32_t>(first & 31);
  w.w1 = w.w0 + 1 == static_cast<uint32_t>(words) ? 0u : w.w0 + 1;
  w.w2 = w.w1 + 1 == static_cast<uint32_t>(words) ? 0u : w.w1 + 1;
  return w;
}

// The lane's eight weights from its three words: four half2 in step order (steps 0,1 | 2,3 | 4,5 |
// 6,7), i.e. tile elements (r0, c0) (r0+1, c0) | (r0+8, c0) (r0+9, c0) | the same rows at c0 + 8,
// r0 = 2 (lane % 4), c0 = lane / 4.
//
// A state is the upper half of the window shifted to it. A state eight or sixteen bits behind another is one byte permute or one
// mask of the other's shifted window instead of a shift of its own and one down: at 2, 2.5 and 4 bits per weight that saves four,
// three and four of some 44 operations (the products' time goes by their number: the output head at 4 bits, one token, 342 us ->
// 330; an MoE block of 4096 tokens at 2.5 bits 1213 -> 1150).
__host__ __device__ constexpr int state_offset(int k2, int j) { return step_end(k2, j) - step_end(k2, 0); }
// The step whose shifted window gives state j: an earlier one that shifts for itself, 8 or 16 bits before, or j.
__host__ __device__ constexpr int state_root(int k2, int j) {
  for (int i = 0; i < j; ++i) {
    const int behind = state_offset(k2, j) - state_offset(k2, i);
    if ((behind == 8 || behind == 16) && state_root(k2, i) == i) return i;
  }
  return j;
}
template <int K2, int J>
__device__ __forceinline__ void decode_state(uint32_t hi, uint32_t mid, uint32_t (&window)[8], uint32_t (&code)[8]) {
  constexpr int d = state_offset(K2, J), root = state_root(K2, J), behind = d - state_offset(K2, root);
  uint32_t state;
  if constexpr (behind == 0) {
    if constexpr (d == 0) window[J] = hi;
    else if constexpr (d < 32) window[J] = __funnelshift_l(mid, hi, d);   // also where a plain shift of `hi` would do: 2 bits, one token a layer 130 us, 141 with it
    else window[J] = mid << (d - 32);
    state = window[J] >> 16;
  } else if constexpr (behind == 8) {
    state = __byte_perm(window[root], 0u, 0x4421);
  } else {
    state = window[root] & 0xFFFFu;
  }
  code[J] = __dp4a(state * kMul1, 0x01010101u, 0x6400u);
}

template <int K2>
__device__ __forceinline__ void decode8(uint32_t a, uint32_t b, uint32_t c, uint32_t off, uint32_t (&frag)[4]) {
  const uint32_t hi = __funnelshift_l(b, a, off);
  const uint32_t mid = __funnelshift_l(c, b, off);
  uint32_t code[8], window[8];
  decode_state<K2, 0>(hi, mid, window, code);
  decode_state<K2, 1>(hi, mid, window, code);
  decode_state<K2, 2>(hi, mid, window, code);
  decode_state<K2, 3>(hi, mid, window, code);
  decode_state<K2, 4>(hi, mid, window, code);
  decode_state<K2, 5>(hi, mid, window, code);
  decode_state<K2, 6>(hi, mid, window, code);
  decode_state<K2, 7>(hi, mid, window, code);
  const __half2 k_inv = __halves2half2(__ushort_as_half(0x1EEE), __ushort_as_half(0x1EEE));
  const __half2 k_bias = __halves2half2(__ushort_as_half(0xC931), __ushort_as_half(0xC931));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t packed = __byte_perm(code[2 * i], code[2 * i + 1], 0x5410);
    const __half2 v = __hfma2(*reinterpret_cast<const __half2 *>(&packed), k_inv, k_bias);
    frag[i] = *reinterpret_cast<const uint32_t *>(&v);
  }
}

__device__ __forceinline__ void decode8_any(uint32_t k2, uint32_t a, uint32_t b, uint32_t c, uint32_t off,
                                            uint32_t (&frag)[4]) {
  switch (k2) {
    case 4: decode8<4>(a, b, c, off, frag); break;
    case 5: decode8<5>(a, b, c, off, frag); break;
    case 6: decode8<6>(a, b, c, off, frag); break;
    case 8: decode8<8>(a, b, c, off, frag); break;
    case 10: decode8<10>(a, b, c, off, frag); break;
    default: decode8<12>(a, b, c, off, frag); break;
  }
}

// v holds elements 4 lane .. 4 lane + 3 of a 128-vector; on return the vector times the natural
// order Sylvester Hadamard / sqrt(128): two stages inside the lane, five across lanes.
__device__ __forceinline__ void hadamard128(float (&v)[4], int lane) {
  const float a = v[0] + v[1], b = v[0] - v[1], c = v[2] + v[3], d = v[2] - v[3];
  v[0] = a + c;
  v[1] = b + d;
  v[2] = a - c;
  v[3] = b - d;
#pragma unroll
  for (int m = 1; m < 32; m <<= 1) {
    // the upper lane of a pair keeps (other - own), the lower (own + other): one fused multiply-add by
    // -1 or +1 gives either, rounded once like the subtraction or the addition it stands for
    const float sign = (lane & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float o = __shfl_xor_sync(0xFFFFFFFFu, v[i], m);
      v[i] = __fmaf_rn(sign, v[i], o);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] *= 0.08838834764831845f;
}

// Two floats at a time (one instruction for both).
__device__ __forceinline__ float2 add_f32x2(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long &>(r)) : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
  return r;
}
__device__ __forceinline__ float2 mul_f32x2(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long &>(r)) : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
  return r;
}
__device__ __forceinline__ float2 fma_f32x2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long &>(r)) : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)), "l"(reinterpret_cast<unsigned long long &>(c)));
  return r;
}

// The same transform, without its 1 / sqrt(128), of a 128-vector that four lanes hold: lane q (0..3) its units q, q + 4, ... of
// 2 PAIRS values each. `low` and `high` are the lane masks of q's two bits. The stages run in hadamard128's order and round
// alike; five of them lie inside a lane, two values an instruction, so that eight vectors in a warp take 192 instructions
// where one takes 56.
template <int UNITS, int PAIRS>
__device__ __forceinline__ void hadamard_quad(float2 (&v)[UNITS][PAIRS], int lane, int low, int high) {
  static_assert(UNITS * PAIRS == 16, "32 values a lane");
  const float2 minus = make_float2(-1.0f, -1.0f);
#pragma unroll
  for (int u = 0; u < UNITS; ++u) {
#pragma unroll
    for (int p = 0; p < PAIRS; ++p) v[u][p] = make_float2(v[u][p].x + v[u][p].y, v[u][p].x - v[u][p].y);
#pragma unroll
    for (int h = 1; h < PAIRS; h <<= 1) {
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) {
        if ((p & h) == 0) {
          const float2 a = v[u][p], b = v[u][p + h];
          v[u][p] = add_f32x2(a, b);
          v[u][p + h] = fma_f32x2(b, minus, a);
        }
      }
    }
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int mask = s == 0 ? low : high;
    const float sign = (lane & mask) != 0 ? -1.0f : 1.0f;   // as in hadamard128
    const float2 sign2 = make_float2(sign, sign);
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) {
        const float2 o = make_float2(__shfl_xor_sync(0xFFFFFFFFu, v[u][p].x, mask), __shfl_xor_sync(0xFFFFFFFFu, v[u][p].y, mask));
        v[u][p] = fma_f32x2(sign2, v[u][p], o);
      }
    }
  }
#pragma unroll
  for (int h = 1; h < UNITS; h <<= 1) {
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
      if ((u & h) == 0) {
#pragma unroll
        for (int p = 0; p < PAIRS; ++p) {
          const float2 a = v[u][p], b = v[u + h][p];
          v[u][p] = add_f32x2(a, b);
          v[u + h][p] = fma_f32x2(b, minus, a);
        }
      }
    }
  }
}

// ---- a row's rotation into fp16, for the tensor-core routes ------------------------------------------------------
// Warp w of the CTA takes blocks 8 w .. + 7 of the row's 128-input blocks (a row has as many warps as that makes, up to 32, and
// goes round beyond), four lanes a block, lane q its units q, q + 4, q + 8, q + 12 of eight inputs. `fetch(k, v)` gives the
// eight products x o suh at input k. One power-of-two scale for the row brings its largest magnitude into [2^13, 2^14); the
// inverse goes to *inv.
constexpr float kHadamardNorm = 0.08838834764831845f;   // 1 / sqrt(128)
__host__ __device__ constexpr uint32_t rotate_warps(uint32_t in) { return (in / 128u + 7u) / 8u < 32u ? (in / 128u + 7u) / 8u : 32u; }

template <class Fetch>
__device__ __forceinline__ void rotate_row(uint32_t in, uint16_t *dst, float *inv, float *warp_max, Fetch fetch) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t nblk = in / 128u, warps = blockDim.x / 32u, q = static_cast<uint32_t>(lane) & 3u;
  float2 v[4][4];
  auto transform = [&](uint32_t bl) {   // block bl of the row, zeros past its end
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (bl < nblk) {
        fetch(bl * 128u + (4u * u + q) * 8u, v[u]);
      } else {
#pragma unroll
        for (int p = 0; p < 4; ++p) v[u][p] = make_float2(0.0f, 0.0f);
      }
    }
    hadamard_quad<4, 4>(v, lane, 1, 2);
  };
  float m = 0.0f;
  const uint32_t first = static_cast<uint32_t>(warp) * 8u + (static_cast<uint32_t>(lane) >> 2);
  const bool once = nblk <= 8u * warps;   // the row's values stay in registers
  for (uint32_t bl0 = 0; bl0 < nblk; bl0 += 8u * warps) {
    transform(bl0 + first);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int p = 0; p < 4; ++p) m = fmaxf(m, fmaxf(fabsf(v[u][p].x), fabsf(v[u][p].y)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if (warps > 1u) {
    if (lane == 0) warp_max[warp] = m;
    __syncthreads();
    m = warp_max[lane < static_cast<int>(warps) ? lane : 0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  }
  m *= kHadamardNorm;
  // m in [2^(e-1), 2^e) with e = (exponent field) - 126: the scale 2^(14 - e), held to what a float carries
  int shift = 0;
  if (m > 0.0f && m <= 3.0e38f) shift = max(-126, min(126, 140 - static_cast<int>(__float_as_uint(m) >> 23)));
  const float scale = __uint_as_float(static_cast<uint32_t>(shift + 127) << 23);
  if (threadIdx.x == 0) *inv = __uint_as_float(static_cast<uint32_t>(127 - shift) << 23);
  for (uint32_t bl0 = 0; bl0 < nblk; bl0 += 8u * warps) {
    if (!once) transform(bl0 + first);
    if (bl0 + first >= nblk) continue;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t packed[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const __half2 h = __floats2half2_rn(v[u][p].x * kHadamardNorm * scale, v[u][p].y * kHadamardNorm * scale);
        packed[p] = *reinterpret_cast<const uint32_t *>(&h);
      }
      *reinterpret_cast<uint4 *>(dst + (bl0 + first) * 128u + (4u * u + q) * 8u) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
  }
}
// Eight inputs times their suh, both in 16-byte pieces: BF16 and FP16.
__device__ __forceinline__ void scaled_inputs(const uint4 x, const uint4 suh, float2 (&v)[4]) {
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ss[4] = {suh.x, suh.y, suh.z, suh.w};
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    v[p] = mul_f32x2(make_float2(bf16_bits_to_f32(xs[p] & 0xFFFFu), __uint_as_float(xs[p] & 0xFFFF0000u)),
                     __half22float2(*reinterpret_cast<const __half2 *>(&ss[p])));
  }
}

}  // namespace trellis_dev
}  // namespace b200q

#endif
