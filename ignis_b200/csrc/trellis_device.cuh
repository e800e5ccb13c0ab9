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
template <int K2>
__device__ __forceinline__ void decode8(uint32_t a, uint32_t b, uint32_t c, uint32_t off, uint32_t (&frag)[4]) {
  const uint32_t hi = __funnelshift_l(b, a, off);
  const uint32_t mid = __funnelshift_l(c, b, off);
  uint32_t code[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    constexpr int base = step_end(K2, 0);
    const int d = step_end(K2, j) - base;  // constant after unrolling
    const uint32_t x = d == 0 ? hi : (d < 32 ? __funnelshift_l(mid, hi, d) : mid << (d - 32));
    code[j] = __dp4a((x >> 16) * kMul1, 0x01010101u, 0x6400u);
  }
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

}  // namespace trellis_dev
}  // namespace b200q

#endif
