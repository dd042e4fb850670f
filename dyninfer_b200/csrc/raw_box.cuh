// Boxes of raw quantised weights in shared memory (rows x 256 weights, brought by tensor copies) and their conversion to the f16
// pairs of a tcgen05 A operand in tensor memory: thread = weight row, 64 weights at a time.
#pragma once

#include "codec.cuh"
#include "umma.cuh"

namespace dyn {

constexpr int GS_UNIT = 256;  // K elements of a box of raw weights

// 32-bit words of a row in a box
__host__ __device__ constexpr int gs_words(int enc) {
  return enc == E_Q4_0 || enc == E_Q4_K ? 36 : enc == E_Q4_1 ? 40 : enc == E_Q8_0 ? 68 : enc == E_Q5_K ? 44 : 32;
}

__device__ __forceinline__ uint32_t gs_h2u(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 gs_u2h(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

// The 64 weights of quarter `g` of a row's box, in two halves of 32: 16 f16 pairs each.
template <int ENC>
struct GsRow {
  // quarter g of Q4_0 / Q8_0 starts g words past a 16-byte boundary, of Q4_1 0 or 2 words
  static constexpr int NV = ENC == E_Q4_0 || ENC == E_Q4_1 ? 12 : ENC == E_Q8_0 ? 20 : ENC == E_Q4_K ? 12 : ENC == E_Q5_K ? 20 : 8;
  uint32_t v[NV];
  uint32_t sc[2], bi[2];  // MLX: scale and bias of the two halves
  int g;

  __device__ __forceinline__ void ld4(int i, const uint8_t* p) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    v[i] = q.x, v[i + 1] = q.y, v[i + 2] = q.z, v[i + 3] = q.w;
  }
  __device__ __forceinline__ void load(const uint8_t* box, int row, int quarter) {
    g = quarter;
    const uint8_t* p = box + row * (gs_words(ENC) * 4);
    if constexpr (ENC == E_Q4_0 || ENC == E_Q4_1 || ENC == E_Q8_0) {
      const int first = ENC == E_Q4_0 ? 8 * g : ENC == E_Q4_1 ? (10 * g) & ~3 : 16 * g;
#pragma unroll
      for (int i = 0; i < NV; i += 4) ld4(i, p + 4 * (first + i));
    } else if constexpr (ENC == E_MLX_U4) {
#pragma unroll
      for (int i = 0; i < 2; i++) ld4(4 * i, p + (((2 * g + i) ^ (row & 7)) << 4));
    } else {
      ld4(0, p);
      if constexpr (ENC == E_Q5_K) ld4(4, p + 16), ld4(8, p + 32);
#pragma unroll
      for (int i = 0; i < 2; i++) ld4(NV - 8 + 4 * i, p + gs_words(ENC) * 4 - 128 + 32 * g + 16 * i);
    }
  }
  // brings the quarter's first word to v[0]; g is the same for the whole warp
  __device__ __forceinline__ void align() {
    if constexpr (ENC == E_Q4_0 || ENC == E_Q8_0) {
      if (g & 1) {
#pragma unroll
        for (int i = 0; i + 1 < NV; i++) v[i] = v[i + 1];
      }
    }
    if constexpr (ENC == E_Q4_0 || ENC == E_Q8_0 || ENC == E_Q4_1) {
      if (ENC == E_Q4_1 ? (g & 1) : (g & 2)) {
#pragma unroll
        for (int i = 0; i + 2 < NV; i++) v[i] = v[i + 2];
      }
    }
  }
  __device__ __forceinline__ void half(int b, uint32_t (&out)[16]) const {
    if constexpr (ENC == E_Q4_0 || ENC == E_Q4_1) {
      const __half2 c1032 = __floats2half2_rn(1032.f, 1032.f), c72 = __floats2half2_rn(-72.f, -72.f);
      const __half2 c16th = __floats2half2_rn(0.0625f, 0.0625f), c1024 = __floats2half2_rn(1024.f, 1024.f);
      const __half2 c64n = __floats2half2_rn(-64.f, -64.f);
      const uint32_t* w = v + (ENC == E_Q4_1 ? 5 * b : 4 * b);
      const uint32_t dm = ENC == E_Q4_1 ? w[0] : (b ? w[0] >> 16 : w[0] & 0xffffu);
      const __half dh = __ushort_as_half((unsigned short)(dm & 0xffffu)), mh = __ushort_as_half((unsigned short)(dm >> 16));
      const __half2 d2 = __halves2half2(dh, dh), m2 = __halves2half2(mh, mh);
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const uint32_t x = ENC == E_Q4_1 || b ? w[1 + t] : __funnelshift_r(w[t], w[t + 1], 16);
        const uint32_t x8 = x >> 8;
        uint32_t l02 = (x & 0x000F000Fu) | 0x64006400u, l13 = (x8 & 0x000F000Fu) | 0x64006400u;
        uint32_t h02 = (x & 0x00F000F0u) | 0x64006400u, h13 = (x8 & 0x00F000F0u) | 0x64006400u;
        if constexpr (ENC == E_Q4_0) {  // (q - 8) * d, the difference exact
          l02 = gs_h2u(__hmul2(__hsub2(gs_u2h(l02), c1032), d2));
          l13 = gs_h2u(__hmul2(__hsub2(gs_u2h(l13), c1032), d2));
          h02 = gs_h2u(__hmul2(__hfma2(gs_u2h(h02), c16th, c72), d2));
          h13 = gs_h2u(__hmul2(__hfma2(gs_u2h(h13), c16th, c72), d2));
        } else {  // q * d + m
          l02 = gs_h2u(__hfma2(__hsub2(gs_u2h(l02), c1024), d2, m2));
          l13 = gs_h2u(__hfma2(__hsub2(gs_u2h(l13), c1024), d2, m2));
          h02 = gs_h2u(__hfma2(__hfma2(gs_u2h(h02), c16th, c64n), d2, m2));
          h13 = gs_h2u(__hfma2(__hfma2(gs_u2h(h13), c16th, c64n), d2, m2));
        }
        // weights 4t..4t+3 (low nibbles) and 16+4t..16+4t+3 (high nibbles) of the block
        out[2 * t] = __byte_perm(l02, l13, 0x5410);
        out[2 * t + 1] = __byte_perm(l02, l13, 0x7632);
        out[8 + 2 * t] = __byte_perm(h02, h13, 0x5410);
        out[8 + 2 * t + 1] = __byte_perm(h02, h13, 0x7632);
      }
    } else if constexpr (ENC == E_Q8_0) {
      const __half2 c1152 = __floats2half2_rn(1152.f, 1152.f);
      const uint32_t* w = v + 8 * b;
      const __half dh = __ushort_as_half((unsigned short)(b ? w[0] >> 16 : w[0] & 0xffffu));
      const __half2 d2 = __halves2half2(dh, dh);
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const uint32_t x = (b ? w[1 + t] : __funnelshift_r(w[t], w[t + 1], 16)) ^ 0x80808080u;
        out[2 * t] = gs_h2u(__hmul2(__hsub2(gs_u2h(__byte_perm(x, 0x64646464u, 0x4140)), c1152), d2));
        out[2 * t + 1] = gs_h2u(__hmul2(__hsub2(gs_u2h(__byte_perm(x, 0x64646464u, 0x4342)), c1152), d2));
      }
    } else if constexpr (ENC == E_MLX_U4) {
      const __half2 c1024 = __floats2half2_rn(1024.f, 1024.f);
      const __half2 s2 = __float2half2_rn(__uint_as_float(sc[b])), b2 = __float2half2_rn(__uint_as_float(bi[b]));
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t x = v[4 * b + j];
        const uint32_t lo = x & 0x0F0F0F0Fu, hi = (x >> 4) & 0x0F0F0F0Fu;  // nibbles 0,2,4,6 / 1,3,5,7
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const uint32_t pr = (__byte_perm(lo, hi, 0x0400 + 0x0101 * e) & 0x00FF00FFu) | 0x64006400u;  // (n 2e, n 2e+1)
          out[4 * j + e] = gs_h2u(__hfma2(__hsub2(gs_u2h(pr), c1024), s2, b2));
        }
      }
    } else {
      // Q4_K, Q5_K: sub-block j = 2 g + b, 6-bit scale and minimum out of the 12 packed bytes (words 1..3); each product
      // and the difference rounded in f32 on its own, as the decoders do
      const int j = 2 * g + b;
      auto sb = [&](int i) { return ((i < 4 ? v[1] : i < 8 ? v[2] : v[3]) >> (8 * (i & 3))) & 0xffu; };
      uint32_t s6, m6;
      if (j < 4) {
        s6 = sb(j) & 63u, m6 = sb(j + 4) & 63u;
      } else {
        s6 = (sb(j + 4) & 15u) | ((sb(j - 4) >> 6) << 4);
        m6 = (sb(j + 4) >> 4) | ((sb(j) >> 6) << 4);
      }
      const float ds = __fmul_rn(f16_bits_to_f32(v[0] & 0xffffu), (float)s6), dm = __fmul_rn(f16_bits_to_f32(v[0] >> 16), (float)m6);
#pragma unroll
      for (int wq = 0; wq < 8; wq++) {
        uint32_t x = (v[NV - 8 + wq] >> (4 * b)) & 0x0F0F0F0Fu;
        if constexpr (ENC == E_Q5_K) x |= ((v[4 + wq] >> j) & 0x01010101u) << 4;
        float f[4];
        f[0] = __fsub_rn(__fmul_rn(ds, __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7440)) - 8388608.f), dm);
        f[1] = __fsub_rn(__fmul_rn(ds, __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7441)) - 8388608.f), dm);
        f[2] = __fsub_rn(__fmul_rn(ds, __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7442)) - 8388608.f), dm);
        f[3] = __fsub_rn(__fmul_rn(ds, __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7443)) - 8388608.f), dm);
        out[2 * wq] = gs_h2u(__floats2half2_rn(f[0], f[1])), out[2 * wq + 1] = gs_h2u(__floats2half2_rn(f[2], f[3]));
      }
    }
  }
};

}  // namespace dyn
