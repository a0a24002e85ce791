// A row tile's product with a superblock on mma.sync, the quantized integers themselves as the A operand: shared by the
// kernels of two to sixteen activation rows (kq_rows.cu, kq_few.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "kq_common.cuh"
#include "kq_imma_q4k.cuh"
#include "kq_tcgen05.cuh"

namespace kq {

namespace {

// sub-blocks of a superblock, min term, 16-byte blocks
__host__ __device__ constexpr int rw_nsub(int c) { return c == Q6_K ? 16 : 8; }
__host__ __device__ constexpr bool rw_min(int c) { return c == Q4_K || c == Q5_K; }
__host__ __device__ constexpr bool rw_al16(int c) { return c == Q4_K || c == Q5_K; }
// what the operand of integer 0 stands for, to be subtracted: the bf16 pattern's 128, and the codec's own offset
template <int C, bool BF>
__host__ __device__ constexpr int rw_base() { return C == IQ4_XS ? 0 : (BF ? 128 : 0) + (C == Q6_K ? 32 : 0); }
template <int C, bool BF>
__host__ __device__ constexpr bool rw_sums() { return rw_min(C) || rw_base<C, BF>() != 0; }
// words per (superblock, activation row) of the sums: heads, tails, padding against bank conflicts
__host__ __device__ constexpr int rw_sum_pitch(int c) { return 2 * rw_nsub(c) + 4; }

__device__ __forceinline__ void rw_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1, __half) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void rw_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1, __nv_bfloat16) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same with accumulators of zero (constants: no registers to clear)
__device__ __forceinline__ void rw_mma0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1, __half) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void rw_mma0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1, __nv_bfloat16) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void rw_mma_tf32(float (&c)[4], const float (&a)[4], float b0, float b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
        "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
__device__ __forceinline__ void rw_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void rw_cp16_upto(uint32_t dst, const void* src, int bytes) {  // the rest is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// byte j of v as a float (the integer sits in the low mantissa bits of 2^23); j may be a lane value
__device__ __forceinline__ float rw_byte(uint32_t v, int j, float minus = 8388608.f) {
  return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u + j)) - minus;
}
__device__ __forceinline__ uint32_t rw_lds(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

// One unit of work: sixteen weight rows (this lane: r0 = row g, r1 = row g + 8) x one superblock, all activation rows.
// xb: this lane's activation row (nt = 0) at the superblock; sums: the stage's sums at the superblock.
template <int C, typename XT, int NT>
struct RowsUnit {
  static constexpr bool kBf = std::is_same<XT, __nv_bfloat16>::value;
  static constexpr uint32_t kMagic = kBf ? 0x43434343u : 0u;
  static constexpr float kUp = C == IQ4_XS || kBf ? 1.f : 16777216.f;  // fp16 operands are scaled by 2^-24
  static constexpr float kSumUp = kBf ? 1.f / 8192.f : 1.f;  // the sums of bf16 rows by 2^13: tails of small ones stay normal
  static constexpr int kBase = rw_base<C, kBf>();
  static constexpr int kP = rw_sum_pitch(C);

  // y += d * (up * acc - base * sum_j sc_j xs_j) - dmin * sum_j mn_j xs_j
  static __device__ __forceinline__ void finish(float (&y)[NT][4], const float (&acc)[NT][4], float d0, float d1) {
#pragma unroll
    for (int n = 0; n < NT; n++) {
      y[n][0] = fmaf(d0 * kUp, acc[n][0], y[n][0]);
      y[n][1] = fmaf(d0 * kUp, acc[n][1], y[n][1]);
      y[n][2] = fmaf(d1 * kUp, acc[n][2], y[n][2]);
      y[n][3] = fmaf(d1 * kUp, acc[n][3], y[n][3]);
    }
  }
  // y += f * sum_j a_j xs_j over the NS sub-blocks; a: coefficients of this lane's (row, sub-block) operand places
  template <int NS>
  static __device__ __forceinline__ void sum_term(float (&y)[NT][4], const float (&a)[NS / 8][4], const float* sums,
                                                  int g, int t, float f0, float f1) {
#pragma unroll
    for (int n = 0; n < NT; n++) {
      const float* s = sums + (n * 8 + g) * kP + t;
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < NS / 8; i++) {
        rw_mma_tf32(c, a[i], s[8 * i], s[8 * i + 4]);
        rw_mma_tf32(c, a[i], s[NS + 8 * i], s[NS + 8 * i + 4]);
      }
      y[n][0] = fmaf(f0, c[0], y[n][0]);
      y[n][1] = fmaf(f0, c[1], y[n][1]);
      y[n][2] = fmaf(f1, c[2], y[n][2]);
      y[n][3] = fmaf(f1, c[3], y[n][3]);
    }
  }
  // four weights of either row (one byte each) against b[n] = four activations of column n
  template <bool FIRST>
  static __device__ __forceinline__ void four(float (&c)[NT][4], uint32_t qa, uint32_t qb, const uint32_t (&b)[NT][2]) {
    const uint32_t a0 = __byte_perm(qa, kMagic, 0x4140), a2 = __byte_perm(qa, kMagic, 0x4342);
    const uint32_t a1 = __byte_perm(qb, kMagic, 0x4140), a3 = __byte_perm(qb, kMagic, 0x4342);
#pragma unroll
    for (int n = 0; n < NT; n++) {
      if constexpr (FIRST) rw_mma0(c[n], a0, a1, a2, a3, b[n][0], b[n][1], XT());
      else rw_mma(c[n], a0, a1, a2, a3, b[n][0], b[n][1], XT());
    }
  }
  static __device__ __forceinline__ void scale_add(float (&acc)[NT][4], const float (&c)[NT][4], float s0, float s1) {
#pragma unroll
    for (int n = 0; n < NT; n++) {
      acc[n][0] = fmaf(s0, c[n][0], acc[n][0]);
      acc[n][1] = fmaf(s0, c[n][1], acc[n][1]);
      acc[n][2] = fmaf(s1, c[n][2], acc[n][2]);
      acc[n][3] = fmaf(s1, c[n][3], acc[n][3]);
    }
  }

  // q4_k / q5_k: 32 quant bytes hold sub-blocks 2 p (low nibbles) and 2 p + 1 (high); a lane takes bytes 8 t .. 8 t + 7
  static __device__ __forceinline__ void run_k4(float (&y)[NT][4], const uint8_t* r0, const uint8_t* r1,
                                                const uint8_t* (&xb)[NT], const float* sums, int g, int t) {
    const uint4 h0 = *reinterpret_cast<const uint4*>(r0), h1 = *reinterpret_cast<const uint4*>(r1);
    const StScales s0 = st_unpack(h0), s1 = st_unpack(h1);
    constexpr int kQs = C == Q5_K ? 48 : 16;
    uint2 u0 = make_uint2(0u, 0u), u1 = u0;  // q5_k: bit j of byte l is the fifth bit of weight l of sub-block j
    if constexpr (C == Q5_K) {
      u0 = *reinterpret_cast<const uint2*>(r0 + 16 + 8 * t);
      u1 = *reinterpret_cast<const uint2*>(r1 + 16 + 8 * t);
    }
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const uint2 wa = *reinterpret_cast<const uint2*>(r0 + kQs + 32 * p + 8 * t);
      const uint2 wb = *reinterpret_cast<const uint2*>(r1 + kQs + 32 * p + 8 * t);
#pragma unroll
      for (int hi = 0; hi < 2; hi++) {
        const int j = 2 * p + hi;
        uint32_t b0[NT][2], b1[NT][2];
#pragma unroll
        for (int n = 0; n < NT; n++) {
          const uint4 b = *reinterpret_cast<const uint4*>(xb[n] + 64 * j + 16 * t);
          b0[n][0] = b.x, b0[n][1] = b.y, b1[n][0] = b.z, b1[n][1] = b.w;
        }
        auto nib = [&](uint32_t w, uint32_t u) {
          uint32_t q = (hi ? w >> 4 : w) & 0x0f0f0f0fu;
          if constexpr (C == Q5_K) q |= (j <= 4 ? u << (4 - j) : u >> (j - 4)) & 0x10101010u;
          return q;
        };
        float c[NT][4];
        four<true>(c, nib(wa.x, u0.x), nib(wb.x, u1.x), b0);
        four<false>(c, nib(wa.y, u0.y), nib(wb.y, u1.y), b1);
        scale_add(acc, c, rw_byte(p < 2 ? s0.scl : s0.sch, j & 3), rw_byte(p < 2 ? s1.scl : s1.sch, j & 3));
      }
    }
    const float2 dd0 = __half22float2(*reinterpret_cast<const __half2*>(&h0.x));  // (d, dmin)
    const float2 dd1 = __half22float2(*reinterpret_cast<const __half2*>(&h1.x));
    finish(y, acc, dd0.x, dd1.x);
    const float m[1][4] = {{rw_byte(s0.mnl, t), rw_byte(s1.mnl, t), rw_byte(s0.mnh, t), rw_byte(s1.mnh, t)}};
    sum_term<8>(y, m, sums, g, t, -kSumUp * dd0.y, -kSumUp * dd1.y);
    if constexpr (kBase != 0) {
      const float s[1][4] = {{rw_byte(s0.scl, t), rw_byte(s1.scl, t), rw_byte(s0.sch, t), rw_byte(s1.sch, t)}};
      sum_term<8>(y, s, sums, g, t, -kSumUp * kBase * dd0.x, -kSumUp * kBase * dd1.x);
    }
  }

  // q6_k (src/kquant_cpu_decode.cpp:238-280): sub-block j = 8 h + 2 quarter + s of sixteen weights is one instruction.
  // PH: the block starts two bytes past a multiple of four. The aligned words around a group of sixteen bytes then
  // are bytes 2 + 4 t .. 5 + 4 t for t < 3, and for t = 3 bytes 14, 15 and the first two of the next group: lane 3
  // takes bytes 0, 1 (from the word before) and 14, 15.
  template <int PH>
  static __device__ __forceinline__ void run_q6(float (&y)[NT][4], const uint8_t* r0, const uint8_t* r1,
                                                const uint8_t* (&xb)[NT], const float* sums, int g, int t) {
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    const uint32_t sel = t == 3 ? 0x5432u : 0x7654u;
    const int xo0 = PH ? (t == 3 ? 0 : 4 + 8 * t) : 8 * t, xo1 = PH ? (t == 3 ? 28 : 8 + 8 * t) : 0;
    uint32_t sc0[4], sc1[4];  // the sixteen signed scales of either row, biased by 128
    {
      if constexpr (PH == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) sc0[i] = rw_lds(r0 + 192 + 4 * i) ^ 0x80808080u, sc1[i] = rw_lds(r1 + 192 + 4 * i) ^ 0x80808080u;
      } else {
        uint32_t a[5], b[5];
#pragma unroll
        for (int i = 0; i < 5; i++) a[i] = rw_lds(r0 + 190 + 4 * i), b[i] = rw_lds(r1 + 190 + 4 * i);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          sc0[i] = __byte_perm(a[i], a[i + 1], 0x5432) ^ 0x80808080u;
          sc1[i] = __byte_perm(b[i], b[i + 1], 0x5432) ^ 0x80808080u;
        }
      }
    }
    auto group = [&](const uint8_t* p, uint32_t& prev) {  // this lane's four bytes of the sixteen at p
      if constexpr (PH == 0) {
        return rw_lds(p + 4 * t);
      } else {
        const uint32_t w = rw_lds(p + 2 + 4 * t);
        const uint32_t r = __byte_perm(prev, w, sel);
        prev = w;
        return r;
      }
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint32_t L[2][4], H[2][2];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint8_t* p = r ? r1 : r0;
        uint32_t pl = 0u, ph = 0u;
        if constexpr (PH) {
          const int po = t == 3 ? -2 : 2;  // only lane 3 uses it
          pl = rw_lds(p + 64 * h + po);
          ph = rw_lds(p + 128 + 32 * h + po);
        }
#pragma unroll
        for (int s = 0; s < 4; s++) L[r][s] = group(p + 64 * h + 16 * s, pl);
#pragma unroll
        for (int s = 0; s < 2; s++) H[r][s] = group(p + 128 + 32 * h + 16 * s, ph);
      }
#pragma unroll
      for (int s = 0; s < 2; s++) {
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
          const int j = 8 * h + 2 * qd + s;
          uint32_t q[2];
#pragma unroll
          for (int r = 0; r < 2; r++) {
            const uint32_t l = L[r][2 * (qd & 1) + s], u = H[r][s];
            const uint32_t hb = qd == 0 ? u << 4 : (qd == 1 ? u << 2 : (qd == 2 ? u : u >> 2));
            q[r] = ((qd & 2 ? l >> 4 : l) & 0x0f0f0f0fu) | (hb & 0x30303030u);
          }
          uint32_t b[NT][2];
#pragma unroll
          for (int n = 0; n < NT; n++) {
            if constexpr (PH == 0) {
              const uint2 v = *reinterpret_cast<const uint2*>(xb[n] + 32 * j + xo0);
              b[n][0] = v.x, b[n][1] = v.y;
            } else {
              b[n][0] = rw_lds(xb[n] + 32 * j + xo0);
              b[n][1] = rw_lds(xb[n] + 32 * j + xo1);
            }
          }
          float c[NT][4];
          four<true>(c, q[0], q[1], b);
          scale_add(acc, c, rw_byte(sc0[j >> 2], j & 3, 8388736.f), rw_byte(sc1[j >> 2], j & 3, 8388736.f));
        }
      }
    }
    const float d0 = __half2float(*reinterpret_cast<const __half*>(r0 + 208));
    const float d1 = __half2float(*reinterpret_cast<const __half*>(r1 + 208));
    finish(y, acc, d0, d1);
    float s[2][4];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      s[i][0] = rw_byte(sc0[2 * i], t, 8388736.f), s[i][1] = rw_byte(sc1[2 * i], t, 8388736.f);
      s[i][2] = rw_byte(sc0[2 * i + 1], t, 8388736.f), s[i][3] = rw_byte(sc1[2 * i + 1], t, 8388736.f);
    }
    sum_term<16>(y, s, sums, g, t, -kSumUp * kBase * d0, -kSumUp * kBase * d1);
  }

  // iq4_xs (src/kquant_cpu_decode.cpp:557-584): a nibble is one of sixteen levels, small integers that both 16-bit
  // types hold exactly: their two bytes come out of two sixteen-byte tables, four weights a permute. A halfword of
  // quant bytes holds the selectors of its four nibbles as they lie (bit 3 chooses the half of the table afterwards).
  struct Pairs {
    uint32_t low, high;  // the low nibbles of two bytes, the high nibbles, as 16-bit floats
  };
  static __device__ __forceinline__ Pairs iq4_pairs(uint32_t half) {
    // bytes of the sixteen levels (-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113), level 0 in the
    // lowest byte: L the low, H the high ones of their fp16 numbers (first row) and of their bf16 numbers
    constexpr uint32_t L[2][4] = {{0x103080f0u, 0x00806020u, 0xc0408000u, 0x109050a0u},
                                  {0x82a6d0feu, 0x20b00c44u, 0x18c85080u, 0xe2b28a54u}};
    constexpr uint32_t H[2][4] = {{0xd4d5d6d7u, 0xc9cdd0d2u, 0x504e4a3cu, 0x57555452u},
                                  {0xc2c2c2c2u, 0xc1c1c2c2u, 0x4241413fu, 0x42424242u}};
    const uint32_t sel = half & 0x7777u, pick = 0x3210u | ((half >> 1) & 0x4444u);
    const uint32_t lo = __byte_perm(__byte_perm(L[kBf][0], L[kBf][1], sel), __byte_perm(L[kBf][2], L[kBf][3], sel), pick);
    const uint32_t hi = __byte_perm(__byte_perm(H[kBf][0], H[kBf][1], sel), __byte_perm(H[kBf][2], H[kBf][3], sel), pick);
    return {__byte_perm(lo, hi, 0x6240), __byte_perm(lo, hi, 0x7351)};
  }
  static __device__ __forceinline__ void run_iq4(float (&y)[NT][4], const uint8_t* r0, const uint8_t* r1,
                                                 const uint8_t* (&xb)[NT], int t) {
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    const uint2 h0 = *reinterpret_cast<const uint2*>(r0), h1 = *reinterpret_cast<const uint2*>(r1);
    // 6-bit scales of the even and the odd sub-blocks, a byte each: four bits of scales_l, two of scales_h
    auto scales = [](const uint2 h, int odd) {
      const uint32_t u = (h.x >> 16) >> (2 * odd);
      const uint32_t top = (u & 3u) | ((u & 0x30u) << 4) | ((u & 0x300u) << 8) | ((u & 0x3000u) << 12);
      return ((h.y >> (4 * odd)) & 0x0f0f0f0fu) | (top << 4);
    };
    const uint32_t s0[2] = {scales(h0, 0), scales(h0, 1)}, s1[2] = {scales(h1, 0), scales(h1, 1)};
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t wa = rw_lds(r0 + 8 + 16 * j + 4 * t), wb = rw_lds(r1 + 8 + 16 * j + 4 * t);
      const Pairs a0 = iq4_pairs(wa), a1 = iq4_pairs(wa >> 16), b0 = iq4_pairs(wb), b1 = iq4_pairs(wb >> 16);
      float c[NT][4];
#pragma unroll
      for (int n = 0; n < NT; n++) {
        const uint2 v0 = *reinterpret_cast<const uint2*>(xb[n] + 64 * j + 8 * t);
        const uint2 v1 = *reinterpret_cast<const uint2*>(xb[n] + 64 * j + 32 + 8 * t);
        rw_mma0(c[n], a0.low, b0.low, a1.low, b1.low, v0.x, v0.y, XT());
        rw_mma(c[n], a0.high, b0.high, a1.high, b1.high, v1.x, v1.y, XT());
      }
      scale_add(acc, c, rw_byte(s0[j & 1], j >> 1, 8388640.f), rw_byte(s1[j & 1], j >> 1, 8388640.f));
    }
    finish(y, acc, __half2float(__ushort_as_half((unsigned short)h0.x)), __half2float(__ushort_as_half((unsigned short)h1.x)));
  }

  static __device__ __forceinline__ void run(float (&y)[NT][4], const uint8_t* r0, const uint8_t* r1,
                                             const uint8_t* (&xb)[NT], const float* sums, int g, int t) {
    if constexpr (C == Q6_K) {
      if ((smem_u32(r0) & 2) == 0) run_q6<0>(y, r0, r1, xb, sums, g, t);
      else run_q6<1>(y, r0, r1, xb, sums, g, t);
    } else if constexpr (C == IQ4_XS) {
      run_iq4(y, r0, r1, xb, t);
    } else {
      run_k4(y, r0, r1, xb, sums, g, t);
    }
  }
};

// The sums of one superblock's sub-blocks for eight activation rows (columns), by ones x activations; lanes 0..3 hold
// columns 2 t, 2 t + 1 and store them as a tf32 head and the rest.
template <int C, typename XT>
__device__ __forceinline__ void rows_sums(const uint8_t* xrow, float* out, int lane) {
  constexpr int NS = rw_nsub(C), P = rw_sum_pitch(C);
  constexpr uint32_t one = std::is_same<XT, __half>::value ? 0x3C003C00u : 0x46004600u;
  const int t = lane & 3;
  uint2 b[16];  // all loads before the first store: the compiler cannot tell that they do not overlap
#pragma unroll
  for (int i = 0; i < 16; i++) {
    if constexpr (NS == 8) {
      if (i & 1) continue;
      const uint4 v = *reinterpret_cast<const uint4*>(xrow + 32 * i + 16 * t);
      b[i] = make_uint2(v.x, v.y), b[i + 1] = make_uint2(v.z, v.w);
    } else {
      b[i] = *reinterpret_cast<const uint2*>(xrow + 32 * i + 8 * t);
    }
  }
  float c[NS][4];
#pragma unroll
  for (int j = 0; j < NS; j++) {
    rw_mma0(c[j], one, one, one, one, b[j * (16 / NS)].x, b[j * (16 / NS)].y, XT());
#pragma unroll
    for (int i = 1; i < 16 / NS; i++) rw_mma(c[j], one, one, one, one, b[j * (16 / NS) + i].x, b[j * (16 / NS) + i].y, XT());
  }
  if (lane < 4) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      float* o = out + (2 * t + i) * P;
#pragma unroll
      for (int j = 0; j < NS; j += 4) {
        float4 h, l;
        float* hp = &h.x;
        float* lp = &l.x;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          hp[q] = __uint_as_float(__float_as_uint(c[j + q][i]) & 0xffffe000u);
          lp[q] = c[j + q][i] - hp[q];
        }
        *reinterpret_cast<float4*>(o + j) = h;
        *reinterpret_cast<float4*>(o + NS + j) = l;
      }
    }
  }
}

// plain_dot (kq_common.cuh) with what is known of the alignment of these codecs' rows here
template <int C, typename XT>
__device__ __noinline__ float rows_plain(const uint8_t* w, const XT* x, int nsb) {
  return plain_dot<C, rw_al16(C) ? 16 : (C == IQ4_XS ? 8 : 2)>(w, x, 256 * nsb);
}

}  // namespace

}  // namespace kq
