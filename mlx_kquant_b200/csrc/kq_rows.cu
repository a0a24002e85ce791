// Decode product of a few activation rows: y[M, N] = x[M, K] . dequant(W)^T for 1 <= M <= 16, on mma.sync with the
// quantized integers themselves as the A operand (sixteen weight rows x sixteen weights an instruction), the
// activations in their own 16-bit type as the B operand, float32 accumulation. Reference: qmv_fused_rows,
// src/kquant_cpu_decode.cpp:1032-1065.
//
// What bounds it: a tile product is a chain of shared-memory loads, permutes and matrix instructions some 2500 cycles
// long, with 16 warps on an SM to hide it (without any weight copy [28672, 8192] x 1 row takes 40 of 48 us; without any
// product 26), half of the issue slots and half of the ALU pipe (byte permutes) busy; HBM is the next bound. Measured
// [14336, 4096] x 8 bf16 rows: q4_k 17.4 us, q5_k x 16 fp16 rows 22.1; q6_k [4096, 14336] x 8 24.0 (25.3, 80, 97.5 on
// the kernels before it). What it is built around:
//   * No value is rounded: a weight is scale x integer (- min), the integer goes into the tensor core as it is and
//     the scale is applied in float32 to the sum over its 16- or 32-weight sub-block. The bytes become operands
//     with one byte permute per two weights: for bf16 rows byte q becomes the bf16 number 128 + q (0x4300 | q), for
//     fp16 rows the subnormal q * 2^-24; what the constant offset adds (and the min term of the codecs that have one)
//     is coefficient_j * (sum of the activations of sub-block j), a product of its own with tf32 instructions over the
//     float32 sums split in two parts. The sums of a stage are made once per CTA by helper warps. No operand is scaled
//     down, so that products with the smallest normal bf16 activations stay normal float32 numbers (with 128 + q scaled
//     by 2^-24, rows of 1e-36 came out with tens of times their size); sums that overflow are caught by rows_plain.
//   * One CTA per SM owns N / SM count consecutive weight rows (rows are independent, so tiles need not be whole) and
//     walks K in stages of WK superblocks: four producer warps bring the stage's bytes of every row, and the
//     activations of that K range, into shared memory with 16-byte asynchronous copies, three or more stages in
//     flight (one bulk copy per row instead was four times slower: a bulk copy costs the SM some 80 cycles); the consumer warps are RT row tiles x WK superblocks, so that a stage is one tile product per warp.
//   * Nothing is read before griddepcontrol.wait: the weights may have been written by the kernel before. Copies of the
//     first stages ahead of the wait were 0.1-0.6 us a launch faster (q4_k bf16 x 8 rows [4096, 4096] 7.1 against 7.3 us,
//     [14336, 4096] 16.8 against 17.4); fetching them into L2 ahead of it instead was slower than waiting (18.8).
// Blocks that are not whole numbers of 16 bytes (q6_k) are copied as the 16-byte aligned window around a row's
// bytes; a block then starts on an even byte, and where that is not a multiple of four the words are taken from the
// next aligned position, with the sub-block's weights handed to the lanes in another order (the sum over a
// sub-block does not care, the activations are read in the same order).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_imma_q4k.cuh"
#include "kq_launch.h"
#include "kq_tcgen05.cuh"

namespace kq {

namespace {

constexpr int kRwMaxStages = 6;
// Warps of a CTA and its shared memory. Dense: one CTA per SM. Gather (an expert's rows are few blocks, a CTA lives a
// few microseconds): two, so that one starts while the other works.
template <bool G>
struct RowsShape {
  static constexpr int kWarps = G ? 8 : 16, kProducers = G ? 2 : 4, kHelpers = G ? 2 : 4;
  static constexpr int kThreads = 32 * (kWarps + kProducers + kHelpers);
  static constexpr int kCtas = G ? 2 : 1;
  static constexpr int kMaxSmem = G ? 112 * 1024 : 226 * 1024;
};
constexpr int kRwMaxEntries = 1024;  // entries of a gather call: every CTA looks through all of them

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

// gather_qmm: entry i multiplies activation row lhs[i] by matrix rhs[i]; grid.y counts the matrices, or (by_entry,
// fewer entries than matrices) the entries, of which the first of every matrix does the work for all. Routing may be
// uneven: a CTA makes at most `deep` passes over its matrix, and CTAs of y >= units take what is left (rows_left_over).
struct RowsGather {
  const uint32_t *lhs, *rhs;
  int n_entries, n_experts, by_entry;
  long long x_batch, expert_stride;
  int units, deep;
};

struct RowsPlan {
  int R;       // weight rows of a row block
  int rt, wk;  // row tiles of 16, warps to a row tile: rt * wk consumer warps work
  int cs;      // superblocks of a stage; warp column k takes k, k + wk, ...
  int wlog, xlog;  // log2 of the producer threads on one row of the weights, of x
  int half;    // != 0: tile rows 0 .. half - 1 are the block's even rows, the others its odd ones
  int stages, wpitch, xpitch, stage_bytes, x_off, sum_off, red_off, list_off, smem;
  int n_blocks;
};

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

// One output by itself: decoded weights times activations in float32, as the generic kernel has it. For outputs that
// the split into integers, offsets and sub-block sums leaves without a finite value although they may have one, or an
// infinity: an infinite activation meets the offset's sum (inf - inf), and a sum of integers can overflow before its
// scale is applied. Rare, so one thread an output, without care for speed.
template <int C, typename XT>
__device__ __noinline__ float rows_plain(const uint8_t* w, const XT* x, int nsb) {
  constexpr int A = rw_al16(C) ? 16 : (C == IQ4_XS ? 8 : 2);
  const IqTables tabs = global_iq_tables();
  float sum = 0.f;
#pragma unroll 1
  for (int o = 0; o < 32 * nsb; o++) {
    float v[8];
    decode8<C, A>(w + (long long)(o >> 5) * bpb_of(C), o & 31, v, tabs);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      float xv;
      if constexpr (std::is_same<XT, __half>::value) xv = __half2float(x[8 * o + i]);
      else xv = __bfloat162float(x[8 * o + i]);
      sum = fmaf(xv, v[i], sum);
    }
  }
  return sum;
}

// The matrix and the first pass of left-over group j: the matrices' passes (of `rows` entries) beyond the first `base`,
// ga.deep of them a group, numbered by matrix. counts: n_experts words of shared memory; all threads of the CTA take
// part. x: the matrix, or n_experts where there is no such group.
template <int TH>
__device__ __forceinline__ int2 rows_left_over(const RowsGather& ga, int rows, int base, int j, int* counts, int2* found) {
  for (int e = threadIdx.x; e < ga.n_experts; e += TH) counts[e] = 0;
  if (threadIdx.x == 0) *found = make_int2(ga.n_experts, 0);
  __syncthreads();
  for (int i = threadIdx.x; i < ga.n_entries; i += TH) {
    const uint32_t e = ga.rhs[i];
    if (e < (uint32_t)ga.n_experts && (long long)ga.lhs[i] < ga.x_batch) atomicAdd(&counts[e], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    for (int e0 = 0; e0 < ga.n_experts; e0 += 32) {
      const int e = e0 + (int)threadIdx.x;
      const int over = e < ga.n_experts ? max(0, (counts[e] + rows - 1) / rows - base) : 0;
      const int groups = (over + ga.deep - 1) / ga.deep;
      int upto = groups;  // of this matrix and those before it among the 32
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if ((int)threadIdx.x >= o) upto += v;
      }
      if (j < upto && j >= upto - groups) *found = make_int2(e, base + (j - upto + groups) * ga.deep);
      const int all = __shfl_sync(0xffffffffu, upto, 31);
      if (j < all) break;
      j -= all;
    }
  }
  __syncthreads();
  return *found;
}

template <int C, typename XT, int NT, bool G>
__global__ void __launch_bounds__(RowsShape<G>::kThreads, RowsShape<G>::kCtas)
rows_kernel(const GemvArgs a, const RowsPlan pl, const RowsGather ga, int* __restrict__ error_word) {
  constexpr int NW = RowsShape<G>::kWarps, BPB = bpb_of(C);
  constexpr int kRwProducers = RowsShape<G>::kProducers, kRwHelpers = RowsShape<G>::kHelpers;
  constexpr bool kBf = std::is_same<XT, __nv_bfloat16>::value;
  constexpr bool kSums = rw_sums<C, kBf>();
  extern __shared__ __align__(128) uint8_t rw_dyn[];
  __shared__ uint64_t full[kRwMaxStages], ready[kRwMaxStages], empty[kRwMaxStages];
  __shared__ int abort_s, count_s;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = pl.stages;
  const int nsb = a.K >> 8, nst = (nsb + pl.cs - 1) / pl.cs;
  // Rows of an odd number of two-byte-aligned blocks start alternately on and between multiples of four: a tile takes
  // rows of one kind, as the lanes' share of a sub-block depends on it.
  auto row_of = [&](int r) { return pl.half == 0 ? r : (r < pl.half ? 2 * r : 2 * (r - pl.half) + 1); };
  const int live = pl.rt * pl.wk;  // consumer warps with work
  if (threadIdx.x == 0) {
    abort_s = count_s = 0;
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 32 * kRwProducers);
      mbar_init(&ready[s], kRwHelpers);
      mbar_init(&empty[s], live + (kSums ? kRwHelpers : 0));
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  // Passes: the dense form walks the row blocks blockIdx.x, + gridDim.x, ... for all M rows; the gather form has one
  // row block of one matrix and walks its entries, 8 NT at a time (grid.z CTAs share them; where there are CTAs for what
  // is left over, at most ga.deep of them).
  int passes = 0;
  __shared__ int2 walk_s;  // first pass over the matrix's entries and step (kept here, and count_s, to spare registers)
  const uint8_t* wmat = a.w;
  int2* list = reinterpret_cast<int2*>(rw_dyn + pl.list_off);  // (row of x, row of y)
  if constexpr (G) {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the routing may come from the kernel before this one
    constexpr int TH = RowsShape<G>::kThreads;
    __shared__ int2 found_s;
    const int share = (int)gridDim.z, base = ga.deep * share;
    const bool more = (int)gridDim.y > ga.units, left_over = (int)blockIdx.y >= ga.units;
    uint32_t e;
    int pass0 = (int)blockIdx.z, pass_step = share;
    if (left_over) {
      const int2 f = rows_left_over<TH>(ga, 8 * NT, base, ((int)blockIdx.y - ga.units) * share + (int)blockIdx.z,
                                        reinterpret_cast<int*>(rw_dyn), &found_s);
      e = (uint32_t)f.x;
      pass0 = f.y;
      pass_step = 1;
    } else {
      e = ga.by_entry ? ga.rhs[blockIdx.y] : blockIdx.y;
    }
    if (e >= (uint32_t)ga.n_experts) return;
    if (threadIdx.x == 0) walk_s = make_int2(pass0, pass_step);
    const bool shared = ga.by_entry || share > 1 || left_over;
    const int total_m = collect_entries<TH>(ga.rhs, ga.lhs, ga.n_entries, ga.x_batch, e, list, &count_s,
                                            shared ? 0 : (more ? 8 * NT * base : ga.n_entries));
    if (total_m == 0 || (ga.by_entry && !left_over && list[0].y != (int)blockIdx.y)) return;
    wmat += (long long)e * ga.expert_stride;
    passes = ((total_m + 8 * NT - 1) / (8 * NT) - pass0 + pass_step - 1) / pass_step;
    if (more) passes = min(passes, ga.deep);
    if (passes <= 0) return;
  } else {
    passes = (pl.n_blocks - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;
  }
  auto row_block = [&](int pass) { return ((int)blockIdx.x + (G ? 0 : pass * (int)gridDim.x)) * pl.R; };
  auto entry0 = [&](int pass) { return 8 * NT * (walk_s.x + pass * walk_s.y); };  // of the pass (gather)
  auto rows_of_x = [&](int pass) { return G ? min(8 * NT, count_s - entry0(pass)) : a.M; };
  volatile int* abort_flag = &abort_s;
  auto wait = [&](uint64_t* bar, int parity) { return mbar_wait_err(bar, parity, abort_flag, 0x100, error_word); };

  if (warp >= NW + kRwHelpers) {
    // ================= producers =================
    const int pw = warp - NW - kRwHelpers;
    const int total = passes * nst;
    const uint8_t* wend = wmat + (long long)a.N * a.row_bytes;
    int pass_w = 0, st_w = 0, slot_w = 0, pass_x = 0, st_x = 0, slot_x = 0;
    // A row's pieces of sixteen bytes go to neighbouring threads (a power of two of them, 1 << wlog: pl.wlog, pl.xlog),
    // every thread walks down the rows: two additions a piece (numbering the pieces of a stage and
    // stepping by the thread count instead: q6_k [4096, 14336] x 8 32 us against 24).
    const int tid = pw * 32 + lane;
    constexpr int kThreads = 32 * kRwProducers;
    auto copy_w = [&]() {
      const int row0 = row_block(pass_w), rows = min(pl.R, a.N - row0), len = min(pl.cs, nsb - st_w * pl.cs) * BPB;
      const int step = kThreads >> pl.wlog, r0 = tid >> pl.wlog;
      const uint8_t* src = wmat + (long long)row0 * a.row_bytes + (long long)st_w * pl.cs * BPB;
      const uint32_t dst = smem_u32(rw_dyn + slot_w * pl.stage_bytes);
      const long long sstep = step * a.row_bytes;
      const int dstep = step * pl.wpitch;
      if (rw_al16(C) || (a.row_bytes & 15) == 0) {
        // every row has the same place within sixteen bytes, and the matrix ends on a whole sixteen
        const int ph = rw_al16(C) ? 0 : (int)(reinterpret_cast<uintptr_t>(src) & 15);
        const int per_row = (len + ph + 15) >> 4;
        for (int c = tid & ((1 << pl.wlog) - 1); c < per_row; c += 1 << pl.wlog) {
          const uint8_t* p = src - ph + 16 * c + r0 * a.row_bytes;
          uint32_t d = dst + 16 * c + r0 * pl.wpitch;
#pragma unroll 4
          for (int r = r0; r < rows; r += step, p += sstep, d += dstep) rw_cp16(d, p);
        }
      } else {  // the aligned window around the row's bytes; the matrix may end inside it
        const int per_row = (len + 30) >> 4;  // a window holds at most that many
        for (int c = tid & ((1 << pl.wlog) - 1); c < per_row; c += 1 << pl.wlog) {
          const uint8_t* p = src + r0 * a.row_bytes;
          uint32_t d = dst + 16 * c + r0 * pl.wpitch;
#pragma unroll 4
          for (int r = r0; r < rows; r += step, p += sstep, d += dstep) {
            const int ph = (int)(reinterpret_cast<uintptr_t>(p) & 15);
            const uint8_t* q = p - ph + 16 * c;
            const long long left = wend - q;
            if (16 * c < len + ph) rw_cp16_upto(d, q, left < 16 ? (int)left : 16);
          }
        }
      }
      if (++st_w == nst) st_w = 0, pass_w++;
      if (++slot_w == S) slot_w = 0;
    };
    auto copy_x = [&]() {  // and the arrival of this thread once all its copies of the stage have landed
      const int per_row = min(pl.cs, nsb - st_x * pl.cs) * 32, m = rows_of_x(pass_x);
      const int step = kThreads >> pl.xlog, r0 = tid >> pl.xlog;
      const uint32_t dst = smem_u32(rw_dyn + slot_x * pl.stage_bytes + pl.x_off);
      const XT* src = static_cast<const XT*>(a.x) + st_x * pl.cs * 256;
      for (int c = tid & ((1 << pl.xlog) - 1); c < per_row; c += 1 << pl.xlog) {
#pragma unroll 2
        for (int r = r0; r < m; r += step) {
          const int row = G ? list[entry0(pass_x) + r].x : r;
          rw_cp16(dst + r * pl.xpitch + 16 * c, src + ((long long)row * a.x_row_stride + 8 * c));
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(&full[slot_x])) : "memory");
      if (++st_x == nst) st_x = 0, pass_x++;
      if (++slot_x == S) slot_x = 0;
    };
    const int first = min(S, total);
    // x and, for all that is known here, the weights may come from the kernel before this one
    if constexpr (!G) asm volatile("griddepcontrol.wait;\n" ::: "memory");
    for (int i = 0; i < first; i++) copy_w();
    for (int i = 0; i < first; i++) copy_x();
    int parity = 0;
    for (int i = first; i < total; i++) {
      if (!wait(&empty[slot_w], parity)) break;
      if (slot_w == S - 1) parity ^= 1;
      copy_w();
      copy_x();
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  } else if (warp >= NW) {
    // ================= helpers: the stage's activation sums =================
    if constexpr (kSums) {
      int s = 0, parity = 0, st = 0, pass = 0;
      for (int i = 0; i < passes * nst; i++) {
        const int m = rows_of_x(pass);
        const int here = min(pl.cs, nsb - st * pl.cs);
        if (!wait(&full[s], parity)) break;
        const uint8_t* xs = rw_dyn + (long long)s * pl.stage_bytes + pl.x_off;
        float* sums = reinterpret_cast<float*>(rw_dyn + (long long)s * pl.stage_bytes + pl.sum_off);
        for (int e = warp - NW; e < here * NT; e += kRwHelpers) {
          const int k = e / NT, n = e % NT;
          if (8 * n >= m) continue;
          rows_sums<C, XT>(xs + min(8 * n + (lane >> 2), m - 1) * pl.xpitch + 512 * k,
                           sums + (k * NT + n) * 8 * rw_sum_pitch(C), lane);
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&ready[s]);
          mbar_arrive(&empty[s]);
        }
        if (++st == nst) st = 0, pass++;
        if (++s == S) s = 0, parity ^= 1;
      }
    }
  } else if (warp < live) {
    // ================= consumers: warp = (row tile, superblock of the stage) =================
    const int tile = warp % pl.rt, ks = warp / pl.rt;
    const int g = lane >> 2, t = lane & 3;
    float* red = reinterpret_cast<float*>(rw_dyn + pl.red_off);
    constexpr int kRedPitch = 8 * NT + 2;
    bool ok = true;
    int s = 0, parity = 0;
    for (int pass = 0; pass < passes; pass++) {
      const int row0 = row_block(pass), rows = min(pl.R, a.N - row0), m = rows_of_x(pass);
      const int p0 = row_of(16 * tile + g), p1 = row_of(16 * tile + g + 8);
      const int l0 = min(p0, rows - 1), l1 = min(p1, rows - 1);  // places past the end read some row, to no effect
      float y[NT][4];
      int xo[NT];  // this lane's activation rows
#pragma unroll
      for (int n = 0; n < NT; n++) {
        y[n][0] = y[n][1] = y[n][2] = y[n][3] = 0.f;
        xo[n] = pl.x_off + min(8 * n + g, m - 1) * pl.xpitch;
      }
      const int w0 = l0 * pl.wpitch, w1 = l1 * pl.wpitch;
      for (int st = 0; st < nst; st++) {
        if (ok) ok = wait(kSums ? &ready[s] : &full[s], parity);
        const uint8_t* base = rw_dyn + s * pl.stage_bytes;
        const int here = ok ? min(pl.cs, nsb - st * pl.cs) : 0;
        for (int k = ks; k < here; k += pl.wk) {
          const uint8_t *r0 = base + w0 + k * BPB, *r1 = base + w1 + k * BPB;
          if constexpr (!rw_al16(C)) {  // the bytes of a row start at their offset within a 16-byte word
            // (a place past the end keeps its own offset: all lanes agree modulo four)
            const long long o0 = (long long)(row0 + p0) * a.row_bytes + (long long)st * pl.cs * BPB;
            const long long o1 = (long long)(row0 + p1) * a.row_bytes + (long long)st * pl.cs * BPB;
            r0 += (int)(o0 & 15), r1 += (int)(o1 & 15);
          }
          const uint8_t* xb[NT];
#pragma unroll
          for (int n = 0; n < NT; n++) xb[n] = base + xo[n] + 512 * k;
          const float* sums = reinterpret_cast<const float*>(base + pl.sum_off) + k * NT * 8 * rw_sum_pitch(C);
          if (!G || NT == 1 || m > 8) {
            RowsUnit<C, XT, NT>::run(y, r0, r1, xb, sums, g, t);
          } else {  // (gather) few enough for one column tile
            const uint8_t* xb1[1] = {xb[0]};
            float y1[1][4] = {{y[0][0], y[0][1], y[0][2], y[0][3]}};
            RowsUnit<C, XT, 1>::run(y1, r0, r1, xb1, sums, g, t);
            y[0][0] = y1[0][0], y[0][1] = y1[0][1], y[0][2] = y1[0][2], y[0][3] = y1[0][3];
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (++s == S) s = 0, parity ^= 1;
      }
      // the superblock columns of a row meet in shared memory, in a fixed order
      float* mine = red + (long long)(ks * pl.rt * 16 + 16 * tile + g) * kRedPitch + 2 * t;
#pragma unroll
      for (int n = 0; n < NT; n++) {
        *reinterpret_cast<float2*>(mine + 8 * n) = make_float2(y[n][0], y[n][1]);
        *reinterpret_cast<float2*>(mine + 8 * kRedPitch + 8 * n) = make_float2(y[n][2], y[n][3]);
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(live * 32) : "memory");
      if (ok) {
        const int rp = pl.rt * 16;
        for (int e = threadIdx.x; e < rp * m; e += live * 32) {
          const int place = e % rp, c = e / rp, r = row_of(place);
          if (r < rows) {
            float v = 0.f;
            for (int k = 0; k < pl.wk; k++) v += red[(long long)(k * rp + place) * kRedPitch + c];
            const int2 entry = G ? list[entry0(pass) + c] : make_int2(c, c);  // (row of x, row of y)
            if (!(fabsf(v) < INFINITY))
              v = rows_plain<C, XT>(wmat + (row0 + r) * a.row_bytes,
                                    static_cast<const XT*>(a.x) + entry.x * a.x_row_stride, nsb);
            if (a.row_scale != nullptr) v *= a.row_scale[c];
            const int orow = entry.y;
            const long long o = (long long)orow * a.y_row_stride + row0 + r;
            if (kBf || a.out_bf16) static_cast<__nv_bfloat16*>(a.y)[o] = __float2bfloat16_rn(v);
            else static_cast<__half*>(a.y)[o] = __float2half_rn(v);
          }
        }
      }
      asm volatile("bar.sync 1, %0;\n" ::"r"(live * 32) : "memory");
    }
  }
}

int rows_sm_count() {
  static int sms[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return 0;
  if (sms[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 0;
    sms[dev] = n;
  }
  return sms[dev];
}

// Row blocks as even as the SM count allows, one per SM and pass; a stage as deep as the warps left over by the
// row tiles can take, shortened until three stages (or all of K) fit shared memory.
template <int C, bool BF, int NT, bool G>
bool rows_plan(const GemvArgs& a, RowsPlan& p, int units) {
  constexpr int NW = RowsShape<G>::kWarps, BPB = bpb_of(C), kMaxSmem = RowsShape<G>::kMaxSmem;
  const int sms = rows_sm_count();
  if (sms <= 0) return false;
  const int nsb = a.K >> 8, max_m = G ? 8 * NT : a.M;
  int r0;
  if (G) {
    // whole blocks of 128 rows where they fill the SMs several times over, smaller ones for fewer matrices
    r0 = 128;
    while (r0 > 32 && (long long)units * ((a.N + r0 - 1) / r0) < 2 * sms) r0 /= 2;
  } else {
    const int passes = (a.N + sms * 16 * NW - 1) / (sms * 16 * NW);
    r0 = std::max(8, (a.N + sms * passes - 1) / (sms * passes));
  }
  const bool alternate = (a.row_bytes & 3) != 0;
  if (alternate) r0 = (r0 + 31) & ~31;  // whole tiles of either kind
  // three stages (or all of K), for the gather form rather with fewer rows; two always fit
  for (int want = 3; want >= 2; want--) {
    for (p.R = r0; p.R == r0 || (G && p.R >= 32); p.R /= 2) {
      p.n_blocks = (a.N + p.R - 1) / p.R;
      p.rt = (p.R + 15) / 16;
      p.half = alternate ? p.R / 2 : 0;
      p.wk = std::min(NW / p.rt, nsb);
      for (p.cs = std::min(2 * p.wk, nsb); p.cs >= 1; p.cs--) {
        p.wk = std::min(p.wk, p.cs);
        int wb = p.cs * BPB;
        if (!rw_al16(C)) wb = (wb + 30 + 15) & ~15;
        // 8-byte reads of four rows, or 4-byte reads of eight, in different banks
        while (rw_al16(C) ? (wb & 63) != 32 : (wb & 31) != 16) wb += 16;
        p.wpitch = wb;
        auto log2_of = [&](int pieces) {
          int l = 0;
          while ((1 << l) < pieces && (2 << l) <= 32 * RowsShape<G>::kProducers) l++;
          return l;
        };
        p.wlog = log2_of((p.cs * BPB + (rw_al16(C) ? 15 : 30)) >> 4);
        p.xlog = log2_of(p.cs * 32);
        p.xpitch = p.cs * 512 + (rw_al16(C) ? 64 : 32);  // 16- and 8-byte reads of the B operand
        p.x_off = (p.R * p.wpitch + 127) & ~127;
        p.sum_off = (p.x_off + max_m * p.xpitch + 15) & ~15;
        p.stage_bytes = (p.sum_off + (rw_sums<C, BF>() ? p.cs * NT * 8 * rw_sum_pitch(C) * 4 : 0) + 127) & ~127;
        const int red = p.wk * p.rt * 16 * (8 * NT + 2) * 4;
        const int nst = (nsb + p.cs - 1) / p.cs * (G ? 1 : (p.n_blocks + sms - 1) / sms);
        p.stages = std::min({kRwMaxStages, nst, (kMaxSmem - red - (G ? 8 * kRwMaxEntries : 0)) / p.stage_bytes});
        if (p.stages >= std::min(want, nst)) {
          p.red_off = p.stages * p.stage_bytes;
          p.list_off = p.red_off + ((red + 15) & ~15);
          p.smem = p.list_off + (G ? 8 * kRwMaxEntries : 0);
          return true;
        }
      }
    }
  }
  return false;
}

template <int C, typename XT, int NT, bool G>
cudaError_t launch_rows_nt(const GemvArgs& a, const RowsGather& ga, cudaStream_t st) {
  RowsPlan p;
  const int units = G ? std::min(ga.n_entries, ga.n_experts) : 1;
  if (!rows_plan<C, std::is_same<XT, __nv_bfloat16>::value, NT, G>(a, p, units)) return cudaErrorInvalidConfiguration;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(rows_kernel<C, XT, NT, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         RowsShape<G>::kMaxSmem);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  int* err = device_error_word();
  if (err == nullptr) return cudaErrorUnknown;
  cudaLaunchConfig_t cfg = {};
  // routing may be uneven: while all CTAs are resident at once, several share a matrix's entries
  int share = 1;
  if (G) share = std::max(1, std::min((ga.n_entries + 8 * NT - 1) / (8 * NT), RowsShape<G>::kCtas * rows_sm_count() / (p.n_blocks * units)));
  // ... and what is more than `deep` passes a CTA goes to CTAs of its own: a matrix of c entries leaves at most
  // (c - 1) / (8 NT deep) - share + 1 groups. Where there are none such a CTA costs some 1.5 us, a pass over few superblocks
  // 3-4 us: two passes there, one where K is long. Before, a busy matrix's passes ran one after the other. 128 matrices
  // of iq4_xs [768, 2048], 512 entries, a fifth of them in one: 221 -> 83 us (the general path 102), evenly at random
  // 85 -> 72; q4_k [512, 512] 1024 entries 83 -> 35, evenly 20.3 -> 20.4.
  RowsGather gl = ga;
  gl.units = units;
  gl.deep = a.K >= 1536 ? 1 : 2;
  int more = 0;
  if (G && 4ll * ga.n_experts <= p.red_off) more = std::max(0, (ga.n_entries - 1) / (8 * NT * gl.deep) - share + 1);
  more = (more + share - 1) / share;
  if (units + more > 65535) more = 0;
  cfg.gridDim = G ? dim3(p.n_blocks, units + more, share) : dim3(std::min(p.n_blocks, rows_sm_count()), 1, 1);
  cfg.blockDim = dim3(RowsShape<G>::kThreads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  static const bool no_pdl = std::getenv("KQ_NO_PDL") != nullptr;  // A/B lever
  cfg.numAttrs = no_pdl ? 0 : 1;
  return cudaLaunchKernelEx(&cfg, rows_kernel<C, XT, NT, G>, a, p, gl, err);
}

template <int C, typename XT>
cudaError_t launch_rows_c(const GemvArgs& a, const RowsGather* ga, cudaStream_t st) {
  // gather: with more than six entries a matrix on average, many have more than eight
  if (ga != nullptr)
    return ga->n_entries <= 6 * ga->n_experts ? launch_rows_nt<C, XT, 1, true>(a, *ga, st)
                                              : launch_rows_nt<C, XT, 2, true>(a, *ga, st);
  if (a.M <= 8) return launch_rows_nt<C, XT, 1, false>(a, RowsGather{}, st);
  return launch_rows_nt<C, XT, 2, false>(a, RowsGather{}, st);
}

cudaError_t launch_rows_any(int codec, int x_dtype, const GemvArgs& a, const RowsGather* ga, cudaStream_t st) {
  if (x_dtype == F16) {
    switch (codec) {
      case Q4_K: return launch_rows_c<Q4_K, __half>(a, ga, st);
      case Q5_K: return launch_rows_c<Q5_K, __half>(a, ga, st);
      case Q6_K: return launch_rows_c<Q6_K, __half>(a, ga, st);
      case IQ4_XS: return launch_rows_c<IQ4_XS, __half>(a, ga, st);
    }
  } else {
    switch (codec) {
      case Q4_K: return launch_rows_c<Q4_K, __nv_bfloat16>(a, ga, st);
      case Q5_K: return launch_rows_c<Q5_K, __nv_bfloat16>(a, ga, st);
      case Q6_K: return launch_rows_c<Q6_K, __nv_bfloat16>(a, ga, st);
      case IQ4_XS: return launch_rows_c<IQ4_XS, __nv_bfloat16>(a, ga, st);
    }
  }
  return cudaErrorInvalidValue;
}

}  // namespace

bool gemv_rows_supported(int codec, int x_dtype, const GemvArgs& a) {
  if (codec != Q4_K && codec != Q5_K && codec != Q6_K && codec != IQ4_XS) return false;
  if (!(x_dtype == F16 || x_dtype == BF16) || a.tasks != nullptr || a.bias != nullptr || a.M < 1 || a.M > 16 || a.N < 8 ||
      a.K < 256 || (a.K & 255) != 0 || a.w_align16 == 0 || a.row_bytes != (long long)(a.K >> 8) * bpb_of(codec))
    return false;
  // iq4_xs: the table lookups (23 instructions for eight weights against 7 of the others) bound it on large matrices:
  // [1000, 1280] x 2 rows 10.3 -> 3.6 us, but [14336, 4096] 22.7 against 28.9
  if (codec == IQ4_XS && (long long)a.N * a.K > (4ll << 20)) return false;
  return (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (a.x_row_stride & 7) == 0;
}

cudaError_t launch_gemv_rows(int codec, int x_dtype, const GemvArgs& a, cudaStream_t st) {
  return launch_rows_any(codec, x_dtype, a, nullptr, st);
}

// gather_qmm with one activation row per entry, in one launch: no grouping passes and no scratch.
bool gather_rows_supported(int codec, int x_dtype, const void* x, int M, int K, const uint8_t* w, long long expert_stride,
                           long long row_bytes, int N, long long n_entries, int n_experts) {
  if (M != 1 || n_entries > kRwMaxEntries || n_experts > 65535 || (expert_stride & 15) != 0) return false;
  // q4_k has a grouped kernel of its own for matrices of this size, as fast from eight entries a matrix on unless K is
  // long: 1024 entries of 128 matrices [2048, 768] 96 us there and 91 here evenly at random, 100 and 108 with a fifth of
  // them in one matrix; 512 entries 88 and 66, 85 and 71; 1024 of [768, 2048] 84 and 70, 84 and 77.
  if (codec == Q4_K && (long long)N * K > (1 << 20) && K < 1536 && n_entries >= 8ll * n_experts) return false;
  GemvArgs a{};
  a.x = x;
  a.x_row_stride = K;
  a.w_align16 = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  a.row_bytes = row_bytes;
  a.N = N;
  a.K = K;
  a.M = 1;
  return gemv_rows_supported(codec, x_dtype, a);
}

cudaError_t launch_gather_rows(int codec, int x_dtype, const void* x, long long x_batch, int K, const uint8_t* w,
                               int n_experts, long long expert_stride, long long row_bytes, int N, const uint32_t* lhs,
                               const uint32_t* rhs, long long n_entries, void* y, cudaStream_t st) {
  GemvArgs a{};
  a.x = x;
  a.x_row_stride = K;
  a.y = y;
  a.y_row_stride = N;
  a.w = w;
  a.w_align16 = 1;
  a.row_bytes = row_bytes;
  a.N = N;
  a.K = K;
  RowsGather ga{lhs, rhs, (int)n_entries, n_experts, n_entries < n_experts ? 1 : 0, x_batch, expert_stride};
  return launch_rows_any(codec, x_dtype, a, &ga, st);
}

}  // namespace kq
