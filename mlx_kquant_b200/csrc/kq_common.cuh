// Shared device-side pieces of the quantized-weight path: the codec registry,
// alignment-aware little loaders, and decode8<> - the bit-exact decoder of
// eight consecutive weights of one block, used by every kernel that needs
// real-valued weights (dequantize, the generic skinny-M matmul, the prefill
// tile producer).
//
// Numerics contract (matches the reference's CPU block decoders,
// src/kquant_cpu_decode.cpp:50-82, 155-397, 441-465, 557-584): every product is
// formed in fp32 in the reference's association order. All of them are exact
// in fp32 (an 11-bit fp16 scale times at most 13 bits of integers), so the only
// rounding is the final subtract of the min-offset codecs, where a fused
// multiply-add and multiply-then-subtract round identically. The file must not
// be compiled with --use_fast_math / -ftz=true: small weights of the min-offset
// codecs are fp16 subnormals on output.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

// The GGUF IQ lookup tables (generated by gen_tables.py) as per-translation-unit
// __device__ arrays: kq_tab_iq4nl[16], kq_tab_iq2xxs_grid[256], kq_tab_ksigns[128], kq_tab_mxfp4[16],
// kq_tab_iq3xxs_grid[256], kq_tab_iq3s_grid[512], kq_tab_iq2xs_grid[512], kq_tab_iq2s_grid[1024],
// kq_tab_iq1s_grid[2048].
#define KQ_TAB_QUAL static __device__
#include "kq_iq_tables.inc"

namespace kq {

// Registry order is the ABI's codec index (kq_codec_info). Geometry follows the
// reference registry, src/kquant_codec.cpp:12-37.
enum Codec : int {
  Q2_K = 0, Q3_K, Q4_K, Q5_K, Q6_K, Q4_0, Q8_0, IQ4_NL, IQ4_XS, IQ2_XXS, Q4_1, Q5_0, Q5_1,
  IQ3_XXS, IQ3_S, IQ2_XS, IQ2_S, IQ1_S, IQ1_M, MXFP4, NVFP4, NUM_CODECS
};

struct CodecInfo {
  const char* name;
  int wpb;   // weights per block
  int bpb;   // bytes per block
  int bits;
  int requires_imatrix;
  int natural_align;  // largest power of two dividing bpb, capped at 16
};

__host__ __device__ constexpr int wpb_of(int c) {
  return (c == Q4_0 || c == Q8_0 || c == IQ4_NL || c == Q4_1 || c == Q5_0 || c == Q5_1 || c == MXFP4) ? 32
       : (c == NVFP4 ? 64 : 256);
}
__host__ __device__ constexpr int bpb_of(int c) {
  return c == Q2_K ? 84 : c == Q3_K ? 110 : c == Q4_K ? 144 : c == Q5_K ? 176 : c == Q6_K ? 210
       : c == Q4_0 ? 18 : c == Q8_0 ? 34 : c == IQ4_NL ? 18 : c == IQ4_XS ? 136 : c == Q4_1 ? 20 : c == Q5_0 ? 22
       : c == Q5_1 ? 24 : c == IQ3_XXS ? 98 : c == IQ3_S ? 110 : c == IQ2_XS ? 74 : c == IQ2_S ? 82 : c == IQ1_S ? 50
       : c == IQ1_M ? 56 : c == MXFP4 ? 17 : c == NVFP4 ? 36 : 66;
}
// weights k .. k + 7 (k a multiple of 8) of a row: which block, which octet of it
template <int C>
__host__ __device__ constexpr long long block_of(long long k) { return k / wpb_of(C); }
template <int C>
__host__ __device__ constexpr int octet_of(long long k) { return (int)(k % wpb_of(C)) >> 3; }

static const CodecInfo kCodecs[NUM_CODECS] = {
    {"q2_k", 256, 84, 2, 0, 4},    {"q3_k", 256, 110, 3, 0, 2},  {"q4_k", 256, 144, 4, 0, 16},
    {"q5_k", 256, 176, 5, 0, 16},  {"q6_k", 256, 210, 6, 0, 2},  {"q4_0", 32, 18, 4, 0, 2},
    {"q8_0", 32, 34, 8, 0, 2},     {"iq4_nl", 32, 18, 4, 0, 2},  {"iq4_xs", 256, 136, 4, 0, 8},
    {"iq2_xxs", 256, 66, 2, 1, 2}, {"q4_1", 32, 20, 4, 0, 4},    {"q5_0", 32, 22, 5, 0, 2},
    {"q5_1", 32, 24, 5, 0, 8},     {"iq3_xxs", 256, 98, 3, 0, 2}, {"iq3_s", 256, 110, 3, 0, 2},
    {"iq2_xs", 256, 74, 2, 1, 2},  {"iq2_s", 256, 82, 2, 0, 2},   {"iq1_s", 256, 50, 1, 1, 2},
    {"iq1_m", 256, 56, 1, 0, 8},   {"mxfp4", 32, 17, 4, 0, 1},    {"nvfp4", 64, 36, 4, 0, 4},
};

enum DType : int { F32 = 0, F16 = 1, BF16 = 2 };

// IQ lookup tables handed to decode8: pointers into shared memory (kernels copy
// them there once per CTA) or into the __device__ copies below.
struct IqTables {
  const int8_t* iq4nl;     // [16]
  const uint64_t* grid;    // [256] iq2_xxs lattice
  const uint8_t* ksigns;   // [128]
  // the tables of the codecs outside the benchmark's ten stay in global memory
  const uint32_t* iq3xxs;  // [256]
  const uint32_t* iq3s;    // [512]
  const uint64_t* iq2xs;   // [512]
  const uint64_t* iq2s;    // [1024]
  const uint64_t* iq1s;    // [2048], signed bytes
  const int8_t* mxfp4;     // [16]
};
__device__ __forceinline__ IqTables global_iq_tables() {
  IqTables t;
  t.iq4nl = reinterpret_cast<const int8_t*>(kq_tab_iq4nl);
  t.grid = reinterpret_cast<const uint64_t*>(kq_tab_iq2xxs_grid);
  t.ksigns = kq_tab_ksigns;
  t.iq3xxs = kq_tab_iq3xxs_grid;
  t.iq3s = kq_tab_iq3s_grid;
  t.iq2xs = reinterpret_cast<const uint64_t*>(kq_tab_iq2xs_grid);
  t.iq2s = reinterpret_cast<const uint64_t*>(kq_tab_iq2s_grid);
  t.iq1s = reinterpret_cast<const uint64_t*>(kq_tab_iq1s_grid);
  t.mxfp4 = reinterpret_cast<const int8_t*>(kq_tab_mxfp4);
  return t;
}

// Bytes of shared memory stage_iq_tables() fills: grid 2048 + ksigns 128 + lut 16.
constexpr int kIqSmemBytes = 2048 + 128 + 16;

// ---- loads with a compile-time alignment guarantee A on the BLOCK start and a
// compile-time-known offset parity; `off` must itself be a multiple of what is
// asked for when A allows the wide load. ----
template <int A>
__device__ __forceinline__ uint32_t ld16(const uint8_t* p) {
  if constexpr (A >= 2) {
    return *reinterpret_cast<const uint16_t*>(p);
  } else {
    return (uint32_t)p[0] | ((uint32_t)p[1] << 8);
  }
}
template <int A>
__device__ __forceinline__ uint32_t ld32(const uint8_t* p) {
  if constexpr (A >= 4) {
    return *reinterpret_cast<const uint32_t*>(p);
  } else if constexpr (A >= 2) {
    return (uint32_t)*reinterpret_cast<const uint16_t*>(p) |
           ((uint32_t)*reinterpret_cast<const uint16_t*>(p + 2) << 16);
  } else {
    return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
  }
}
template <int A>
__device__ __forceinline__ float ldf16(const uint8_t* p) {
  return __half2float(__ushort_as_half((unsigned short)ld16<A>(p)));
}

// Small integers to float through the mantissa of 2^23 (exact): one permute or logic instruction and one subtraction
// where the conversion instruction runs at a quarter of the rate or less. A decode of eight weights had eight of them.
__device__ __forceinline__ float u2f(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.f; }  // v < 2^23
// byte c of w, minus `off`
__device__ __forceinline__ float b2f(uint32_t w, int c, float off = 0.f) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + c)) - (8388608.f + off);
}

// Eight 6-bit (scale, min) pairs packed in 12 bytes (q4_k / q5_k),
// src/kquant_cpu_decode.cpp:155-174. s0..s2 are the three little-endian words.
__device__ __forceinline__ void k4_scale_min(uint32_t s0, uint32_t s1, uint32_t s2, int i, uint32_t& sc,
                                             uint32_t& mn) {
  // byte b of the 12: word b/4, shift 8*(b%4)
  auto byte_at = [&](int b) -> uint32_t {
    uint32_t w = b < 4 ? s0 : (b < 8 ? s1 : s2);
    return (w >> (8 * (b & 3))) & 0xffu;
  };
  if (i < 4) {
    sc = byte_at(i) & 63u;
    mn = byte_at(i + 4) & 63u;
  } else {
    sc = (byte_at(i + 4) & 15u) | ((byte_at(i - 4) >> 6) << 4);
    mn = (byte_at(i + 4) >> 4) | ((byte_at(i) >> 6) << 4);
  }
}

// decode8<C, A>(blk, j, v, tabs): weights 8j .. 8j+7 of the block at `blk`
// (any address space), A = guaranteed alignment of blk in bytes (1, 2, 4, 8, 16).
template <int C, int A>
__device__ __forceinline__ void decode8(const uint8_t* __restrict__ blk, int j, float (&v)[8], const IqTables& tabs) {
  if constexpr (C == Q8_0) {
    // [f16 d][32 x int8], src/kquant_cpu_decode.cpp:50-63
    const float d = ldf16<A>(blk);
    const uint32_t a = ld32<(A >= 2 ? 2 : 1)>(blk + 2 + 8 * j);
    const uint32_t b = ld32<(A >= 2 ? 2 : 1)>(blk + 6 + 8 * j);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      v[c] = d * b2f(a ^ 0x80808080u, c, 128.f);
      v[c + 4] = d * b2f(b ^ 0x80808080u, c, 128.f);
    }
  } else if constexpr (C == Q4_0 || C == IQ4_NL) {
    // [f16 d][16 B nibbles]: low nibble -> weight i, high nibble -> weight i+16,
    // src/kquant_cpu_decode.cpp:66-82, 383-397
    const float d = ldf16<A>(blk);
    const int hi = j >> 1;  // octets 2,3 are the high nibbles
    const uint8_t* q = blk + 2 + 8 * (j & 1);
    const uint32_t a = ld32<(A >= 2 ? 2 : 1)>(q);
    const uint32_t b = ld32<(A >= 2 ? 2 : 1)>(q + 4);
    const uint32_t na = (hi ? a >> 4 : a) & 0x0f0f0f0fu, nb = (hi ? b >> 4 : b) & 0x0f0f0f0fu;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      if constexpr (C == Q4_0) {
        v[c] = d * b2f(c < 4 ? na : nb, c & 3, 8.f);
      } else {
        v[c] = d * (float)tabs.iq4nl[((c < 4 ? na : nb) >> (8 * (c & 3))) & 15u];
      }
    }
  } else if constexpr (C == Q4_1 || C == Q5_0 || C == Q5_1) {
    // q4_1 [d][m][16 B nibbles]: d q + m; q5_0 [d][qh u32][16 B]: d (q - 16), bit i of qh is the fifth bit of
    // weight i; q5_1 [d][m][qh][16 B]: d q + m (src/kquant_cpu_decode.cpp:84-153). d q is exact in fp32, so the
    // product-then-add here rounds once, like the reference's expression.
    constexpr int kQs = C == Q4_1 ? 4 : (C == Q5_0 ? 6 : 8);
    const float d = ldf16<A>(blk);
    float m = 0.f;
    if constexpr (C != Q5_0) m = ldf16<A>(blk + 2);
    uint32_t qh = 0;
    if constexpr (C == Q5_0) qh = ld32<(A >= 2 ? 2 : 1)>(blk + 2);
    if constexpr (C == Q5_1) qh = ld32<(A >= 4 ? 4 : (A >= 2 ? 2 : 1))>(blk + 4);
    const int hi = j >> 1;  // octets 2, 3 are the high nibbles
    const uint8_t* q = blk + kQs + 8 * (j & 1);
    const uint32_t a = ld32<(A >= 2 ? 2 : 1)>(q);
    const uint32_t b = ld32<(A >= 2 ? 2 : 1)>(q + 4);
    uint32_t na = (hi ? a >> 4 : a) & 0x0f0f0f0fu, nb = (hi ? b >> 4 : b) & 0x0f0f0f0fu;
    if constexpr (C != Q4_1) {  // four bits spread over four bytes by a multiplication
      const uint32_t u = qh >> (8 * j);
      na |= (((u & 15u) * 0x00204081u) & 0x01010101u) << 4;
      nb |= ((((u >> 4) & 15u) * 0x00204081u) & 0x01010101u) << 4;
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
      if constexpr (C == Q5_0) v[c] = d * b2f(c < 4 ? na : nb, c & 3, 16.f);
      else v[c] = d * b2f(c < 4 ? na : nb, c & 3) + m;
    }
  } else if constexpr (C == Q4_K || C == Q5_K) {
    // q4_k: [d][dmin][12 B scales][128 B qs]; q5_k adds qh[32] at +16, qs at +48,
    // src/kquant_cpu_decode.cpp:177-235
    const uint32_t h = ld32<A>(blk);
    const float d = __half2float(__ushort_as_half((unsigned short)(h & 0xffff)));
    const float dmin = __half2float(__ushort_as_half((unsigned short)(h >> 16)));
    const uint32_t s0 = ld32<A>(blk + 4), s1 = ld32<A>(blk + 8), s2 = ld32<A>(blk + 12);
    const int s = j >> 2;          // 32-weight sub-block 0..7
    const int i0 = (j & 3) * 8;    // first weight inside the sub-block
    uint32_t rsc, rmn;
    k4_scale_min(s0, s1, s2, s, rsc, rmn);
    const float sc = d * u2f(rsc);
    const float mn = dmin * u2f(rmn);
    const uint8_t* qs = blk + (C == Q4_K ? 16 : 48) + (s >> 1) * 32 + i0;
    const uint32_t a = ld32<A>(qs), b = ld32<A>(qs + 4);
    uint32_t ha = 0, hb = 0;
    if constexpr (C == Q5_K) {
      ha = ld32<A>(blk + 16 + i0) >> s;
      hb = ld32<A>(blk + 20 + i0) >> s;
    }
    const int sh = (s & 1) * 4;
    uint32_t na = (a >> sh) & 0x0f0f0f0fu, nb = (b >> sh) & 0x0f0f0f0fu;
    if constexpr (C == Q5_K) {
      na |= (ha & 0x01010101u) << 4;
      nb |= (hb & 0x01010101u) << 4;
    }
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = sc * b2f(c < 4 ? na : nb, c & 3) - mn;
  } else if constexpr (C == Q6_K) {
    // [ql 128][qh 64][int8 sc 16][f16 d @208], src/kquant_cpu_decode.cpp:238-280
    const float d = ldf16<A>(blk + 208);
    const int half = j >> 4;
    const int jj = j & 15;
    const int qd = jj >> 2;          // 0: l, 1: l+32, 2: l+64, 3: l+96
    const int l0 = (jj & 3) * 8;
    const uint8_t* ql = blk + half * 64 + ((qd & 1) ? 32 : 0) + l0;
    const uint8_t* qh = blk + 128 + half * 32 + l0;
    const uint32_t la = ld32<A>(ql), lb = ld32<A>(ql + 4);
    const uint32_t ha = ld32<A>(qh), hb = ld32<A>(qh + 4);
    const int is = half * 8 + (l0 >> 4) + 2 * qd;
    const float dsc = d * (float)(int)(int8_t)blk[192 + is];
    const int nsh = 2 * (qd & 2);
    const uint32_t qa = ((la >> nsh) & 0x0f0f0f0fu) | (((ha >> (2 * qd)) & 0x03030303u) << 4);
    const uint32_t qb = ((lb >> nsh) & 0x0f0f0f0fu) | (((hb >> (2 * qd)) & 0x03030303u) << 4);
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = dsc * b2f(c < 4 ? qa : qb, c & 3, 32.f);
  } else if constexpr (C == Q3_K || C == Q2_K) {
    // q3_k: [hmask 32][qs 64][scales 12][d @108]; q2_k: [scales 16][qs 64][d @80][dmin @82],
    // src/kquant_cpu_decode.cpp:282-377. Output order: half h (128 w), shift si
    // (32 w), then the 32 q bytes in order.
    const int h = j >> 4;
    const int si = (j >> 2) & 3;
    const int e0 = (j & 3) * 8;
    const int is = h * 8 + si * 2 + (e0 >> 4);
    const uint8_t* q = blk + (C == Q3_K ? 32 : 16) + h * 32 + e0;
    const uint32_t a = ld32<A>(q) >> (2 * si), b = ld32<A>(q + 4) >> (2 * si);
    if constexpr (C == Q3_K) {
      const float d = ldf16<A>(blk + 108);
      const uint8_t* s = blk + 96;
      const int k = is & 3, grp = is >> 2;
      const uint32_t lo4 = ((uint32_t)s[k + ((grp & 1) ? 4 : 0)] >> ((grp & 2) ? 4 : 0)) & 15u;
      const uint32_t hi2 = ((uint32_t)s[8 + k] >> (2 * grp)) & 3u;
      const float dl = d * (float)((int)(lo4 | (hi2 << 4)) - 32);
      const uint32_t ma = ld32<A>(blk + e0) >> (h * 4 + si), mb = ld32<A>(blk + e0 + 4) >> (h * 4 + si);
      const uint32_t qa = (a & 0x03030303u) | ((ma & 0x01010101u) << 2);  // minus 4 where the mask bit is clear
      const uint32_t qb = (b & 0x03030303u) | ((mb & 0x01010101u) << 2);
#pragma unroll
      for (int c = 0; c < 8; c++) v[c] = dl * b2f(c < 4 ? qa : qb, c & 3, 4.f);
    } else {
      const uint32_t dd = ld32<A>(blk + 80);
      const float d = __half2float(__ushort_as_half((unsigned short)(dd & 0xffff)));
      const float dmin = __half2float(__ushort_as_half((unsigned short)(dd >> 16)));
      const uint32_t scb = blk[is];
      const float dl = d * u2f(scb & 15u), ml = dmin * u2f(scb >> 4);
#pragma unroll
      for (int c = 0; c < 8; c++) v[c] = dl * b2f((c < 4 ? a : b) & 0x03030303u, c & 3) - ml;
    }
  } else if constexpr (C == IQ4_XS) {
    // [d][u16 scales_h][4 B scales_l][128 B qs], src/kquant_cpu_decode.cpp:441-465
    const uint32_t h = ld32<A>(blk);
    const float d = __half2float(__ushort_as_half((unsigned short)(h & 0xffff)));
    const uint32_t sh = h >> 16;
    const uint32_t sl = ld32<A>(blk + 4);
    const int ib = j >> 2;
    const int e0 = (j & 3) * 8;
    const uint32_t ls = ((sl >> (4 * ib)) & 15u) | (((sh >> (2 * ib)) & 3u) << 4);
    const float dl = d * (float)((int)ls - 32);
    const uint8_t* q = blk + 8 + ib * 16 + (e0 & 8);
    const uint32_t a = ld32<A>(q), b = ld32<A>(q + 4);
    const int hi = e0 >> 4;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const uint32_t byte = ((c < 4 ? a : b) >> (8 * (c & 3))) & 0xff;
      v[c] = dl * (float)tabs.iq4nl[hi ? (byte >> 4) : (byte & 15u)];
    }
  } else if constexpr (C == IQ3_XXS) {
    // [d][qs 64][8 x u32: 4 x 7-bit sign index + 4-bit scale], src/kquant_cpu_decode.cpp:468-503
    const float d = ldf16<A>(blk);
    const int ib = j >> 2, l = j & 3;
    const uint32_t aux = ld32<(A >= 2 ? 2 : 1)>(blk + 66 + 4 * ib);
    const float db = d * (0.5f + (float)(aux >> 28)) * 0.5f;
    const uint32_t signs = tabs.ksigns[(aux >> (7 * l)) & 127u];
    const uint8_t* q = blk + 2 + 8 * ib + 2 * l;
    const uint32_t g1 = tabs.iq3xxs[q[0]], g2 = tabs.iq3xxs[q[1]];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float gv = (float)(((c < 4 ? g1 : g2) >> (8 * (c & 3))) & 0xffu);
      v[c] = db * gv * (((signs >> c) & 1u) ? -1.f : 1.f);
    }
  } else if constexpr (C == IQ3_S) {
    // [d][qs 64][qh 8][signs 32][scales 4], src/kquant_cpu_decode.cpp:505-556
    const float d = ldf16<A>(blk);
    const int ib = j >> 2, l = j & 3;
    const uint32_t sb = blk[106 + (ib >> 1)];
    const float db = d * (float)(1 + 2 * (int)((ib & 1) ? (sb >> 4) : (sb & 15u)));
    const uint32_t qh = blk[66 + ib];
    const uint8_t* q = blk + 2 + 8 * ib + 2 * l;
    const uint32_t g1 = tabs.iq3s[q[0] | ((qh << (8 - 2 * l)) & 256u)];
    const uint32_t g2 = tabs.iq3s[q[1] | ((qh << (7 - 2 * l)) & 256u)];
    const uint32_t signs = blk[74 + 4 * ib + l];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float gv = (float)(((c < 4 ? g1 : g2) >> (8 * (c & 3))) & 0xffu);
      v[c] = db * gv * (((signs >> c) & 1u) ? -1.f : 1.f);
    }
  } else if constexpr (C == IQ2_XS || C == IQ2_S) {
    // iq2_xs [d][32 x u16: 9-bit lattice index | 7-bit sign index][scales 8], src/kquant_cpu_decode.cpp:586-616
    // iq2_s  [d][qs 32][signs 32][qh 8][scales 8], src/kquant_cpu_decode.cpp:618-649
    const float d = ldf16<A>(blk);
    const int ib = j >> 2, l = j & 3;
    const uint32_t sb = blk[(C == IQ2_XS ? 66 : 74) + ib];
    const float db = d * (0.5f + (float)((l < 2) ? (sb & 15u) : (sb >> 4))) * 0.25f;
    uint64_t g;
    uint32_t signs;
    if constexpr (C == IQ2_XS) {
      const uint32_t q = ld16<(A >= 2 ? 2 : 1)>(blk + 2 + 2 * (4 * ib + l));
      g = tabs.iq2xs[q & 511u];
      signs = tabs.ksigns[q >> 9];
    } else {
      const uint32_t qh = blk[66 + ib];
      g = tabs.iq2s[blk[2 + 4 * ib + l] | ((qh << (8 - 2 * l)) & 0x300u)];
      signs = blk[34 + 4 * ib + l];
    }
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float gv = (float)(uint32_t)((g >> (8 * c)) & 0xff);
      v[c] = db * gv * (((signs >> c) & 1u) ? -1.f : 1.f);
    }
  } else if constexpr (C == IQ1_S) {
    // [d][qs 32][8 x u16 qh], src/kquant_cpu_decode.cpp:658-685
    const float d = ldf16<A>(blk);
    const int ib = j >> 2, l = j & 3;
    const uint32_t qh = ld16<(A >= 2 ? 2 : 1)>(blk + 34 + 2 * ib);
    const float dl = d * (float)(2 * (int)((qh >> 12) & 7u) + 1);
    const float delta = (qh & 0x8000u) ? -0.125f : 0.125f;
    const uint64_t g = tabs.iq1s[blk[2 + 4 * ib + l] | (((qh >> (3 * l)) & 7u) << 8)];
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = dl * ((float)(int)(int8_t)((g >> (8 * c)) & 0xff) + delta);
  } else if constexpr (C == IQ1_M) {
    // [qs 32][qh 16][4 x u16 scales, top nibbles = the fp16 super-scale], src/kquant_cpu_decode.cpp:687-735
    const uint32_t s01 = ld32<(A >= 4 ? 4 : A)>(blk + 48), s23 = ld32<(A >= 4 ? 4 : A)>(blk + 52);
    const uint32_t sc[4] = {s01 & 0xffffu, s01 >> 16, s23 & 0xffffu, s23 >> 16};
    const uint32_t dbits = (sc[0] >> 12) | ((sc[1] >> 8) & 0x00f0u) | ((sc[2] >> 4) & 0x0f00u) | (sc[3] & 0xf000u);
    const float d = __half2float(__ushort_as_half((unsigned short)dbits));
    const int ib = j >> 2, l = j & 3;
    const uint32_t w = sc[ib >> 1] >> (6 * (ib & 1) + (l < 2 ? 0 : 3));
    const float dl = d * (float)(2 * (int)(w & 7u) + 1);
    const uint32_t qh = blk[32 + 2 * ib + (l >> 1)];
    const uint32_t idx = blk[4 * ib + l] | ((qh << ((l & 1) ? 4 : 8)) & 0x700u);
    const float delta = (qh & ((l & 1) ? 0x80u : 0x08u)) ? -0.125f : 0.125f;
    const uint64_t g = tabs.iq1s[idx];
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = dl * ((float)(int)(int8_t)((g >> (8 * c)) & 0xff) + delta);
  } else if constexpr (C == MXFP4) {
    // [e8m0 scale][qs 16]: out[i] = d * lut[qs[i] & 15], out[i + 16] = d * lut[qs[i] >> 4], src/kquant_cpu_decode.cpp:404-419
    const uint32_t e = blk[0];
    const float d = __uint_as_float(e < 2u ? (0x00200000u << e) : ((e - 1u) << 23));   // 2^(e - 127) / 2
    const uint8_t* q = blk + 1 + 8 * (j & 1);
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = d * (float)tabs.mxfp4[(j >> 1) ? (q[c] >> 4) : (q[c] & 15u)];
  } else if constexpr (C == NVFP4) {
    // [4 x ue4m3 scale][4 x 8 bytes]: group g = 16 weights, src/kquant_cpu_decode.cpp:421-438
    const int gq = j >> 1;
    const uint32_t x = blk[gq];
    float d = 0.f;
    if (x != 0u && x != 0x7fu) {
      const int ex = (int)((x >> 3) & 15u);
      const float man = (float)(x & 7u);
      const float raw = ex == 0 ? man * 0.001953125f : ldexpf(1.0f + man * 0.125f, ex - 7);
      d = raw * 0.5f;
    }
    const uint8_t* q = blk + 4 + 8 * gq;
#pragma unroll
    for (int c = 0; c < 8; c++) v[c] = d * (float)tabs.mxfp4[(j & 1) ? (q[c] >> 4) : (q[c] & 15u)];
  } else {
    static_assert(C == IQ2_XXS, "unknown codec");
    // [d][8 x (4 grid-index bytes, u32: 4 x 7-bit sign index + 4-bit scale)],
    // src/kquant_cpu_decode.cpp:557-584
    const float d = ldf16<A>(blk);
    const int ib = j >> 2, l = j & 3;
    const uint8_t* qs = blk + 2 + 8 * ib;
    const uint32_t aux0 = ld32<(A >= 2 ? 2 : 1)>(qs);
    const uint32_t aux1 = ld32<(A >= 2 ? 2 : 1)>(qs + 4);
    const float db = d * (0.5f + (float)(aux1 >> 28)) * 0.25f;
    const uint64_t g = tabs.grid[(aux0 >> (8 * l)) & 0xff];
    const uint32_t signs = tabs.ksigns[(aux1 >> (7 * l)) & 127u];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float gv = (float)(uint32_t)((g >> (8 * c)) & 0xff);
      v[c] = db * gv * (((signs >> c) & 1u) ? -1.f : 1.f);
    }
  }
}

// silu of the mixture-of-experts block, shared by every kernel that applies it (the fused and the separate
// forms must round alike)
__device__ __forceinline__ float silu_f(float v) { return __fdividef(v, 1.f + __expf(-v)); }

// Copy the IQ tables to shared memory (call from all threads, then sync).
__device__ __forceinline__ IqTables stage_iq_tables(uint8_t* smem, int tid, int nthreads) {
  uint64_t* sg = reinterpret_cast<uint64_t*>(smem);
  uint8_t* sk = smem + 2048;
  int8_t* sl = reinterpret_cast<int8_t*>(smem + 2048 + 128);
  for (int i = tid; i < 256; i += nthreads) sg[i] = kq_tab_iq2xxs_grid[i];
  for (int i = tid; i < 128; i += nthreads) sk[i] = kq_tab_ksigns[i];
  for (int i = tid; i < 16; i += nthreads) sl[i] = kq_tab_iq4nl[i];
  IqTables t = global_iq_tables();
  t.iq4nl = sl;
  t.grid = sg;
  t.ksigns = sk;
  return t;
}

// N words from byte 4 W + odd_bits / 8 of a 16-byte aligned window on
template <int W, int N>
__device__ __forceinline__ void window_words(const uint8_t* win, uint32_t odd_bits, uint32_t (&out)[N]) {
  uint32_t w[(W + N + 4) / 4 * 4];
#pragma unroll
  for (int i = 0; i < (W + N + 4) / 4; i++) {
    const uint4 v = *reinterpret_cast<const uint4*>(win + 16 * i);
    w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < N; i++) out[i] = __funnelshift_r(w[W + i], w[W + i + 1], odd_bits);
}

// One output by itself: decoded weights times activations in float32 (float32 rows rounded to bf16 first), as the generic
// kernel has it. For outputs that a split into integers, offsets, sums and scales leaves without a finite value although they
// may have one, or an infinity: an infinite activation meets an offset's sum (inf - inf) or integers of zero, and a sum can
// overflow before its scale is applied. Rare, so one thread an output, without care for speed.
template <int C, int A, typename XT>
__device__ __forceinline__ float plain_dot(const uint8_t* w, const XT* x, int K) {
  const IqTables tabs = global_iq_tables();
  float sum = 0.f;
#pragma unroll 1
  for (int k = 0; k < K; k += 8) {
    float v[8];
    decode8<C, A>(w + block_of<C>(k) * bpb_of(C), octet_of<C>(k), v, tabs);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      float xv;
      // (from L2: the kernels start before x is written)
      if constexpr (std::is_same<XT, __half>::value) xv = __half2float(__ldcg(x + k + i));
      else if constexpr (std::is_same<XT, float>::value) xv = __bfloat162float(__float2bfloat16_rn(__ldcg(x + k + i)));
      else xv = __bfloat162float(__ldcg(x + k + i));
      sum = fmaf(xv, v[i], sum);
    }
  }
  return sum;
}

// The entries i of a gather call that multiply by matrix e, with an activation row in range, as (row of x, i), in the
// order of i (CTAs that share them must agree on it), in any if there are at most `unordered` of them; all threads of the
// CTA take part, `count` (shared) starts at 0. n at most 4 * TH.
// `meanwhile` runs in all threads while the indices are on their way.
template <int TH, typename F>
__device__ __forceinline__ int collect_entries(const uint32_t* rhs, const uint32_t* lhs, int n, long long x_batch, uint32_t e,
                                               int2* list, int* count, int unordered, F&& meanwhile) {
  // both indices of a thread's entries in flight at once: one latency, not one for each
  uint32_t r[4], l[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int at = threadIdx.x + q * TH;
    r[q] = at < n ? rhs[at] : ~e;
    l[q] = at < n ? lhs[at] : 0;
  }
  meanwhile();
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (r[q] == e && (long long)l[q] < x_batch) list[atomicAdd(count, 1)] = make_int2((int)l[q], (int)threadIdx.x + q * TH);
  __syncthreads();
  const int c = *count;
  if (c <= unordered) return c;
  int2 mine[4];
  int rank[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {  // the atomics leave any order: a place is the number of smaller entries
    const int at = threadIdx.x + q * TH;
    rank[q] = -1;
    if (at < c) {
      mine[q] = list[at];
      rank[q] = 0;
      for (int j = 0; j < c; j++) rank[q] += list[j].y < mine[q].y;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (rank[q] >= 0) list[rank[q]] = mine[q];
  __syncthreads();
  return c;
}

}  // namespace kq
