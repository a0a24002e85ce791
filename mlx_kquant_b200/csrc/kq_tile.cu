// Tile kernel for more than 16 activation rows: y[M, N] = x[M, K] . dequant(W)^T on the 5th-generation tensor cores,
// with the WEIGHTS as the A operand. Reference: the dequantize-then-GEMM CPU path
// (src/kquant_cpu_decode.cpp:1299-1352), the Metal tile kernels (src/kquant_matmul.cpp:313-527).
//
// A tile is 128 weight rows per CTA (256 per CTA pair, tcgen05 cta_group::2) x up to 256 activation rows ("tokens",
// the N dimension of the instruction, any multiple of 16: a ragged last tile pays for the tokens it has).
//   * q4_k / q6_k: producer threads own a weight row (a TMEM lane) each and write its dequantized fp16 values straight
//     into tensor memory (tcgen05.st), from where tcgen05.mma takes its A operand: the weights pass neither through a
//     swizzled shared-memory tile nor through the async-proxy fence, and shared memory only feeds the activations.
//     Wire blocks come through a ring of TMA boxes, one superblock of the tile's rows each.
//   * fp16 weights (the copy path of kq_gemm.cu): both operands by TMA, no producers.
//   * A CTA pair halves the activation bytes that each SM loads and keeps; single CTAs serve few rows or small matrices.
//   * One barrier per stage (128 of K; 64 on the copy path) counts the producer warps and the activation bytes of both
//     CTAs; one commit frees the stage in both. CTAs are persistent, and the epilogue has warps of its own: it works beside
//     the next tile's stages, with two accumulators where tensor memory has room for them (up to 128 tokens; 160 for a pair).
//   * Few tiles: K is split over a cluster, partial tiles meet through distributed shared memory.
//   * Warps that issue tensor or TMA instructions stay converged and predicate them: from a lane-0 branch an MMA costs 60
//     cycles of issue and a commit 240 (operands moved to uniform registers one by one), predicated 10 and 200.
// What bounds it. Up to ~100 tokens the producers: 370 cycles for 128 x 64 weights ([28672, 8192] q4_k x 61: 64 us against
// 106 with the tile kernel before, whose producers went through shared memory), instruction issue 60 % busy. From 200 tokens
// on the tensor pipe: 1010-1030 cycles a stage of 256 tokens where the pipe needs 1024; then the power limit ([14336, 4096] x
// 8192: 1.4 GHz, 690 us against 802; fp16 weights 650 = 1480 TFLOP/s, cuBLAS 646). In between, waves: [14336, 4096] x 509 has
// 112 tiles for 74 pairs (62 us, before 65).
// Both operands are fp16 (see kq_gemm.cu, which also holds the pre-pass that makes the fp16 rows).
// Every wait is bounded: on expiry the CTA raises a flag in the device error word and leaves.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_launch.h"
#include "kq_tcgen05.cuh"
#include "kq_tma_map.h"

namespace cg = cooperative_groups;

namespace kq {

namespace {

enum TileSource { kSrcQ4K = 0, kSrcQ6K = 1, kSrcHalf = 2 };

constexpr int kMaxStages = 8, kMaxRaw = 6, kMaxTokens = 256;
constexpr int kMaxDynSmem = 227 * 1024 - 2048;  // beside the static part
constexpr int kStep = 64;               // weights of a K-step: one 128-byte swizzle row of fp16
constexpr int kWTileBytes = 128 * 128;  // fp16 weight tile of a CTA and K-step (copy path)
// bytes of a row in the raw ring: the q4_k superblock; for q6_k the 16-byte aligned window around it
__host__ __device__ constexpr int raw_row_bytes(int src) { return src == kSrcQ4K ? 144 : (src == kSrcQ6K ? 240 : 0); }
// warps 0-3 epilogue (TMEM lane quarter = warp), 4 MMA, 5 activation loader, 6 wire-byte loader, 8.. producers
__host__ __device__ constexpr int tile_threads(int src) { return src == kSrcHalf ? 192 : 768; }
// K-steps of a stage. A commit costs the issuing warp 200 cycles, as long as three K-steps of 32 tokens or one of 100.
__host__ __device__ constexpr int stage_steps(int src) { return src == kSrcHalf ? 1 : 2; }

struct TilePlan {
  void* y;
  long long y_row_stride;
  const float* row_scale;     // factor per activation row, or nullptr
  const int* yrow;            // output row of each activation row, or nullptr
  const GemmTile* tiles;      // grouped mode: device-built row tiles; nullptr = dense
  const int* n_tiles_dev;
  int M, N, K;
  int tn;                     // tokens of a full tile
  int nblk, tblk, raster;     // weight-row blocks, token blocks, weight-row blocks that are walked together
  int stages, raw_stages, n_acc, acc_cols, tmem_cols;
  int lg;                     // wire rows are whole multiples of 16 bytes in groups of 1 << lg (q4_k: 0)
  int row_bytes;
  int after_prepass;          // the launch before is the pre-pass of this call: its results are waited for here
  int stage_bytes, raw_off, stg_off, stg_tokens;
  int* error_word;
};

// ------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// (predicated like the tensor instructions below: what follows is often an instruction of the whole warp)
__device__ __forceinline__ void arrive_cluster(uint32_t e, uint32_t addr) {
  asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q mbarrier.arrive.shared::cluster.b64 _, [%0];\n}\n" ::"r"(addr),
               "r"(e)
               : "memory");
}
__device__ __forceinline__ void arrive_local(uint32_t e, uint64_t* bar) {
  asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q mbarrier.arrive.shared::cta.b64 _, [%0];\n}\n" ::"r"(smem_u32(bar)),
               "r"(e)
               : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
  return p;
}
// try_wait with a limit (ns) for which the hardware may keep the thread suspended: a waiting warp that polls takes issue
// slots from the producers.
__device__ __forceinline__ bool try_wait_ns(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(1000000u)
      : "memory");
  return ok != 0;
}
// Bounded wait of a whole warp (see mbar_wait_err). Every exit is by a vote, so that what follows is known to run
// converged: instructions that take uniform registers (tcgen05.mma, commit, TMA) otherwise pay for moving each operand
// there, 60 cycles an MMA and 240 a commit instead of 10 and 200.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code, int* error_word) {
  if (__all_sync(0xffffffffu, try_wait_ns(bar, parity))) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (int spin = 0;; spin++) {
    if (__all_sync(0xffffffffu, try_wait_ns(bar, parity))) return true;
    if ((spin & 15) == 15) {
      const bool late = globaltimer_ns() - t0 > 2000000000ull;
      if (late) *abort_flag = 1, atomicOr(error_word, code);
      if (__any_sync(0xffffffffu, late || *abort_flag != 0)) return false;
    }
  }
}
template <int CG>
__device__ __forceinline__ void tmem_alloc_g(uint32_t* dst, uint32_t ncols) {
  if constexpr (CG == 1) {
    tmem_alloc(dst, ncols);
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc_g(uint32_t taddr, uint32_t ncols) {
  if constexpr (CG == 1) tmem_dealloc(taddr, ncols);
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
// The MMAs and commits are predicated instead of branched around (e: non-zero in the one lane that issues): the warp
// stays converged, so that descriptors and addresses are made in uniform registers.
template <int CG>
__device__ __forceinline__ void umma_ts(uint32_t e, uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(e)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(e)
        : "memory");
}
template <int CG>
__device__ __forceinline__ void umma_ss(uint32_t e, uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(e)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
        " @q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(e)
        : "memory");
}
// arrives on the barrier at this offset in every CTA of the pair (mask) once the MMAs issued so far have completed
template <int CG>
__device__ __forceinline__ void umma_commit_g(uint32_t e, uint64_t* bar, uint16_t mask) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(bar)),
        "r"(e)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n"
        " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n" ::"r"(
            smem_u32(bar)),
        "h"(mask), "r"(e)
        : "memory");
}
// Box into this CTA's shared memory, bytes counted on `bar` (pair: the barrier of the pair's first CTA). No multicast.
template <int CG>
__device__ __forceinline__ void load_2d(uint32_t e, uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  if constexpr (CG == 1)
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
        " @q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}\n" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "r"(e)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
        " @q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];\n}\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "r"(e)
        : "memory");
}
__device__ __forceinline__ void load_3d(uint32_t e, uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %6, 0;\n"
      " @q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n}\n" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)), "r"(e)
      : "memory");
}
__device__ __forceinline__ void expect_tx(uint32_t e, uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n" ::"r"(
          smem_u32(bar)),
      "r"(bytes), "r"(e)
      : "memory");
}
// 16 lanes x 16 columns of tensor memory: thread t holds lanes t / 4 (r[0], r[1], r[4], r[5]) and 8 + t / 4, columns
// 2 (t % 4) and the one after it of the first eight (r[0] .. r[3]) and of the second
__device__ __forceinline__ void tmem_ld_16x16(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// four 8 x 8 matrices of 16-bit values, transposed: thread i gives the address of row i % 8 of matrix i / 8
__device__ __forceinline__ void store_trans(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3])
               : "memory");
}

// ------------------------------------------------------------------ producers: half a superblock of a row
// A producer thread makes 128 weights of its row at a time, 64 TMEM columns in two pieces of 32 registers: what a
// piece of work costs besides the weights (waits, arrivals, the block's header) was half of the instructions with 64.
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }

// q4_k, sub-blocks 4 half .. 4 half + 3 (src/kquant_cpu_decode.cpp:177-202). A weight is fma(sc * q, d, -fp16(dmin * mn)):
// sc * q is an exact integer in fp16, so there is one rounding besides the min's. Nibbles become fp16 by one permute per
// two weights: low ones as 1024 + q, high ones, left in place, as 64 + q.
template <int UNIT>
struct Q4kHalf {
  uint4 hdr, q[2 * UNIT];
  uint32_t sc, mn;  // the four scales and mins, a byte each
  __device__ __forceinline__ void load(const uint8_t* blk, int, int half, int piece) {
    const uint4* b = reinterpret_cast<const uint4*>(blk);
    hdr = b[0];
#pragma unroll
    for (int i = 0; i < 2 * UNIT; i++) q[i] = b[1 + 4 * half + (UNIT == 1 ? 2 * piece : 0) + i];
  }
  __device__ __forceinline__ void header(int half) {
    if (half == 0) {
      sc = hdr.y & 0x3f3f3f3fu;
      mn = hdr.z & 0x3f3f3f3fu;
    } else {
      sc = (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u);
      mn = ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u);
    }
  }
  template <int P>  // the first or the second two sub-blocks
  __device__ __forceinline__ void make(uint32_t (&o)[32]) const {
    const __half2 d2 = as_h2(__byte_perm(hdr.x, 0u, 0x1010)), dmin2 = as_h2(__byte_perm(hdr.x, 0u, 0x3232));
    const uint4 q0 = q[UNIT == 2 ? 2 * P : 0], q1 = q[UNIT == 2 ? 2 * P + 1 : 1];
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const __half2 k1024 = __float2half2_rn(1024.f);
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
      const uint32_t pick = 0x4040u + 0x0101u * (2 * P + hh);
      const __half2 s = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, pick)), k1024);
      const __half2 m = __hsub2(as_h2(__byte_perm(mn, 0x64646464u, pick)), k1024);
      const __half2 off = __hmul2(s, __float2half2_rn(hh ? -64.f : -1024.f));
      const __half2 ndm = __hneg2(__hmul2(dmin2, m));
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t n4 = w[i] & (hh ? 0xf0f0f0f0u : 0x0f0f0f0fu);
        const uint32_t magic = hh ? 0x54545454u : 0x64646464u;
        o[16 * hh + 2 * i] = as_u32(__hfma2(__hfma2(as_h2(__byte_perm(n4, magic, 0x4140)), s, off), d2, ndm));
        o[16 * hh + 2 * i + 1] = as_u32(__hfma2(__hfma2(as_h2(__byte_perm(n4, magic, 0x4342)), s, off), d2, ndm));
      }
    }
  }
};

// q6_k (src/kquant_cpu_decode.cpp:238-280): a half is four quarters of 32 weights; the low nibbles of its 64 ql bytes are
// quarters 0 and 1, the high ones 2 and 3, bits 2 j of its 32 qh bytes belong to quarter j. A weight is
// (q - 32) * (d * scale), the scale in two fp16 parts, so that the product is rounded once but for the last bit of a small
// correction, as dequantization to fp16 is (a scale in one part: errors a third larger; 4-8 % faster). The block starts `phase` bytes (even, the same for all rows) into a 16-byte aligned window.
template <int UNIT>
struct Q6kHalf {
  uint32_t ql[16], qh[8], sc[2];
  float d;
  template <int W>
  __device__ __forceinline__ void load_at(const uint8_t* win, uint32_t odd_bits, int half) {
    window_words<W, 16>(win + 64 * half, odd_bits, ql);
    window_words<W, 8>(win + 128 + 32 * half, odd_bits, qh);
    const uint32_t* s = reinterpret_cast<const uint32_t*>(win + 192 + 8 * half + 4 * W);
    const uint32_t s0 = s[0], s1 = s[1], s2 = s[2];
    sc[0] = __funnelshift_r(s0, s1, odd_bits), sc[1] = __funnelshift_r(s1, s2, odd_bits);
  }
  __device__ __forceinline__ void load(const uint8_t* win, int phase, int half, int) {
    const uint32_t odd_bits = 8u * (phase & 2);
    d = __half2float(*reinterpret_cast<const __half*>(win + phase + 208));
    switch (phase >> 2) {
      case 0: load_at<0>(win, odd_bits, half); break;
      case 1: load_at<1>(win, odd_bits, half); break;
      case 2: load_at<2>(win, odd_bits, half); break;
      default: load_at<3>(win, odd_bits, half); break;
    }
  }
  __device__ __forceinline__ void header(int) {}
  // v = hi + lo; a scale that overflows stays an infinity
  static __device__ __forceinline__ void two(float v, __half2& hi, __half2& lo) {
    hi = __float2half2_rn(v);
    const float rest = v - __low2float(hi);
    lo = __float2half2_rn(fabsf(rest) < 65504.f ? rest : 0.f);
  }
  template <int P>
  __device__ __forceinline__ void make(uint32_t (&o)[32]) const {
    const __half2 k1056 = __float2half2_rn(1056.f);
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
      __half2 sA, sB, tA, tB;
      two(d * (float)(int)(int8_t)((sc[P] >> (16 * hh)) & 0xffu), sA, tA);
      two(d * (float)(int)(int8_t)((sc[P] >> (16 * hh + 8)) & 0xffu), sB, tB);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t hb = P == 0 ? (hh == 0 ? qh[i] << 4 : qh[i] << 2) : (hh == 0 ? qh[i] : qh[i] >> 2);
        const uint32_t l = ql[8 * hh + i];
        const uint32_t q4 = ((P ? l >> 4 : l) & 0x0f0f0f0fu) | (hb & 0x30303030u);
        const __half2 s = i < 4 ? sA : sB, t = i < 4 ? tA : tB;
        const __half2 q0 = __hsub2(as_h2(__byte_perm(q4, 0x64646464u, 0x4140)), k1056);
        const __half2 q1 = __hsub2(as_h2(__byte_perm(q4, 0x64646464u, 0x4342)), k1056);
        o[16 * hh + 2 * i] = as_u32(__hfma2(q0, s, __hmul2(q0, t)));
        o[16 * hh + 2 * i + 1] = as_u32(__hfma2(q1, s, __hmul2(q1, t)));
      }
    }
  }
};

// ------------------------------------------------------------------ the kernel
// CG: CTAs that share a tile (cta_group). gridDim.z > 1: that many slices of K, one tile per cluster.
template <int SRC, typename OT, int CG, int UNIT>
__global__ void __launch_bounds__(tile_threads(SRC), 1)
tile_kernel(const TilePlan a, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w) {
  constexpr bool kFused = SRC != kSrcHalf;
  constexpr int KS = stage_steps(SRC);
  constexpr int kRawRow = raw_row_bytes(SRC), kRawSlot = 128 * kRawRow;
  constexpr bool kHalfOut = std::is_same<OT, __half>::value;
  extern __shared__ __align__(1024) uint8_t tile_smem[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tile_smem) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[kMaxStages], empty[kMaxStages], raw_full[kMaxRaw], raw_empty[kMaxRaw], acc_full[2], acc_empty[2];
  __shared__ __align__(16) float s_scale[kMaxTokens];
  __shared__ uint32_t tmem_s;
  __shared__ int abort_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool clustered = CG == 2 || gridDim.z > 1;
  const uint32_t crank = __shfl_sync(0xffffffffu, clustered ? cluster_rank() : 0u, 0);
  const uint32_t rank = CG == 2 ? (crank & 1u) : 0u, leader = crank - rank;  // place in the pair; the pair's first CTA
  const int S = a.stages, R = a.raw_stages;

  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 1 + (kFused ? 8 / UNIT * CG : 0));
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < R; s++) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], 16 / UNIT);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4 * CG);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 4) tmem_alloc_g<CG>(&tmem_s, a.tmem_cols);
  tc_fence_before();
  __syncthreads();
  if (clustered) cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_s, 0);
  volatile int* abort_flag = &abort_s;
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
    return wait_warp(bar, parity, abort_flag, code, a.error_word);
  };
  const uint32_t full_at = map_rank(smem_u32(full), leader), acc_empty_at = map_rank(smem_u32(acc_empty), leader);
  const uint16_t pair_mask = (uint16_t)(3u << leader);

  // stages of K of this CTA: a slice of all of them
  const int steps = (a.K + KS * kStep - 1) / (KS * kStep) / (int)gridDim.z, kb0 = (int)blockIdx.z * steps;
  const uint32_t x_tile = (uint32_t)(a.tn / CG * 128);  // bytes of a K-step's activations in this CTA
  const int total = __shfl_sync(0xffffffffu, a.nblk * (a.tiles != nullptr ? *a.n_tiles_dev : a.tblk), 0);
  const int first = (int)blockIdx.x / CG, stride = (int)gridDim.x / CG;  // first >= total: nothing to do
  struct Tile {
    int n0, m0, rows, expert, cols;  // first weight row (of the pair), first activation row, live ones, expert, MMA columns
  };
  auto tile_at = [&](int t) {
    Tile r;
    int nb;
    t = max(0, min(t, total - 1));
    if (a.tiles != nullptr) {
      nb = t % a.nblk;
      const GemmTile g = a.tiles[t / a.nblk];
      r.m0 = g.row_start, r.rows = g.rows, r.expert = g.expert;
    } else {
      const int per = a.raster * a.tblk, grp = t / per, rem = t - grp * per;
      const int wide = min(a.raster, a.nblk - grp * a.raster);
      nb = grp * a.raster + rem % wide;
      r.m0 = rem / wide * a.tn, r.rows = min(a.tn, a.M - r.m0), r.expert = 0;
    }
    r.n0 = nb * 128 * CG;
    r.cols = max(16, (r.rows + 15) & ~15);
    return r;
  };

  if (warp < 4) {
    // ================= epilogue =================
    bool ok = true;
    int done = 0;
    Tile next = tile_at(first);
    if (a.after_prepass) asm volatile("griddepcontrol.wait;\n" ::: "memory");  // row_scale, yrow
    for (int t = first; t < total && ok; t += stride, done++) {
      const Tile tl = next;
      if (t + stride < total) next = tile_at(t + stride);  // (fetched a tile ahead: grouped tiles come from memory)
      const int as = done % a.n_acc;
      for (int i = threadIdx.x; i < tl.cols; i += 128)
        s_scale[i] = a.row_scale != nullptr && i < tl.rows ? a.row_scale[tl.m0 + i] : 1.f;
      asm volatile("bar.sync 2, 128;\n" ::: "memory");
      ok = wait(&acc_full[as], (done / a.n_acc) & 1, 4);
      // all four warps go on together or not at all: the passes below meet at barriers
      {
        int all;
        asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n barrier.cta.red.and.pred q, 2, 128, p;\n selp.s32 %0, 1, 0, q;\n}\n"
                     : "=r"(all)
                     : "r"((int)ok)
                     : "memory");
        ok = all != 0;
      }
      if (!ok) break;
      tc_fence_after();
      const uint32_t acc = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(as * a.acc_cols);
      if (gridDim.z > 1) {
        // weight row of this thread's TMEM lane: classes of rows modulo 1 << lg one after the other
        const int at = 32 * warp + lane, n_row = ((at & ((128 >> a.lg) - 1)) << a.lg) | (at >> (7 - a.lg));
        float* part = reinterpret_cast<float*>(ring);  // [token][128] (the rings are idle: every MMA has completed)
        for (int c0 = 0; c0 < tl.cols; c0 += 16) {
          uint32_t v[16];
          tmem_ld16(acc + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; i++) part[(c0 + i) * 128 + n_row] = __uint_as_float(v[i]) * s_scale[c0 + i];
        }
        break;
      }
      for (int cb = 0; cb < tl.cols; cb += a.stg_tokens) {
        // Rows of the accumulator are columns of y: the fragments are stored transposed, [token][128], the sixteen 16-byte
        // pieces of a row XOR-swizzled by the token. The next columns are on their way while these are rounded. (A thread
        // per weight row with a two-byte store per token took 27 cycles a column, 7000 a tile; now 8.)
        const int ce = min(tl.cols, cb + a.stg_tokens);
        const int tok = lane & 7, piece = 4 * warp + (lane >> 3);
        const uint32_t stg = smem_u32(ring) + a.stg_off + tok * 256 + ((piece ^ tok) << 4);
        uint32_t r0[2][8], r1[2][8];
        auto fetch = [&](uint32_t (&r)[2][8], int c) {
          tmem_ld_16x16(acc + c, r[0]);
          tmem_ld_16x16(acc + (16u << 16) + c, r[1]);
        };
        auto put = [&](const uint32_t (&r)[2][8], int c) {
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const float2 f = *reinterpret_cast<const float2*>(&s_scale[c + 8 * j + 2 * (lane & 3)]);
            uint32_t v[4];
#pragma unroll
            for (int h = 0; h < 4; h++) {
              const float lo = __uint_as_float(r[h >> 1][4 * j + 2 * (h & 1)]) * f.x;
              const float hi = __uint_as_float(r[h >> 1][4 * j + 2 * (h & 1) + 1]) * f.y;
              if constexpr (kHalfOut) {
                const __half2 o = __floats2half2_rn(lo, hi);
                v[h] = *reinterpret_cast<const uint32_t*>(&o);
              } else {
                const __nv_bfloat162 o = __floats2bfloat162_rn(lo, hi);
                v[h] = *reinterpret_cast<const uint32_t*>(&o);
              }
            }
            store_trans(stg + (c + 8 * j - cb) * 256, v);
          }
        };
        fetch(r0, cb);
        for (int c0 = cb; c0 < ce; c0 += 32) {
          tmem_ld_wait();
          if (c0 + 16 < ce) fetch(r1, c0 + 16);
          put(r0, c0);
          if (c0 + 16 < ce) {
            tmem_ld_wait();
            if (c0 + 32 < ce) fetch(r0, c0 + 32);
            put(r1, c0 + 16);
          }
        }
        if (ce == tl.cols) {  // the accumulator has been read
          tc_fence_before();
          __syncwarp();
          arrive_cluster(lane == 0, acc_empty_at + 8 * as);
        }
        asm volatile("bar.sync 2, 128;\n" ::: "memory");
        // whole rows of 128 outputs, sixteen bytes a lane, two rows a warp and pass; the output rows of grouped tiles
        // come from a table: lane i fetches those of pass i up front
        const int live = min(tl.rows, ce) - cb;
        const int sub = lane >> 4, chunk = lane & 15;
        const int col = tl.n0 + 128 * (int)rank + 8 * chunk;
        const int n_end = a.N;
        long long mine0 = 0, mine1 = 0;
        {
          const int r0 = 2 * warp + 8 * lane, m = tl.m0 + cb + r0;
          if (r0 < live) mine0 = a.yrow ? (long long)a.yrow[m] : (long long)m;
          if (r0 + 1 < live) mine1 = a.yrow ? (long long)a.yrow[m + 1] : (long long)(m + 1);
        }
        const int passes = (live + 7) / 8;
        for (int i = 0; i < passes; i++) {
          const long long o0 = __shfl_sync(0xffffffffu, mine0, i), o1 = __shfl_sync(0xffffffffu, mine1, i);
          const int r = 2 * warp + sub + 8 * i;
          if (r >= live) continue;
          const uint8_t* row = ring + a.stg_off + r * 256;
          uint4 q;
          if (SRC != kSrcQ6K || a.lg == 0) {
            q = *reinterpret_cast<const uint4*>(row + ((chunk ^ (r & 7)) << 4));
          } else {  // rows of one class lie together: eight neighbouring rows are in as many places
            uint32_t* qw = &q.x;
#pragma unroll
            for (int e = 0; e < 8; e++) {
              const int n = 8 * chunk + e, at = (n >> a.lg) | ((n & ((1 << a.lg) - 1)) << (7 - a.lg));
              const uint32_t v = *reinterpret_cast<const unsigned short*>(row + (((at >> 3) ^ (r & 7)) << 4) + 2 * (at & 7));
              qw[e >> 1] = (e & 1) ? qw[e >> 1] | (v << 16) : v;
            }
          }
          OT* yp = static_cast<OT*>(a.y) + (sub ? o1 : o0) * a.y_row_stride + col;
          if (col + 8 <= n_end && (reinterpret_cast<uintptr_t>(yp) & 15) == 0) {
            *reinterpret_cast<uint4*>(yp) = q;
          } else {
            const OT* qe = reinterpret_cast<const OT*>(&q);
#pragma unroll
            for (int e = 0; e < 8; e++)
              if (col + e < n_end) yp[e] = qe[e];
          }
        }
        asm volatile("bar.sync 2, 128;\n" ::: "memory");
      }
    }
  } else if (warp == 4) {
    // ================= MMA issuer: the pair's first CTA =================
    if (rank == 0) {
      bool ok = true;
      int done = 0, s = 0;
      uint32_t ph = 0;
      const uint32_t issuer = elect_one();
      const uint32_t a_col = tmem + (uint32_t)(a.n_acc * a.acc_cols);
      Tile next = tile_at(first);
      for (int t = first; t < total && ok; t += stride, done++) {
        const Tile tl = next;
        if (t + stride < total) next = tile_at(t + stride);
        const int as = done % a.n_acc;
        if (done >= a.n_acc) ok = wait(&acc_empty[as], ((done / a.n_acc) & 1) ^ 1, 8);
        if (!ok) break;
        tc_fence_after();
        const uint32_t acc = tmem + (uint32_t)(as * a.acc_cols);
        const uint32_t idesc = (1u << 4) | ((uint32_t)(__shfl_sync(0xffffffffu, tl.cols, 0) >> 3) << 17) | ((uint32_t)(8 * CG) << 24);
        for (int kb = 0; kb < steps; kb++) {
          ok = wait(&full[s], ph, 2);
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = smem_u32(ring) + s * a.stage_bytes;
          if constexpr (kFused) {
#pragma unroll
            for (int j = 0; j < KS * kStep / 16; j++)
              umma_ts<CG>(issuer, acc, a_col + 32 * KS * s + 8 * j, umma_desc_sw128(st + (j >> 2) * x_tile) + 2 * (j & 3), idesc,
                          (kb > 0 || j > 0) ? 1u : 0u);
          } else {
#pragma unroll
            for (int j = 0; j < KS * kStep / 16; j++)
              umma_ss<CG>(issuer, acc, umma_desc_sw128(st + (j >> 2) * kWTileBytes) + 2 * (j & 3),
                          umma_desc_sw128(st + KS * kWTileBytes + (j >> 2) * x_tile) + 2 * (j & 3), idesc,
                          (kb > 0 || j > 0) ? 1u : 0u);
          }
          umma_commit_g<CG>(issuer, &empty[s], pair_mask);
          if (++s == S) s = 0, ph ^= 1;
        }
        if (ok) umma_commit_g<CG>(issuer, &acc_full[as], pair_mask);
      }
    }
  } else if (warp == 5) {
    // ================= loader: activations (and fp16 weights) of a K-step =================
    const uint32_t e = elect_one(), e0 = rank == 0 ? e : 0u;
    bool ok = true;
    int s = 0, it = 0;
    uint32_t ph = 1;
    const uint32_t bytes = KS * CG * (x_tile + (kFused ? 0 : kWTileBytes));
    if (a.after_prepass) asm volatile("griddepcontrol.wait;\n" ::: "memory");  // fp16 rows, or fp16 weights
    Tile next = tile_at(first);
    for (int t = first; t < total && ok; t += stride) {
      const Tile tl = next;
      if (t + stride < total) next = tile_at(t + stride);
      const int m = __shfl_sync(0xffffffffu, tl.m0 + (int)rank * (tl.cols / CG), 0);
      for (int kb = 0; kb < steps; kb++, it++) {
        if (it >= S) ok = wait(&empty[s], ph, 1);
        if (!ok) break;
        expect_tx(e0, &full[s], bytes);
        uint32_t dst = smem_u32(ring) + s * a.stage_bytes;
        if constexpr (!kFused) {
#pragma unroll
          for (int j = 0; j < KS; j++)
            load_2d<CG>(e, dst + j * kWTileBytes, &map_w, ((kb0 + kb) * KS + j) * kStep, tl.n0 + 128 * (int)rank, full_at + 8 * s);
          dst += KS * kWTileBytes;
        }
#pragma unroll
        for (int j = 0; j < KS; j++)
          load_2d<CG>(e, dst + j * x_tile, &map_x, ((kb0 + kb) * KS + j) * kStep, m, full_at + 8 * s);
        if (++s == S) s = 0, ph ^= 1;
      }
    }
  } else if (warp == 6) {
    // ================= loader: wire bytes, one superblock of the CTA's 128 rows at a time =================
    if constexpr (kFused) {
      const uint32_t e = elect_one();
      bool ok = true;
      int r = 0, it = 0;
      uint32_t ph = 1;
      constexpr int kBlk = SRC == kSrcQ4K ? 144 : 210;
      Tile next = tile_at(first);
      for (int t = first; t < total && ok; t += stride) {
        const Tile tl = next;
        if (t + stride < total) next = tile_at(t + stride);
        for (int sb = 0; sb < steps / 2; sb++, it++) {
          if (it >= R) ok = wait(&raw_empty[r], ph, 16);
          if (!ok) break;
          expect_tx(e, &raw_full[r], kRawSlot);
          const uint32_t dst = smem_u32(ring) + a.raw_off + r * kRawSlot;
          const int x0 = (kb0 / 2 + sb) * kBlk, row0 = (tl.n0 + 128 * (int)rank) >> a.lg;
          if (SRC == kSrcQ4K || a.lg == 0) {
            load_3d(e, dst, &map_w, x0 & ~15, row0, tl.expert, &raw_full[r]);
          } else {  // a box per class
            for (int j = 0; j < 1 << a.lg; j++)
              load_3d(e, dst + j * (kRawSlot >> a.lg), &map_w, (x0 + j * a.row_bytes) & ~15, row0, tl.expert, &raw_full[r]);
          }
          if (++r == R) r = 0, ph ^= 1;
        }
      }
    }
  } else if (warp >= 8) {
    // ================= producers =================
    if constexpr (kFused) {
      // UNIT 2: warpgroup g makes the stages g, g + 4, ..., i.e. half g & 1 of every second superblock;
      // UNIT 1: half a stage at a time, quarter g of every superblock
      const int g = (warp - 8) >> 2, q = warp & 3;
      const int half = UNIT == 2 ? g & 1 : g >> 1, j0 = UNIT == 2 ? g : g >> 1, sb0 = UNIT == 2 ? g >> 1 : 0;
      bool ok = true;
      const uint8_t* rows = ring + a.raw_off + (32 * q + lane) * kRawRow;
      const uint32_t a_col = tmem + (uint32_t)(a.n_acc * a.acc_cols) + ((uint32_t)(32 * q) << 16);
      const int n = first < total ? ((total - 1 - first) / stride + 1) * steps : 0, per_tile = steps / 2;
      const int row_class = (32 * q + lane) >> (7 - a.lg);
      int r = sb0, s = j0, sb = sb0 % per_tile;
      uint32_t rph = 0, ph = 1;
      typename std::conditional<SRC == kSrcQ4K, Q4kHalf<UNIT>, Q6kHalf<UNIT>>::type raw;
      auto fetch = [&]() {
        ok = wait(&raw_full[r], rph, 32);
        raw.load(rows + r * kRawSlot, ((kb0 / 2 + sb) * 210 + (SRC == kSrcQ6K ? row_class * a.row_bytes : 0)) & 15, half, g & 1);
        if constexpr (SRC == kSrcQ6K) __syncwarp();  // rows of eight classes: two phases in a warp
      };
      if (j0 < n) fetch();
      for (int j = j0; j < n && ok; j += 2 * UNIT) {
        uint32_t o[32];
        raw.header(half);
        if (UNIT == 2 || (g & 1) == 0) raw.template make<0>(o);
        else raw.template make<1>(o);
        if (j >= S) ok = wait(&empty[s], ph, 64);
        if (!ok) break;
        tc_fence_after();
        tmem_st32(a_col + 64 * s + (UNIT == 2 ? 0 : 32 * (g & 1)), o);
        if constexpr (UNIT == 2) {
          raw.template make<1>(o);
          tmem_st32(a_col + 64 * s + 32, o);
        }
        __syncwarp();
        arrive_local(lane == 0, &raw_empty[r]);
        if ((r += UNIT) >= R) r -= R, rph ^= 1;
        for (sb += UNIT; sb >= per_tile;) sb -= per_tile;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        arrive_cluster(lane == 0, full_at + 8 * s);
        if ((s += 2 * UNIT) >= S) s -= S, ph ^= 1;
        if (j + 2 * UNIT < n) fetch();
      }
    }
  }

  if (abort_s != 0) {  // given up: what is in flight (copies, MMAs) lands long before this
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) {
    }
  }
  // ================= split K: the slices of a cluster meet through distributed shared memory =================
  if (gridDim.z > 1) {
    __syncwarp();
    cluster_sync_all();  // every slice's partial tile is in its shared memory
    const Tile tl = tile_at(first);
    const int Z = (int)gridDim.z, z = (int)blockIdx.z;
    cg::cluster_group cluster = cg::this_cluster();
    const int n = tl.n0 + 128 * (int)rank + 4 * lane;
    for (int c = z + Z * warp; c < tl.rows; c += Z * (int)(blockDim.x / 32)) {
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = 0; k < Z; k++) {
        const float* part = cluster.map_shared_rank(reinterpret_cast<float*>(ring), rank + CG * k);
        const float4 v = *reinterpret_cast<const float4*>(part + c * 128 + 4 * lane);
        sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
      }
      OT* yp = static_cast<OT*>(a.y) + (long long)(tl.m0 + c) * a.y_row_stride + n;
      const float f[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (n + i < a.N) {
          if constexpr (kHalfOut) yp[i] = __float2half_rn(f[i]);
          else yp[i] = __float2bfloat16_rn(f[i]);
        }
      }
    }
  }
  // ================= teardown =================
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (clustered) cluster_sync_all();  // the other CTA's barriers, operands and partial tiles are done with
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc_g<CG>(tmem, a.tmem_cols);
  }
}

// ------------------------------------------------------------------ host
// fp16 matrix [rows, K], row stride in elements: boxes of 64 x box_rows, 128B swizzle
bool half_map(CUtensorMap* map, const void* p, long long row_stride, long long rows, int K, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kStep, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(p), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// wire bytes [experts, N, row_bytes], 1 << lg rows taken as one: boxes of the 128 rows' (or those of a class of them)
// superblock or the aligned window around it
bool wire_map(CUtensorMap* map, const uint8_t* w, long long row_bytes, int lg, int N, int n_experts,
              long long expert_stride, int box_bytes) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)row_bytes << lg, (cuuint64_t)(N >> lg), (cuuint64_t)n_experts};
  const cuuint64_t strides[2] = {(cuuint64_t)row_bytes << lg, (cuuint64_t)(n_experts > 1 ? expert_stride : row_bytes * N)};
  const cuuint32_t box[3] = {(cuuint32_t)box_bytes, 128u >> lg, 1u};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(w), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Ring depths within shared and tensor memory of a shape; false: does not fit.
bool plan_rings(TilePlan& p, int src, int cg, int unit, int tn, bool one_acc, size_t* dyn) {
  const int smem = kMaxDynSmem - 1024;  // less the alignment of the tiles
  const bool fused = src != kSrcHalf;
  const int ks = stage_steps(src), slot = 128 * raw_row_bytes(src);
  p.tn = tn;
  p.acc_cols = (tn + 31) & ~31;
  p.stage_bytes = ks * (tn / cg * 128 + (fused ? 0 : kWTileBytes));
  // UNIT 2: a producer group takes every fourth stage and every second superblock, and waits for the use before. It has
  // seen the one before that done if there are four stages or more and an even number of slots; otherwise it could be two
  // uses ahead, where the barrier's parity reads as if the stage were free.
  const int least = unit == 2 && fused ? 4 : 3;
  for (p.n_acc = one_acc ? 1 : 2; p.n_acc >= 1; p.n_acc--) {
    const int left = 512 - p.n_acc * p.acc_cols;
    const int most = std::min(kMaxStages, fused ? left / (32 * ks) : kMaxStages);
    if (left < 0 || most < least) continue;
    for (p.raw_stages = fused ? kMaxRaw : 0; p.raw_stages >= (fused ? 2 : 0); p.raw_stages -= unit) {
      // the epilogue's buffer: all tokens where there is one accumulator, which is then free again sooner
      p.stg_tokens = p.n_acc == 1 ? tn : std::min(tn, 128);
      p.stages = std::min(most, (smem - p.raw_stages * slot - p.stg_tokens * 256) / p.stage_bytes);
      if (p.stages < least || (p.raw_stages > 3 && p.stages < std::min(most, 4))) continue;
      p.raw_off = p.stages * p.stage_bytes;
      p.stg_off = p.raw_off + p.raw_stages * slot;
      *dyn = (size_t)p.stg_off + p.stg_tokens * 256 + 1024;
      const int need = p.n_acc * p.acc_cols + (fused ? 32 * ks * p.stages : 0);
      p.tmem_cols = 32;
      while (p.tmem_cols < need) p.tmem_cols *= 2;
      return true;
    }
  }
  return false;
}

struct TileCall {
  TilePlan p;
  const void* x;
  long long x_row_stride, x_rows;
  const uint8_t* w;
  long long row_bytes, expert_stride;
  int n_experts;
  int grid_units;  // persistent CTAs or pairs
  int ks;
};

template <int SRC, typename OT, int CG, int UNIT>
cudaError_t launch_tile_t(TileCall c, int tn, cudaStream_t st) {
  auto kern = tile_kernel<SRC, OT, CG, UNIT>;
  size_t dyn = 0;
  if (!plan_rings(c.p, SRC, CG, UNIT, tn, c.ks > 1, &dyn)) return cudaErrorInvalidConfiguration;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  if ((c.p.error_word = device_error_word()) == nullptr) return cudaErrorUnknown;
  alignas(64) CUtensorMap map_x, map_w;
  const bool maps = half_map(&map_x, c.x, c.x_row_stride, c.x_rows, c.p.K, tn / CG) &&
                    (SRC == kSrcHalf ? half_map(&map_w, c.w, c.p.K, c.p.N, c.p.K, 128)
                                     : wire_map(&map_w, c.w, c.row_bytes, c.p.lg, c.p.N, c.n_experts, c.expert_stride,
                                                raw_row_bytes(SRC)));
  if (!maps) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CG * c.grid_units, 1, c.ks);
  cfg.blockDim = dim3(tile_threads(SRC));
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = st;
  // Everything before the pre-pass has ended when this kernel may start (the pre-pass itself is launched plainly), so the
  // weights, tile lists and so on are read at once; only what the pre-pass writes is waited for.
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CG;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = c.ks;
  const int skip = c.p.after_prepass ? 0 : 1;
  cfg.attrs = attr + skip;
  cfg.numAttrs = (CG * c.ks > 1 ? 2 : 1) - skip;
  return cudaLaunchKernelEx(&cfg, kern, c.p, map_x, map_w);
}

// CTAs that reside at once in clusters of n = 1, 2, 4, 8 (148, 148, 132 and 120 on a B200: clusters of more than two
// leave SMs of the smaller GPCs idle).
int resident_ctas(int n) {
  static int known[16][9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 0;
  if (known[dev][n] == 0) {
    int got = 0;
    if (n == 1) {
      if (cudaDeviceGetAttribute(&got, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) got = 0;
    } else {
      auto kern = tile_kernel<kSrcQ4K, __half, 2, 2>;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(n, 1, 1);
      cfg.blockDim = dim3(tile_threads(kSrcQ4K));
      cfg.dynamicSmemBytes = kMaxDynSmem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = n;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&got, kern, &cfg) != cudaSuccess || got <= 0) {
        (void)cudaGetLastError();
        got = 120 / n;
      }
      got *= n;
    }
    known[dev][n] = got;
  }
  return known[dev][n];
}

// Cycles of a call with tiles of tn tokens on cg CTAs and K in ks slices. A stage costs its producers (`make`: 128 weights of
// 128 rows; the copy path's loads) or the tensor pipe (4 cycles a token and 128 of K, the same for a pair as for one CTA of
// half the rows), whichever is more; a tile its epilogue, most of it in the open where tensor memory holds one accumulator.
// Constants fitted to a sweep of shapes over 150 sizes (N, K of 1024 to 28672, 17 to 2048 rows; q4_k, q6_k and fp16):
// the shape taken is within 1-2 % of the best one on average, 25 % at worst. With K up to 1024 the q4_k producers' work is too short
// to hide an epilogue that shares the issue slots with it: 50 cycles a token whatever the shape (as 2500 + 8 to 26
// a token: q4_k x 1500 [28672, 512] 101 us, now 92, [14997, 768] 92 and 77, [19861, 768] 119 and 99).
double tile_cost(int src, int M, int N, int K, int cg, int tn, int ks, int cap) {
  const bool fused = src != kSrcHalf;
  const long long tiles = (long long)((N + 128 * cg - 1) / (128 * cg)) * ((M + tn - 1) / tn);
  const int units = cap / (cg * ks);
  const long long turns = (tiles + units - 1) / units;
  const double per_step = fused ? 2.0 : 1.0, steps = std::ceil(K / (kStep * per_step)) / ks;
  const double make = src == kSrcQ4K ? 750.0 : (src == kSrcQ6K ? 830.0 + tn : 200.0 + 1.3 * tn / cg);
  const bool open = turns == 1 || (fused && tn > (cg == 1 ? 128 : 160));
  const double drain = src == kSrcQ4K && K <= 1024 ? 50.0 * tn : 2500.0 + (open ? 26.0 : 8.0) * tn;
  const double tile = steps * std::max(make, 2.04 * per_step * tn) + drain;
  return turns * tile + 9000.0 + (ks > 1 ? 3500.0 + 12.0 * ks * tn : 0.0);
}

struct TileShape {
  int cg, tn, ks;
  double cycles;
};
TileShape pick_shape(int src, int M, int N, int K) {
  TileShape best{2, kMaxTokens, 1, 1e300};
  const int least = (M + kMaxTokens - 1) / kMaxTokens;
  for (int cg = 1; cg <= 2; cg++) {
    int last = 0;
    for (int blocks = least; blocks <= std::max(least + 7, std::min(8, (M + 63) / 64)); blocks++) {
      const int tn = ((M + blocks - 1) / blocks + 15) & ~15;
      // a CTA alone: rings of fewer stages and slots beyond this, always slower than a pair
      if (tn == last || (cg == 1 && src != kSrcHalf && tn > 112)) continue;
      if (tn < 64 && blocks > least) break;
      last = tn;
      const long long tiles = (long long)((N + 128 * cg - 1) / (128 * cg)) * ((M + tn - 1) / tn);
      for (int ks = 1; cg * ks <= 8; ks *= 2) {
        const int cap = resident_ctas(cg * ks);
        if (cap < cg * ks) continue;
        const int steps = src == kSrcHalf ? (K + kStep - 1) / kStep : K / 256;  // slices hold whole superblocks
        if (ks > 1 && (steps % ks != 0 || tiles * cg * ks > cap)) break;
        const double c = tile_cost(src, M, N, K, cg, tn, ks, cap);
        if (c < best.cycles) best = {cg, tn, ks, c};
      }
    }
  }
  return best;
}

template <int SRC, typename OT>
cudaError_t launch_tile_src(TileCall& c, int tile_rows, cudaStream_t st) {
  TilePlan& p = c.p;
  TileShape sh{2, tile_rows, 1, 0.0};  // grouped: the tile list is cut for this many rows
  const int max_tiles = p.tblk;
  if (p.tiles == nullptr) sh = pick_shape(SRC, p.M, p.N, p.K);
  // Weight-row blocks walked together: all of them where the wire bytes stay in L2 from one token block to the next
  // (their fp16 copy, four times the size: eight), else sixteen ([14336, 4096] fp16 x 8192: 626 us with eight, 720 with all)
  p.raster = SRC == kSrcHalf ? 8 : (c.row_bytes * p.N <= (64ll << 20) ? 1 << 20 : 16);
  p.nblk = (p.N + 128 * sh.cg - 1) / (128 * sh.cg);
  p.raster = std::min(p.raster, p.nblk);
  if (p.tiles == nullptr) p.tblk = (p.M + sh.tn - 1) / sh.tn;
  const long long total = (long long)p.nblk * (p.tiles != nullptr ? max_tiles : p.tblk);
  const int cap = resident_ctas(sh.cg);
  if (cap < sh.cg || total > 0x7fffffffll) return cudaErrorInvalidConfiguration;
  c.ks = sh.ks;
  c.grid_units = (int)(sh.ks > 1 ? total : std::min<long long>(total, cap / sh.cg));
  if constexpr (SRC != kSrcHalf)
    if (sh.cg == 2 && sh.tn > 128) return launch_tile_t<SRC, OT, 2, 1>(c, sh.tn, st);
  if (sh.cg == 2) return launch_tile_t<SRC, OT, 2, 2>(c, sh.tn, st);
  return launch_tile_t<SRC, OT, 1, 2>(c, sh.tn, st);
}

// rows of 16-byte alignment in groups of 1 << lg
int row_group(long long row_bytes) {
  int lg = 0;
  while (((row_bytes << lg) & 15) != 0) lg++;
  return lg;
}

}  // namespace

bool tile_supported(int codec, const uint8_t* w, long long row_bytes, int N, int K, long long expert_stride) {
  if ((codec != Q4_K && codec != Q6_K) || row_bytes != (long long)(K >> 8) * bpb_of(codec) || (K & 255) != 0) return false;
  return (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (expert_stride & 15) == 0 && (N & ((1 << row_group(row_bytes)) - 1)) == 0 &&
         row_bytes <= (1 << 24);
}

bool tile_rows_fit(int codec, int N, int K) {
  return (codec == Q4_K || codec == Q6_K) && (K & 255) == 0 && (N & ((1 << row_group((long long)(K >> 8) * bpb_of(codec))) - 1)) == 0;
}

double tile_cycles(int codec, bool half_weights, int M, int N, int K) {
  const TileShape sh = pick_shape(half_weights ? kSrcHalf : (codec == Q4_K ? kSrcQ4K : kSrcQ6K), M, N, K);
  // Rows that are no whole sixteens leave the accumulator in classes and are put right output by output, 60 cycles a token.
  // Where the choice between producers and copy left that out, q6_k [28672, 512] x 620 took 78 us with producers (copy 45.5),
  // [20000, 1024] x 620 69 (47), [8192, 3072] x 1500 88 (69). (In the choice of the shape it does not help: [8192, 3072] x 125
  // 20.7 -> 23.6.)
  double sorting = 0.0;
  if (!half_weights && sh.ks == 1 && row_group((long long)(K >> 8) * bpb_of(codec)) != 0) {
    const long long tiles = (long long)((N + 128 * sh.cg - 1) / (128 * sh.cg)) * ((M + sh.tn - 1) / sh.tn);
    const int units = std::max(1, resident_ctas(sh.cg) / sh.cg);
    sorting = 60.0 * sh.tn * (double)((tiles + units - 1) / units);
  }
  return sh.cycles + sorting;
}

cudaError_t launch_tile(int codec, bool half_weights, bool out_half, const TileArgs& t, cudaStream_t st) {
  TileCall c{};
  c.p.y = t.y;
  c.p.y_row_stride = t.y_row_stride;
  c.p.row_scale = t.row_scale;
  c.p.yrow = t.yrow;
  c.p.tiles = t.tiles;
  c.p.n_tiles_dev = t.n_tiles_dev;
  c.p.M = t.M;
  c.p.N = t.N;
  c.p.K = t.K;
  c.p.tblk = t.max_tiles;
  c.p.lg = half_weights ? 0 : row_group(t.row_bytes);
  c.p.row_bytes = (int)t.row_bytes;
  c.p.after_prepass = t.after_prepass;
  c.x = t.x;
  c.x_row_stride = t.x_row_stride;
  c.x_rows = t.M;
  c.w = t.w;
  c.row_bytes = t.row_bytes;
  c.expert_stride = t.expert_stride;
  c.n_experts = t.n_experts;
  const int rows = t.tile_rows;
  if (half_weights)
    return out_half ? launch_tile_src<kSrcHalf, __half>(c, rows, st) : launch_tile_src<kSrcHalf, __nv_bfloat16>(c, rows, st);
  if (codec == Q4_K)
    return out_half ? launch_tile_src<kSrcQ4K, __half>(c, rows, st) : launch_tile_src<kSrcQ4K, __nv_bfloat16>(c, rows, st);
  return out_half ? launch_tile_src<kSrcQ6K, __half>(c, rows, st) : launch_tile_src<kSrcQ6K, __nv_bfloat16>(c, rows, st);
}

}  // namespace kq
