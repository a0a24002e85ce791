// More than 16 activation rows: the entry (launch_gemm, launch_gemm_tiles), the pre-pass that makes fp16 rows of bf16 and
// float32 ones, the copy path that dequantizes a matrix to fp16 once, and the tile kernel for weights that kq_tile.cu does
// not take: y[M, N] = x[M, K] . dequant(W)^T on the 5th-generation tensor cores, replacing the reference's
// dequantize-then-GEMM CPU path (src/kquant_cpu_decode.cpp:1299-1352) and its Metal tile kernels
// (src/kquant_matmul.cpp:313-527).
//
// The tile kernel here serves every codec and alignment through decode8<> - small matrices, weights off the 16-byte grid,
// grouped calls of codecs other than q4_k and q6_k. One CTA computes a (128*MT) x 128 output tile, MT in {1, 2, 4}:
//   warps 0-7  weight producers: wire bytes -> fp16 in registers -> the
//              128B-swizzled K-major tile of a 3-deep ring; fence.proxy.async +
//              mbarrier arrive. Two threads per weight row, 32 weights each.
//   warp 8..   one thread per issuer warp issues tcgen05.mma (M=128, N=128, K=16, kind::f16, fp32
//              accumulators in tensor memory: MT x 128 columns); tcgen05.commit
//              hands activation slots and weight stages back.
//   last warp  one thread streams activation tiles [128 rows x 64] with TMA
//              (cp.async.bulk.tensor.2d, 128B swizzle, zero fill past M and K)
//              into a ring of 4 or 8 slots, ahead of the MMAs.
//   warps 0-7  epilogue: tcgen05.ld the accumulators, round once, whole rows through shared memory.
// Both operands are fp16: rounding a dequantized weight to bf16 alone would cost
// 1.6e-3 relative error and break the 2e-3 budget together with a bf16 output
// (fp16 costs 3e-4), and kind::f16 takes no bf16 A operand next to an fp16 B
// operand, so bf16 / f32 activations are first
// converted to fp16 by convert_x_kernel - exactly, with a per-row power-of-two
// factor that the epilogue undoes.
//
// Every mbarrier wait is bounded (2 s of %globaltimer): on expiry the CTA raises
// a flag in g_kq_device_error, stops issuing work, frees its tensor memory and
// returns, so a logic error can never leave the GPU spinning.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_launch.h"
#include "kq_tcgen05.cuh"
#include "kq_tma_map.h"

namespace cg = cooperative_groups;

namespace kq {

constexpr int kBN = 128;
constexpr int kBK = 64;
constexpr int kBStages = 3;  // weight-tile ring
// Eight producer warps, then the MMA issuer warp(s) and one TMA warp; two producer threads per weight row (32 weights
// each per K-step).
constexpr int kProducerThreads = 256;
// One thread issues the MMAs of an accumulator row block; a tcgen05.mma costs its issuing thread ~75 cycles
// (measured) against 128 cycles of tensor-pipe time, and every K-step adds barrier waits and commits, so ONE
// issuer for two or four row blocks leaves the pipe idle half of the time: tiles with two or more row blocks
// have two issuer warps (row blocks h = 0, 2 and h = 1, 3).
__host__ __device__ constexpr int mma_warps(int MT) { return MT >= 2 ? 2 : 1; }
__host__ __device__ constexpr int gemm_threads(int MT) { return kProducerThreads + 32 * (mma_warps(MT) + 1); }
__host__ __device__ constexpr int a_slots(int MT) { return MT == 1 ? 4 : 8; }  // activation-tile ring
constexpr int kTileBytes = 128 * 128;  // 128 rows x 64 16-bit elements

__device__ int g_kq_device_error = 0;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  return mbar_wait_err(bar, parity, abort_flag, code, &g_kq_device_error);
}

__device__ __forceinline__ uint32_t pack_h2f(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
constexpr int kTileGridCap = 256;  // grid.y of the grouped kernel, see launch_gemm_tiles

struct GemmArgs {
  const void* x;
  long long x_row_stride;
  void* y;
  long long y_row_stride;
  const uint8_t* w;
  long long row_bytes;
  int M, N, K;
  const float* row_scale;  // per-row factor applied in the epilogue, or nullptr
  // grouped (mixture-of-experts) mode: CTA row tiles come from a device-built list
  const GemmTile* tiles;       // nullptr = dense
  const int* n_tiles_dev;      // valid entries of `tiles`
  long long w_expert_stride;   // bytes between expert matrices
  const int* yrow;             // output row of each (expert-sorted) activation row
};

// ---- weight producers: 64 consecutive weights of one row -> eight swizzled 16-byte chunks
// hh = 0 / 1: which 32 of the 64 weights this thread makes (chunks 4hh .. 4hh+3)
template <int C, int A>
__device__ __forceinline__ void produce_w_generic(const uint8_t* row, int kb, int K, uint8_t* dst_row, int r, int hh,
                                                  const IqTables& tabs) {
  constexpr int BPB = bpb_of(C);
#pragma unroll 2
  for (int c = 4 * hh; c < 4 * hh + 4; c++) {
    const int k = kb * kBK + c * 8;
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    if (k < K) {
      float v[8];
      decode8<C, A>(row + block_of<C>(k) * BPB, octet_of<C>(k), v, tabs);
      out = make_uint4(pack_h2f(v[0], v[1]), pack_h2f(v[2], v[3]), pack_h2f(v[4], v[5]), pack_h2f(v[6], v[7]));
    }
    *reinterpret_cast<uint4*>(dst_row + ((c ^ (r & 7)) << 4)) = out;
  }
}

// q6_k (src/kquant_cpu_decode.cpp:238-280): K-chunk kb is weights 64 p .. 64 p + 63 of superblock kb >> 2,
// p = kb & 3: half hf = p >> 1, quarters qd = 2 (p & 1) + hh for the row's two threads. Thread hh makes the 32
// weights l = 0..31 of its quarter: q = nibble of ql[64 hf + 32 hh + l] (high nibbles for the upper two
// quarters) | two bits 2 qd of qh[32 hf + l] << 4. The six-bit value becomes fp16 through the 1024 + q bit
// pattern, q - 32 is exact, and the weight is (q - 32) * fp16(d * scale): two roundings (scale, product)
// instead of the generic path's one, 2^-10 at worst, for a third of the instructions.
template <int A>
__device__ __forceinline__ void produce_w_q6k(const uint8_t* row, int kb, uint8_t* dst_row, int r, int hh) {
  const uint8_t* blk = row + (long long)(kb >> 2) * 210;
  const int p = kb & 3, hf = p >> 1, qd = 2 * (p & 1) + hh;
  const float d = ldf16<A>(blk + 208);
  const int is = 8 * hf + 2 * qd;
  const uint32_t sc2 = (uint32_t)blk[192 + is] | ((uint32_t)blk[193 + is] << 8);
  const __half2 sA = __float2half2_rn(d * (float)(int)(int8_t)(sc2 & 0xffu));
  const __half2 sB = __float2half2_rn(d * (float)(int)(int8_t)(sc2 >> 8));
  const __half2 k1056 = __float2half2_rn(1056.f);
  const uint8_t* ql = blk + 64 * hf + 32 * hh;
  const uint8_t* qh = blk + 128 + 32 * hf;
  const int nsh = (qd & 2) ? 4 : 0;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    uint32_t o[4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t L = ld32<A>(ql + 8 * c + 4 * h), H = ld32<A>(qh + 8 * c + 4 * h);
      const uint32_t hb = (qd < 2) ? (H << (4 - 2 * (qd & 1))) : (H >> (2 * (qd & 1)));
      const uint32_t q4 = ((L >> nsh) & 0x0f0f0f0fu) | (hb & 0x30303030u);
      const __half2 s = c < 2 ? sA : sB;
      const uint32_t m0 = __byte_perm(q4, 0x64646464u, 0x4140), m1 = __byte_perm(q4, 0x64646464u, 0x4342);
      const __half2 w0 = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&m0), k1056), s);
      const __half2 w1 = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&m1), k1056), s);
      o[2 * h] = *reinterpret_cast<const uint32_t*>(&w0);
      o[2 * h + 1] = *reinterpret_cast<const uint32_t*>(&w1);
    }
    *reinterpret_cast<uint4*>(dst_row + (((c + 4 * hh) ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// ------------------------------------------------------------------ the kernel
// Activations are always fp16 here (bf16 / f32 callers go through
// convert_x_kernel first) and arrive through the tensor map. OT: output type.
template <int C, int A, typename OT, int MT>
__global__ void __launch_bounds__(gemm_threads(MT), 1)
gemm_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap tmap_x) {
  constexpr int kGemmThreads = gemm_threads(MT), kMmaWarp = kProducerThreads / 32, kMmaWarps = mma_warps(MT);
  constexpr bool kHalf = std::is_same<OT, __half>::value;
  constexpr int NA = a_slots(MT), BN = kBN;
  constexpr bool kIq = (C == IQ4_NL || C == IQ4_XS || C == IQ2_XXS);
  extern __shared__ __align__(1024) uint8_t gemm_smem[];
  // 1024-byte alignment of the tiles is what the 128B swizzle pattern assumes
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm_smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* b_ring = tiles;                          // kBStages weight tiles
  uint8_t* a_ring = tiles + kBStages * kTileBytes;  // NA activation slots
  __shared__ uint64_t b_full[kBStages], b_empty[kBStages], a_full[NA], a_empty[NA], accum_bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  __shared__ __align__(16) uint8_t s_tabs[kIq ? kIqSmemBytes : 16];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kBN, n_end = min(a.N, n0 + kBN);
  // Grouped mode: the CTA takes tile blockIdx.y of the device-built list, then every gridDim.y-th after it (the
  // grid is sized on the host for the largest list the call could produce, capped; the list is usually far
  // shorter, and a CTA with no tile leaves before it allocates anything).
  const int n_list = a.tiles != nullptr ? *a.n_tiles_dev : 0;
  if (a.tiles != nullptr && (int)blockIdx.y >= n_list) return;
  // K-steps of this CTA: all of them, or slice blockIdx.z of gridDim.z equal slices (split K, below)
  const int KB = (a.K + kBK - 1) / kBK / (int)gridDim.z;
  const int kb0 = (int)blockIdx.z * KB;
  constexpr uint32_t kTmemCols = MT * BN;               // 128, 256 or 512: a power of two >= 32

  IqTables tabs = global_iq_tables();
  if constexpr (kIq) tabs = stage_iq_tables(s_tabs, threadIdx.x, kGemmThreads);
  if (threadIdx.x == 0) abort_s = 0;
  if (warp == kMmaWarp) tmem_alloc(&tmem_base_s, kTmemCols);
  volatile int* abort_flag = &abort_s;
  uint32_t tmem_base = 0;

  for (int tile = (int)blockIdx.y;; tile += (int)gridDim.y) {
    int m0 = tile * (128 * MT), m_end = a.M;
    const uint8_t* wbase = a.w;
    if (a.tiles != nullptr) {
      const GemmTile t = a.tiles[tile];
      m0 = t.row_start;
      m_end = t.row_start + t.rows;
      wbase += (long long)t.expert * a.w_expert_stride;
    }
    const int mt_live = min(MT, (m_end - m0 + 127) / 128);  // activation tiles of this CTA that hold rows
    // Every tile starts from freshly initialised barriers (phase 0): nothing is in flight between tiles - the
    // loader has waited for its last loads, the issuers' MMAs have completed, the epilogue has stored.
    if (threadIdx.x == 0) {
      const bool again = tile != (int)blockIdx.y;
      for (int s = 0; s < kBStages; s++) {
        if (again) mbar_inval(&b_full[s]), mbar_inval(&b_empty[s]);
        mbar_init(&b_full[s], kProducerThreads / 32);
        mbar_init(&b_empty[s], kMmaWarps);
      }
      for (int s = 0; s < NA; s++) {
        if (again) mbar_inval(&a_full[s]), mbar_inval(&a_empty[s]);
        mbar_init(&a_full[s], 1);
        mbar_init(&a_empty[s], 1);
      }
      if (again) mbar_inval(&accum_bar);
      mbar_init(&accum_bar, kMmaWarps);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem_base = tmem_base_s;

    if (warp < kMmaWarp) {
      // ================= weight producers =================
      const int tid = threadIdx.x;
      const int wr = tid % 128, hh = tid / 128;  // weight row of the tile; which 32 of its 64 weights per K-step
      const uint8_t* wrow = wbase + (long long)min(n0 + wr, a.N - 1) * a.row_bytes;
      bool ok = true;
      for (int it = 0; it < KB && ok; it++) {
        const int s = it % kBStages;
        if (it >= kBStages) ok = mbar_wait(&b_empty[s], ((it / kBStages) & 1) ^ 1, abort_flag, 1);
        if (!ok) break;
        uint8_t* wdst = b_ring + s * kTileBytes + wr * 128;
        if constexpr (C == Q6_K && A >= 2) produce_w_q6k<2>(wrow, kb0 + it, wdst, wr, hh);  // blocks are 2-byte aligned
        else produce_w_generic<C, A>(wrow, kb0 + it, a.K, wdst, wr, hh, tabs);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_full[s]);
      }
      // ================= epilogue =================
      if (ok) ok = mbar_wait(&accum_bar, 0, abort_flag, 4);
      if (ok) {
        tc_fence_after();
        const int lq = warp & 3;                   // TMEM lane quarter this warp may read
        constexpr int kColSpan = BN / (kProducerThreads / 128);  // four warps (one per lane quarter) per column span
        const int cbeg = (warp >> 2) * kColSpan;
        if (gridDim.z > 1) {
          // split K: this CTA's partial tile goes to shared memory (the rings are idle now) as fp32
          // [rows][BN], 16-byte chunks XOR-swizzled by the row so that a warp's stores spread over the banks
          if constexpr (MT <= 2) {  // the partial tile fits the rings
  #pragma unroll 1
            for (int h = 0; h < mt_live; h++) {
              const int rl = h * 128 + lq * 32 + lane;
              const float rs = (a.row_scale && m0 + rl < m_end) ? a.row_scale[m0 + rl] : 1.f;
              float* srow = reinterpret_cast<float*>(tiles) + rl * BN;
  #pragma unroll 1
              for (int c0 = cbeg; c0 < cbeg + kColSpan; c0 += 16) {
                uint32_t v[16];
                tmem_ld16(tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(h * BN + c0), v);
                tmem_ld_wait();
  #pragma unroll
                for (int i = 0; i < 4; i++)
                  *reinterpret_cast<float4*>(srow + 4 * (((c0 >> 2) + i) ^ (rl & 31))) =
                      make_float4(__uint_as_float(v[4 * i]) * rs, __uint_as_float(v[4 * i + 1]) * rs,
                                  __uint_as_float(v[4 * i + 2]) * rs, __uint_as_float(v[4 * i + 3]) * rs);
              }
            }
          }
        } else {
          // A thread owns one accumulator row (a TMEM lane): storing from here would write 32 rows x 32 bytes per
          // instruction, one memory transaction per lane. The rounded tile goes through shared memory instead (the
          // rings are idle: every MMA has completed), rows of BN outputs with their 16-byte chunks XOR-swizzled by
          // the row, and leaves as whole rows, 16 bytes per lane.
          constexpr int kRowBytes = BN * 2, kChunks = BN / 8;
          uint8_t* stage = tiles;
  #pragma unroll 1
          for (int h = 0; h < mt_live; h++) {
            const int rl = h * 128 + lq * 32 + lane;
            const float rs = (a.row_scale && m0 + rl < m_end) ? a.row_scale[m0 + rl] : 1.f;
            uint8_t* srow = stage + rl * kRowBytes;
  #pragma unroll 1
            for (int c0 = cbeg; c0 < cbeg + kColSpan; c0 += 32) {
              uint32_t va[16], vb[16];
              tmem_ld16(tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(h * BN + c0), va);
              tmem_ld16(tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(h * BN + c0 + 16), vb);
              tmem_ld_wait();
              uint32_t o[16];
  #pragma unroll
              for (int i = 0; i < 16; i++) {
                const uint32_t u0 = i < 8 ? va[2 * i] : vb[2 * i - 16], u1 = i < 8 ? va[2 * i + 1] : vb[2 * i - 15];
                const float f0 = __uint_as_float(u0) * rs, f1 = __uint_as_float(u1) * rs;
                if constexpr (kHalf) {
                  o[i] = pack_h2f(f0, f1);
                } else {
                  __nv_bfloat162 bb = __floats2bfloat162_rn(f0, f1);
                  o[i] = *reinterpret_cast<uint32_t*>(&bb);
                }
              }
  #pragma unroll
              for (int q = 0; q < 4; q++)
                *reinterpret_cast<uint4*>(srow + ((((c0 >> 3) + q) ^ (rl & (kChunks - 1))) << 4)) =
                    make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            }
          }
          asm volatile("bar.sync 2, %0;\n" ::"n"(kProducerThreads) : "memory");
          const int rows_live = min(m_end - m0, mt_live * 128);
          constexpr int kRowsPerPass = 32 / kChunks;  // two rows of 128 columns per warp instruction
          const int chunk = lane % kChunks;
          const int col = n0 + chunk * 8;
          OT* ybase = static_cast<OT*>(a.y);
          // Output rows come from a table in grouped mode. A load per row inside the loop would put a global-memory
          // round trip before every store (measured: 12 k of a tile's 18 k epilogue cycles), so lane i fetches the
          // rows of pass i up front (at most 32 passes for every tile shape) and the passes read them by shuffle.
          constexpr int kPassRows = (kProducerThreads / 32) * kRowsPerPass;
          const int passes = (rows_live + kPassRows - 1) / kPassRows;
          const int sub = lane / kChunks;  // which of the pass's rows of this warp (kRowsPerPass = 2) the lane stores
          long long mine0 = 0, mine1 = 0;
          {
            const int r0 = warp * kRowsPerPass + lane * kPassRows;
            if (r0 < rows_live) mine0 = a.yrow ? (long long)a.yrow[m0 + r0] : (long long)(m0 + r0);
            if (r0 + 1 < rows_live) mine1 = a.yrow ? (long long)a.yrow[m0 + r0 + 1] : (long long)(m0 + r0 + 1);
          }
          for (int i = 0; i < passes; i++) {
            const long long o0 = __shfl_sync(0xffffffffu, mine0, i), o1 = __shfl_sync(0xffffffffu, mine1, i);
            const int r = warp * kRowsPerPass + sub + i * kPassRows;
            if (r >= rows_live) continue;
            const long long orow = sub ? o1 : o0;
            const uint4 q = *reinterpret_cast<const uint4*>(stage + r * kRowBytes + ((chunk ^ (r & (kChunks - 1))) << 4));
            OT* yp = ybase + orow * a.y_row_stride + col;
            if (col + 8 <= n_end && (reinterpret_cast<uintptr_t>(yp) & 15) == 0) {
              *reinterpret_cast<uint4*>(yp) = q;
            } else {
              const OT* qe = reinterpret_cast<const OT*>(&q);
              for (int e = 0; e < 8; e++)
                if (col + e < n_end) yp[e] = qe[e];
            }
          }
        }
      }
    } else if (warp < kMmaWarp + kMmaWarps) {
      // ================= MMA issuers =================
      // Issuer w takes the row blocks h = w, w + kMmaWarps, ...; the activation tile of (K-step kb, row block h)
      // is tile number kb * mt_live + h of the loader's sequence. Every issuer arrives on every stage barrier
      // (a commit with no MMA of its own completes at once), so the counts do not depend on mt_live.
      const uint32_t idesc = umma_idesc(0u, kBN);
      const int w = warp - kMmaWarp;
      bool ok = true;
      for (int kb = 0; kb < KB && ok; kb++) {  // kb counts this CTA's own K-steps
        const int s = kb % kBStages;
        ok = mbar_wait(&b_full[s], (kb / kBStages) & 1, abort_flag, 2);
        if (!ok) break;
        const uint32_t bt = smem_u32(b_ring + s * kTileBytes);
        for (int h = w; h < mt_live && ok; h += kMmaWarps) {
          const int t = kb * mt_live + h;
          const int slot = t % NA;
          ok = mbar_wait(&a_full[slot], (t / NA) & 1, abort_flag, 16);
          if (!ok) break;
          tc_fence_after();
          if (lane == 0) {
            const uint32_t at = smem_u32(a_ring + slot * kTileBytes);
  #pragma unroll
            for (int j = 0; j < kBK / 16; j++)
              umma_f16(tmem_base + h * BN, umma_desc_sw128(at + j * 32), umma_desc_sw128(bt + j * 32), idesc,
                       (kb > 0 || j > 0) ? 1u : 0u);
            umma_commit(&a_empty[slot]);  // the slot is free once these MMAs have read it
          }
          __syncwarp();
        }
        if (ok && lane == 0) umma_commit(&b_empty[s]);
        __syncwarp();
      }
      if (lane == 0) umma_commit(&accum_bar);  // also on the abort path: lets the wait below see the MMAs drain
      __syncwarp();
      if (!ok) mbar_wait(&accum_bar, 0, abort_flag, 8);
    } else {
      // ================= activation loader (TMA) =================
      bool ok = true;
      int t = 0;
      for (int kb = 0; kb < KB && ok; kb++) {
        for (int h = 0; h < mt_live && ok; h++, t++) {
          const int slot = t % NA;
          if (t >= NA) ok = mbar_wait(&a_empty[slot], ((t / NA) & 1) ^ 1, abort_flag, 32);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&a_full[slot], kTileBytes);
            tma_load_2d(a_ring + slot * kTileBytes, &tmap_x, (kb0 + kb) * kBK, m0 + h * 128, &a_full[slot]);
          }
          __syncwarp();
        }
      }
      // In-flight loads must have landed before the CTA may exit: wait (bounded) for the last ones.
      if (ok && t > 0) {
        const int first = t > NA ? t - NA : 0;
        for (int u = first; u < t; u++)
          if (!mbar_wait(&a_full[u % NA], (u / NA) & 1, abort_flag, 64)) break;
      }
    }

    // ================= split K: the slices of a cluster meet through distributed shared memory =================
    if (gridDim.z > 1) {
      if constexpr (MT <= 2) {
        cg::cluster_group cluster = cg::this_cluster();
        tc_fence_before();
        cluster.sync();  // every slice's partial tile is in its shared memory
        const int S = (int)gridDim.z, z = (int)blockIdx.z;
        if (warp < kMmaWarp) {
          const float* peer[8];
  #pragma unroll
          for (int q = 0; q < 8; q++)
            peer[q] = q < S ? cluster.map_shared_rank(reinterpret_cast<float*>(tiles), q) : nullptr;
          for (int rl = z + S * (threadIdx.x >> 5); rl < mt_live * 128; rl += S * (kProducerThreads / 32)) {
            const int row = m0 + rl;
            if (row >= m_end) continue;
            const int c = threadIdx.x & 31;  // 16-byte chunk = four columns
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  #pragma unroll
            for (int q = 0; q < 8; q++) {
              if (q < S) {
                const float4 v = *reinterpret_cast<const float4*>(peer[q] + rl * BN + 4 * (c ^ (rl & 31)));
                acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
              }
            }
            OT* yp = static_cast<OT*>(a.y) + (long long)row * a.y_row_stride + n0 + 4 * c;
            const float f[4] = {acc.x, acc.y, acc.z, acc.w};
  #pragma unroll
            for (int i = 0; i < 4; i++) {
              if (n0 + 4 * c + i < n_end) {
                if constexpr (kHalf) yp[i] = __float2half_rn(f[i]);
                else yp[i] = __float2bfloat16_rn(f[i]);
              }
            }
          }
        }
        cluster.sync();  // peers may still be reading this CTA's partial tile
      }
    }

    // ================= end of the tile =================
    tc_fence_before();
    __syncthreads();
    if (a.tiles == nullptr || tile + (int)gridDim.y >= n_list || abort_s != 0) break;
  }  // tile loop

  // ================= teardown =================
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------ activation pre-pass
// bf16 / f32 activations -> fp16 for the tensor-core tile kernel (kind::f16 does
// not accept a bf16 A operand next to an fp16 B operand). float input is first
// rounded to bf16, as the reference's op does (src/kquant_ops.cpp:159-168). A
// bf16 value converts to fp16 exactly unless it is out of fp16's range, so each
// row is divided by a power of two 2^e (e = 0 for every row whose largest
// magnitude is below 32768, i.e. practically always) and the factor is handed to
// the epilogue: nothing saturates, nothing is rounded twice.
// Gather mode (order != nullptr): output row r is activation row
// lhs[order[r / M]] * M + r % M of x, and yrow[r] = order[r / M] * M + r % M says where
// its result goes; this is the expert-sorted copy the grouped kernel streams with TMA.
template <typename XT>
__global__ void __launch_bounds__(256)
convert_x_scalar_kernel(const XT* __restrict__ x, long long x_row_stride, int K, __half* __restrict__ xh,
                 float* __restrict__ row_scale, const int* __restrict__ order, const uint32_t* __restrict__ lhs, int M,
                 int* __restrict__ yrow, const int* __restrict__ n_valid) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");  // the tile kernel fetches weights meanwhile
  const long long row = blockIdx.x;
  long long src_row = row;
  // gather mode: entries whose expert index is out of range were never placed in `order`; its tail is unset
  if (n_valid != nullptr && row >= (long long)(*n_valid) * M) return;
  if (order != nullptr) {
    const int entry = order[row / M], i = (int)(row % M);
    src_row = (long long)lhs[entry] * M + i;
    if (threadIdx.x == 0) yrow[row] = entry * M + i;
  } else if (lhs != nullptr) {
    src_row = (long long)lhs[row / M] * M + row % M;  // entry order, no sort
  }
  const XT* xr = x + src_row * x_row_stride;
  __half* o = xh + row * (long long)K;
  if constexpr (std::is_same<XT, __half>::value) {
    for (int k = threadIdx.x * 8; k < K; k += 256 * 8)
      *reinterpret_cast<uint4*>(o + k) = __ldg(reinterpret_cast<const uint4*>(xr + k));
    if (threadIdx.x == 0) row_scale[row] = 1.f;
    return;
  } else {
    __shared__ float s_max[8];
    float mx = 0.f;
    for (int k = threadIdx.x; k < K; k += 256) {
      float v;
      if constexpr (sizeof(XT) == 2) v = __bfloat162float(xr[k]);
      else v = __bfloat162float(__float2bfloat16_rn(xr[k]));
      v = fabsf(v);
      if (v < INFINITY) mx = fmaxf(mx, v);  // inf / nan propagate on their own
    }
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = s_max[0];
    for (int i = 1; i < 8; i++) mx = fmaxf(mx, s_max[i]);
    // Every row is normalised: its largest magnitude lands in [16384, 32768), so small rows keep their
    // mantissas instead of turning into fp16 subnormals. The factor 2^-e is applied in two exact halves
    // (2^-e alone overflows float32 for the smallest bf16 magnitudes).
    int e = 0;
    if (mx > 0.f) e = ilogbf(mx) - 14;
    const int eh = (-e) / 2;
    const float down1 = ldexpf(1.f, eh), down2 = ldexpf(1.f, -e - eh);
    if (threadIdx.x == 0) row_scale[row] = ldexpf(1.f, e);
    for (int k = threadIdx.x; k < K; k += 256) {
      float v;
      if constexpr (sizeof(XT) == 2) v = __bfloat162float(xr[k]);
      else v = __bfloat162float(__float2bfloat16_rn(xr[k]));
      o[k] = __float2half_rn(v * down1 * down2);
    }
  }
}


// ---- the same pre-pass, eight activations per access: one warp per row, the first 2048 activations of a row
// stay in registers between the two passes (largest magnitude, then the scaled copy). Rows and K must be whole
// numbers of 16 bytes (callers fall back to the scalar kernel above otherwise).
// GLU: the source row holds gate | up (2 K values); the activation is h = silu(gate) * up, rounded to XT first -
// the value a separate activation kernel would have stored - so the fused form changes no bit of the product.
// Eight consecutive activations as four bf16 pairs (float input rounded to bf16 as the reference's op does).
template <typename XT>
__device__ __forceinline__ uint4 cvt_load8_bf16(const XT* p) {
  if constexpr (sizeof(XT) == 4) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    const __nv_bfloat162 q0 = __floats2bfloat162_rn(a.x, a.y), q1 = __floats2bfloat162_rn(a.z, a.w),
                         q2 = __floats2bfloat162_rn(b.x, b.y), q3 = __floats2bfloat162_rn(b.z, b.w);
    return make_uint4(*reinterpret_cast<const uint32_t*>(&q0), *reinterpret_cast<const uint32_t*>(&q1),
                      *reinterpret_cast<const uint32_t*>(&q2), *reinterpret_cast<const uint32_t*>(&q3));
  } else {
    return __ldg(reinterpret_cast<const uint4*>(p));
  }
}
// The fused activation over eight gate / up pairs of 16-bit type XT: h = silu(gate) * up rounded to XT, returned
// as XT pairs.
template <typename XT>
__device__ __forceinline__ uint4 cvt_glu8(const XT* xr, int K, int c) {
  const uint4 g = __ldg(reinterpret_cast<const uint4*>(xr + 8 * c));
  const uint4 u = __ldg(reinterpret_cast<const uint4*>(xr + K + 8 * c));
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if constexpr (std::is_same<XT, __half>::value) {
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&gw[i]));
      const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&uw[i]));
      o[i] = pack_h2f(silu_f(a.x) * b.x, silu_f(a.y) * b.y);
    } else {
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&uw[i]));
      const __nv_bfloat162 h = __floats2bfloat162_rn(silu_f(a.x) * b.x, silu_f(a.y) * b.y);
      o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
template <typename XT, bool GLU>
__device__ __forceinline__ uint4 cvt_fetch8(const XT* xr, int K, int c) {
  if constexpr (GLU) return cvt_glu8<XT>(xr, K, c);
  else return cvt_load8_bf16<XT>(xr + 8 * c);
}
__device__ __forceinline__ __nv_bfloat162 cvt_absmax(__nv_bfloat162 m, const uint4& q) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));  // skips NaNs
  return m;
}
__device__ __forceinline__ float cvt_finite_absmax(float m, const uint4& q) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    if (fabsf(f.x) < INFINITY) m = fmaxf(m, fabsf(f.x));
    if (fabsf(f.y) < INFINITY) m = fmaxf(m, fabsf(f.y));
  }
  return m;
}
// bf16 pairs times s1 * s2 (powers of two: exact) -> fp16 pairs
__device__ __forceinline__ uint4 cvt_scale8(const uint4& q, float s1, float s2) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    o[i] = pack_h2f(f.x * s1 * s2, f.y * s1 * s2);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
constexpr int kCvtChunks = 8;
// A CTA per row, for calls with fewer rows than the SMs hold warps: a row's chunks are then read by 256 threads at once
// instead of one after the other by 32 (61 rows of 8192 bf16: the call 110.9 -> 106.9 us); with 2300 rows
// it is 3 us slower. Dense rows only.
template <typename XT>
__global__ void __launch_bounds__(256)
convert_rows_kernel(const XT* __restrict__ x, long long x_row_stride, int K, __half* __restrict__ xh,
                    float* __restrict__ row_scale) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  __shared__ float s_max[8];
  const XT* xr = x + blockIdx.x * x_row_stride;
  __half* o = xh + blockIdx.x * (long long)K;
  const int nch = K >> 3;
  uint4 keep[kCvtChunks];  // further chunks are read again
  float mx = 0.f;
#pragma unroll
  for (int j = 0; j < kCvtChunks; j++) {
    const int c = threadIdx.x + 256 * j;
    if (c < nch) {
      keep[j] = cvt_load8_bf16<XT>(xr + 8 * c);
      mx = cvt_finite_absmax(mx, keep[j]);  // infinities propagate on their own, the factor comes from the finite values
    }
  }
  for (int c = threadIdx.x + 256 * kCvtChunks; c < nch; c += 256) mx = cvt_finite_absmax(mx, cvt_load8_bf16<XT>(xr + 8 * c));
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = s_max[0];
#pragma unroll
  for (int i = 1; i < 8; i++) mx = fmaxf(mx, s_max[i]);
  // normalised as in convert_x_kernel; 2^-e in two exact halves, since it can overflow float32
  int e = 0;
  if (mx > 0.f) e = ilogbf(mx) - 14;
  const int eh = (-e) / 2;
  const float down1 = ldexpf(1.f, eh), down2 = ldexpf(1.f, -e - eh);
  if (threadIdx.x == 0) row_scale[blockIdx.x] = ldexpf(1.f, e);
#pragma unroll
  for (int j = 0; j < kCvtChunks; j++) {
    const int c = threadIdx.x + 256 * j;
    if (c < nch) *reinterpret_cast<uint4*>(o + 8 * c) = cvt_scale8(keep[j], down1, down2);
  }
  for (int c = threadIdx.x + 256 * kCvtChunks; c < nch; c += 256)
    *reinterpret_cast<uint4*>(o + 8 * c) = cvt_scale8(cvt_load8_bf16<XT>(xr + 8 * c), down1, down2);
}

// CH: chunks of a lane that stay in registers. Rows of at most 1024 values need four, which lets twice the warps reside:
// a row is a chain of loads, a reduction and stores, and only other rows hide it.
template <typename XT, bool GLU, int CH>
__global__ void __launch_bounds__(256, CH == 4 ? 6 : 3)
convert_x_kernel(const XT* __restrict__ x, long long x_row_stride, int K, __half* __restrict__ xh,
                 float* __restrict__ row_scale, const int* __restrict__ order, const uint32_t* __restrict__ lhs,
                 int lhs_div, int M, int* __restrict__ yrow, const int* __restrict__ n_valid, long long rows) {
  static_assert(!GLU || sizeof(XT) == 2, "the fused activation takes fp16 / bf16 gate | up rows");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int lane = threadIdx.x & 31;
  // rows that exist: all, or the first *n_valid * M in gather mode (see the scalar kernel). The grid is capped on
  // the host and the warps stride over the rows, so a list sized for many more rows than it holds costs nothing.
  const long long limit = n_valid != nullptr ? min(rows, (long long)(*n_valid) * M) : rows;
  for (long long row = blockIdx.x * 8LL + (threadIdx.x >> 5); row < limit; row += gridDim.x * 8LL) {
    long long src_row = row;
    if (order != nullptr) {
      const int entry = order[row / M], i = (int)(row % M);
      // the activation row of an entry: that of unit u = entry / lhs_div (lhs_div = k routed rows per token when
      // the entries are a [tokens, k] routing table, else 1), through lhs when there is an index array
      const int u = entry / lhs_div;
      src_row = (lhs != nullptr ? (long long)lhs[u] : (long long)u) * M + i;
      if (lane == 0 && yrow != nullptr) yrow[row] = entry * M + i;
    } else if (lhs != nullptr) {
      src_row = (long long)lhs[row / M] * M + row % M;
    }
    const XT* xr = x + src_row * x_row_stride;
    __half* o = xh + row * (long long)K;
    const int nch = K >> 3;
    if constexpr (std::is_same<XT, __half>::value) {
      for (int c = lane; c < nch; c += 32) *reinterpret_cast<uint4*>(o + 8 * c) = cvt_fetch8<XT, GLU>(xr, K, c);
      if (lane == 0) row_scale[row] = 1.f;
    } else {
      uint4 keep[CH];  // the row's values as bf16 pairs (they are bf16 values: nothing is lost)
      __nv_bfloat162 m2 = __floats2bfloat162_rn(0.f, 0.f);
  #pragma unroll
      for (int j = 0; j < CH; j++) {
        const int c = lane + 32 * j;
        if (c < nch) {
          keep[j] = cvt_fetch8<XT, GLU>(xr, K, c);
          m2 = cvt_absmax(m2, keep[j]);
        }
      }
      for (int c = lane + 32 * CH; c < nch; c += 32) m2 = cvt_absmax(m2, cvt_fetch8<XT, GLU>(xr, K, c));
      float mx = fmaxf(__low2float(m2), __high2float(m2));
      for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      if (!(mx < INFINITY)) {
        // a row with infinities: they propagate on their own, the factor comes from the finite values
        mx = 0.f;
  #pragma unroll
        for (int j = 0; j < CH; j++)
          if (lane + 32 * j < nch) mx = cvt_finite_absmax(mx, keep[j]);
        for (int c = lane + 32 * CH; c < nch; c += 32) mx = cvt_finite_absmax(mx, cvt_fetch8<XT, GLU>(xr, K, c));
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      }
      // Every row is normalised (see the scalar kernel); 2^-e in two exact halves, since it can overflow float32.
      int e = 0;
      if (mx > 0.f) e = ilogbf(mx) - 14;
      const int eh = (-e) / 2;
      const float down1 = ldexpf(1.f, eh), down2 = ldexpf(1.f, -e - eh);
      if (lane == 0) row_scale[row] = ldexpf(1.f, e);
  #pragma unroll
      for (int j = 0; j < CH; j++) {
        const int c = lane + 32 * j;
        if (c < nch) *reinterpret_cast<uint4*>(o + 8 * c) = cvt_scale8(keep[j], down1, down2);
      }
      for (int c = lane + 32 * CH; c < nch; c += 32)
        *reinterpret_cast<uint4*>(o + 8 * c) = cvt_scale8(cvt_fetch8<XT, GLU>(xr, K, c), down1, down2);
    }
  }
}

template <typename XT>
static void launch_convert_t(const void* x, long long x_row_stride, int K, long long rows, const int* order,
                             const uint32_t* lhs, int lhs_div, int M, __half* o, float* row_scale, int* yrow,
                             const int* n_valid, bool glu, bool vec, cudaStream_t st) {
  const XT* xp = static_cast<const XT*>(x);
  const unsigned gv = (unsigned)std::min<long long>((rows + 7) / 8, 148 * 64);  // strided beyond; a lower cap left a thin second pass
  if (glu) {
    if constexpr (sizeof(XT) == 2)
      (K <= 1024 ? convert_x_kernel<XT, true, 4> : convert_x_kernel<XT, true, kCvtChunks>)<<<gv, 256, 0, st>>>(
          xp, x_row_stride, K, o, row_scale, order, lhs, lhs_div, M, yrow, n_valid, rows);
  } else if (vec && !std::is_same<XT, __half>::value && order == nullptr && lhs == nullptr &&
             n_valid == nullptr && rows <= 148 * 4) {
    if constexpr (!std::is_same<XT, __half>::value)
      convert_rows_kernel<XT><<<(unsigned)rows, 256, 0, st>>>(xp, x_row_stride, K, o, row_scale);
  } else if (vec) {
    (K <= 1024 ? convert_x_kernel<XT, false, 4> : convert_x_kernel<XT, false, kCvtChunks>)<<<gv, 256, 0, st>>>(
        xp, x_row_stride, K, o, row_scale, order, lhs, lhs_div, M, yrow, n_valid, rows);
  } else {
    convert_x_scalar_kernel<XT><<<(unsigned)rows, 256, 0, st>>>(xp, x_row_stride, K, o, row_scale, order, lhs, M, yrow,
                                                                n_valid);
  }
}

// One launch of the pre-pass: rows [rows, K] of x (dtype x_dtype, row stride in elements) -> xh, row_scale.
// order / lhs / lhs_div / M / yrow / n_valid as in the kernels; glu: x rows hold gate | up (2 K values).
cudaError_t launch_convert(int x_dtype, const void* x, long long x_row_stride, int K, long long rows, const int* order,
                           const uint32_t* lhs, int lhs_div, int M, void* xh, float* row_scale, int* yrow,
                           const int* n_valid, bool glu, cudaStream_t st) {
  if (rows <= 0 || K <= 0) return cudaSuccess;
  __half* o = static_cast<__half*>(xh);
  const size_t es = x_dtype == F32 ? 4 : 2;
  const bool vec = (K % 8) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ((size_t)x_row_stride * es) % 16 == 0 &&
                   (reinterpret_cast<uintptr_t>(xh) & 15) == 0;
  if (glu && (!vec || x_dtype == F32)) return cudaErrorInvalidValue;
  if (!vec && order != nullptr && (lhs == nullptr || lhs_div != 1)) return cudaErrorInvalidValue;  // vector kernel only
  if (x_dtype == F16)
    launch_convert_t<__half>(x, x_row_stride, K, rows, order, lhs, lhs_div, M, o, row_scale, yrow, n_valid, glu, vec, st);
  else if (x_dtype == BF16)
    launch_convert_t<__nv_bfloat16>(x, x_row_stride, K, rows, order, lhs, lhs_div, M, o, row_scale, yrow, n_valid, glu,
                                    vec, st);
  else
    launch_convert_t<float>(x, x_row_stride, K, rows, order, lhs, lhs_div, M, o, row_scale, yrow, n_valid, glu, vec, st);
  return cudaGetLastError();
}

cudaError_t launch_convert_rows(int x_dtype, const void* x, long long x_row_stride, int K, long long rows,
                                const uint32_t* lhs, int M, void* xh, float* row_scale, cudaStream_t st) {
  return launch_convert(x_dtype, x, x_row_stride, K, rows, nullptr, lhs, 1, M, xh, row_scale, nullptr, nullptr, false, st);
}

size_t gemm_workspace_bytes(int x_dtype, long long rows, int K) {
  // rows 2..16 of bf16 / f32 activations use the same fp16 copy (q4_k decode kernel); one row never does
  if (x_dtype == F16 || rows <= 1) return 0;
  const size_t xh = ((size_t)rows * (size_t)K * 2 + 255) & ~(size_t)255;
  return xh + (((size_t)rows * 4 + 255) & ~(size_t)255);
}

// ------------------------------------------------------------------ launch
// Tensor map of an fp16 matrix [M, K] (row stride in elements): boxes of 64 x box_rows, 128B swizzle.
static cudaError_t make_x_map(CUtensorMap* map, const void* x, long long x_row_stride, int M, int K, int box_rows = 128) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t strides[1] = {(cuuint64_t)x_row_stride * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int C, int A, typename OT, int MT>
static cudaError_t launch_g(GemmArgs a, cudaStream_t st, int grid_y = 0, int ksplit = 1) {
  auto kern = gemm_kernel<C, A, OT, MT>;
  const size_t dyn = (size_t)(kBStages + a_slots(MT)) * kTileBytes + 1024;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 16 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  alignas(64) CUtensorMap map;
  cudaError_t e = make_x_map(&map, a.x, a.x_row_stride, a.M, a.K);
  if (e != cudaSuccess) return e;
  if (MT > 2) ksplit = 1;  // split K needs the fp32 partial tile in shared memory
  const dim3 grid((a.N + kBN - 1) / kBN, grid_y > 0 ? grid_y : (a.M + 128 * MT - 1) / (128 * MT), ksplit);
  if (ksplit == 1) {
    kern<<<grid, gemm_threads(MT), dyn, st>>>(a, map);
    return cudaGetLastError();
  }
  // split K: the ksplit CTAs of one output tile form a cluster
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(gemm_threads(MT));
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ksplit;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a, map);
}

template <int C, int A>
static cudaError_t launch_shape(bool out_half, const GemmArgs& a, cudaStream_t st) {
  // Tile heights: 512 rows amortise the weight dequantization best, smaller ones fill the GPU at small M.
  const long long n_tiles = (a.N + kBN - 1) / kBN;
  int mt = a.M > 256 ? 4 : (a.M > 128 ? 2 : 1);
  if (mt == 4 && n_tiles * ((a.M + 511) / 512) < 148) mt = 2;
  // Few output tiles (small M on a matrix with few 128-row groups): split K over a cluster so that
  // the weights stream through more SMs. The slices must be equal: K-steps % ksplit == 0.
  const int kb_total = (a.K + kBK - 1) / kBK;
  int ksplit = 1;
  if (mt <= 2) {
    const long long ctas = n_tiles * ((a.M + 128 * mt - 1) / (128 * mt));
    while (ksplit < 8 && ctas * ksplit * 2 <= 160 && kb_total % (ksplit * 2) == 0 && kb_total / (ksplit * 2) >= 4) ksplit *= 2;
  }
  if (out_half) {
    if (mt == 4) return launch_g<C, A, __half, 4>(a, st);
    if (mt == 2) return launch_g<C, A, __half, 2>(a, st, 0, ksplit);
    return launch_g<C, A, __half, 1>(a, st, 0, ksplit);
  }
  if (mt == 4) return launch_g<C, A, __nv_bfloat16, 4>(a, st);
  if (mt == 2) return launch_g<C, A, __nv_bfloat16, 2>(a, st, 0, ksplit);
  return launch_g<C, A, __nv_bfloat16, 1>(a, st, 0, ksplit);
}

template <int C, int NAT>
static cudaError_t launch_codec(bool out_half, const GemmArgs& a, bool aligned, cudaStream_t st) {
  return aligned ? launch_shape<C, NAT>(out_half, a, st) : launch_shape<C, 1>(out_half, a, st);
}

// ---- many rows: the weights are dequantized to fp16 once and the tiles of both operands come by TMA
// rows of the matrix per pass: the fp16 copy stays below kHalfBytes (or 256 rows), so that most of it is still in
// the 126 MB L2 when it is read
constexpr long long kHalfBytes = 128ll << 20;
static int half_chunk(int N, int K) {
  const long long most = std::max<long long>(256, kHalfBytes / (2ll * K) / 128 * 128);
  const long long n = (N + most - 1) / most;
  return (int)std::min<long long>(N, ((N + n - 1) / n + 127) / 128 * 128);
}
static size_t half_bytes(int N, int K) { return (2 * (size_t)half_chunk(N, K) * (size_t)K + 255) & ~(size_t)255; }
// Calls that may use the copy, by size: all codecs without a producer of their own in kq_tile.cu - decode8<> makes a
// K-step's weights several times slower than the tensor cores use them - once the matrix outweighs the extra launch; q6_k
// with many rows (see launch_gemm), and whatever its size where its rows cannot be fetched there: beside the general kernel
// [763, 1024] x 53 16.2 -> 12.8 us, [3001, 1024] x 798 50 -> 23, 144 sizes up to 4 M weights 0.68 of the time on average (one of
// them, [2047, 256] x 2000, 1.10).
// With up to 256 rows and short K the lighter decoders keep up: q2_k [4096, 1024] x 128 13.7 / 16.6 us (x 300 22.0 / 19.7),
// iq4_xs 14.9 / 17.5, q4_0 17.4 / 17.4 there but [16384, 512] 17.8 / 19.8; q5_k and the others gain at every K.
static int half_min_k(int codec) {
  switch (codec) {
    case Q2_K: return 2560;
    case IQ4_XS: case IQ2_XXS: case IQ3_XXS: case IQ2_XS: case IQ2_S: case IQ1_S: case IQ1_M: return 1536;
    case Q4_0: case IQ4_NL: case MXFP4: return 1024;
  }
  return 0;
}
static bool use_half(int codec, long long M, int N, int K) {
  if (codec == Q6_K && !tile_rows_fit(codec, N, K)) return true;
  if (codec == Q4_K || (long long)N * K < (4ll << 20)) return false;
  if (codec == Q6_K && (K & 1023) == 0 && ((K & 2047) == 0 || (N & 1) == 0)) return M > 256;
  return M > 256 || K >= half_min_k(codec);
}
size_t gemm_workspace_bytes_n(int codec, int x_dtype, long long rows, int N, int K) {
  return gemm_workspace_bytes(x_dtype, rows, K) + (use_half(codec, rows, N, K) ? half_bytes(N, K) : 0);
}

cudaError_t launch_gemm(int codec, int x_dtype, const void* x, long long x_row_stride, void* y, long long y_row_stride,
                        const uint8_t* w, long long row_bytes, int M, int N, int K, void* workspace,
                        size_t workspace_bytes, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
  GemmArgs a;
  a.x = x;
  a.x_row_stride = x_row_stride;
  a.y = y;
  a.y_row_stride = y_row_stride;
  a.w = w;
  a.row_bytes = row_bytes;
  a.M = M;
  a.N = N;
  a.K = K;
  a.row_scale = nullptr;
  a.tiles = nullptr;
  a.n_tiles_dev = nullptr;
  a.w_expert_stride = 0;
  a.yrow = nullptr;
  if (x_dtype != F16) {
    __half* xh = static_cast<__half*>(workspace);
    float* rs = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + (((size_t)M * K * 2 + 255) & ~(size_t)255));
    cudaError_t e = launch_convert(x_dtype, x, x_row_stride, K, M, nullptr, nullptr, 1, 1, xh, rs, nullptr, nullptr, false, st);
    if (e != cudaSuccess) return e;
    a.x = xh;
    a.x_row_stride = K;
    a.row_scale = rs;
  }
  const bool out_half = x_dtype == F16;
  const size_t base = gemm_workspace_bytes(x_dtype, M, K);
  TileArgs t{};
  t.x = a.x;
  t.x_row_stride = a.x_row_stride;
  t.w = w;
  t.row_bytes = row_bytes;
  t.n_experts = 1;
  t.y = y;
  t.y_row_stride = y_row_stride;
  t.row_scale = a.row_scale;
  t.M = M;
  t.N = N;
  t.K = K;
  t.after_prepass = x_dtype != F16;
  // fp16 rows need no workspace: one that cannot hold the copy, for its size or its alignment, is left alone
  const bool room = use_half(codec, M, N, K) && workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0 &&
                    workspace_bytes >= base + half_bytes(N, K) &&
                    row_bytes == (long long)(K / kCodecs[codec].wpb) * kCodecs[codec].bpb;
  // q6_k with many rows: the producers cost more than dequantizing once (0.0009 cycles a weight). [14336, 4096] x 2048
  // 224 us fused, 208 by the copy; x 512 68 and 84.
  const bool fused = tile_supported(codec, w, row_bytes, N, K, 0) &&
                     !(codec == Q6_K && room &&
                       tile_cycles(codec, true, M, N, K) + 5000.0 + 0.0009 * N * K < tile_cycles(codec, false, M, N, K));
  if (fused) return launch_tile(codec, false, out_half, t, st);
  if (room) {
    uint8_t* wh = static_cast<uint8_t*>(workspace) + base;
    const int chunk = half_chunk(N, K);
    t.w = wh;
    t.row_bytes = 2ll * K;
    t.after_prepass = 1;
    for (int n0 = 0; n0 < N; n0 += chunk) {
      t.N = std::min(chunk, N - n0);
      cudaError_t e = launch_dequantize(codec, w + (long long)n0 * row_bytes, (long long)t.N * (K / kCodecs[codec].wpb), F16,
                                        wh, st);
      if (e != cudaSuccess) return e;
      t.y = static_cast<uint8_t*>(y) + 2ll * n0;
      if ((e = launch_tile(codec, true, out_half, t, st)) != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  const bool aligned = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  switch (codec) {
    case Q2_K: return launch_codec<Q2_K, 4>(out_half, a, aligned, st);
    case Q3_K: return launch_codec<Q3_K, 2>(out_half, a, aligned, st);
    case Q4_K: return launch_codec<Q4_K, 16>(out_half, a, aligned, st);
    case Q5_K: return launch_codec<Q5_K, 16>(out_half, a, aligned, st);
    case Q6_K: return launch_codec<Q6_K, 2>(out_half, a, aligned, st);
    case Q4_0: return launch_codec<Q4_0, 2>(out_half, a, aligned, st);
    case Q8_0: return launch_codec<Q8_0, 2>(out_half, a, aligned, st);
    case IQ4_NL: return launch_codec<IQ4_NL, 2>(out_half, a, aligned, st);
    case IQ4_XS: return launch_codec<IQ4_XS, 8>(out_half, a, aligned, st);
    case IQ2_XXS: return launch_codec<IQ2_XXS, 2>(out_half, a, aligned, st);
    case Q4_1: return launch_codec<Q4_1, 4>(out_half, a, aligned, st);
    case Q5_0: return launch_codec<Q5_0, 2>(out_half, a, aligned, st);
    case Q5_1: return launch_codec<Q5_1, 8>(out_half, a, aligned, st);
    case IQ3_XXS: return launch_codec<IQ3_XXS, 2>(out_half, a, aligned, st);
    case IQ3_S: return launch_codec<IQ3_S, 2>(out_half, a, aligned, st);
    case IQ2_XS: return launch_codec<IQ2_XS, 2>(out_half, a, aligned, st);
    case IQ2_S: return launch_codec<IQ2_S, 2>(out_half, a, aligned, st);
    case IQ1_S: return launch_codec<IQ1_S, 2>(out_half, a, aligned, st);
    case IQ1_M: return launch_codec<IQ1_M, 8>(out_half, a, aligned, st);
    case MXFP4: return launch_codec<MXFP4, 1>(out_half, a, aligned, st);
    case NVFP4: return launch_codec<NVFP4, 4>(out_half, a, aligned, st);
  }
  return cudaErrorInvalidValue;
}

// ------------------------------------------------------------------ grouped (MoE prefill)
// Row tiles of at most 256 expert-sorted rows; workspace pieces are laid out by the caller (kq_gather.cu).
template <int C, int NAT>
static cudaError_t launch_grouped_codec(bool out_half, const GemmArgs& a, bool aligned, int grid_y, cudaStream_t st) {
  if (out_half)
    return aligned ? launch_g<C, NAT, __half, 2>(a, st, grid_y) : launch_g<C, 1, __half, 2>(a, st, grid_y);
  return aligned ? launch_g<C, NAT, __nv_bfloat16, 2>(a, st, grid_y) : launch_g<C, 1, __nv_bfloat16, 2>(a, st, grid_y);
}

cudaError_t launch_gemm_grouped(int codec, int x_dtype, const void* x, int M, int K, const uint8_t* w,
                                long long expert_stride, long long row_bytes, int N, const uint32_t* lhs,
                                const int* order, long long rows_total, void* y, __half* xh, float* row_scale,
                                int* yrow, const void* tiles, const int* n_tiles_dev, int max_tiles,
                                int n_experts, int tile_rows, const int* n_valid_dev, cudaStream_t st) {
  if (rows_total <= 0 || N <= 0 || K <= 0) return cudaSuccess;
  cudaError_t e = launch_convert(x_dtype, x, K, K, rows_total, order, lhs, 1, M, xh, row_scale, yrow, n_valid_dev, false, st);
  if (e != cudaSuccess) return e;
  return launch_gemm_tiles(codec, x_dtype == F16, xh, rows_total, K, w, expert_stride, row_bytes, N, y,
                           x_dtype == F16 ? nullptr : row_scale, yrow, tiles, n_tiles_dev, max_tiles, n_experts, tile_rows,
                           true, st);
}

// The tile kernels over a device-built list of (expert, row_start, rows <= tile_rows) tiles: fp16 activations xh
// [rows_total, K] (dense), output row yrow[r] (or r when yrow == nullptr), y = out_half ? fp16 : bf16.
cudaError_t launch_gemm_tiles(int codec, bool out_half, const void* xh, long long rows_total, int K, const uint8_t* w,
                              long long expert_stride, long long row_bytes, int N, void* y, const float* row_scale,
                              const int* yrow, const void* tiles, const int* n_tiles_dev, int max_tiles, int n_experts,
                              int tile_rows, bool after_prepass, cudaStream_t st) {
  if (rows_total <= 0 || N <= 0 || K <= 0 || max_tiles <= 0) return cudaSuccess;
  if (max_tiles > 65535) return cudaErrorInvalidConfiguration;
  if (tile_supported(codec, w, row_bytes, N, K, expert_stride)) {
    TileArgs t{xh,   K,         w,    row_bytes, expert_stride,  n_experts, y, N, row_scale, yrow, (int)rows_total,
               N,    K,         static_cast<const GemmTile*>(tiles), n_tiles_dev, max_tiles, tile_rows,
               after_prepass};
    return launch_tile(codec, false, out_half, t, st);
  }
  // The list may hold up to max_tiles tiles but usually holds far fewer (an expert-parallel rank sizes it for all
  // ranks' rows and owns an eighth of them): a CTA without a tile still costs about 2 us of an SM (one CTA per
  // SM by shared memory), so the grid is capped and CTAs loop over the list when it is longer.
  if (max_tiles > kTileGridCap) max_tiles = kTileGridCap;
  GemmArgs a;
  a.x = xh;
  a.x_row_stride = K;
  a.y = y;
  a.y_row_stride = N;
  a.w = w;
  a.row_bytes = row_bytes;
  a.M = (int)rows_total;
  a.N = N;
  a.K = K;
  a.row_scale = row_scale;
  a.tiles = static_cast<const GemmTile*>(tiles);
  a.n_tiles_dev = n_tiles_dev;
  a.w_expert_stride = expert_stride;
  a.yrow = yrow;
  const bool aligned = (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (expert_stride & 15) == 0;
  switch (codec) {
    case Q2_K: return launch_grouped_codec<Q2_K, 4>(out_half, a, aligned, max_tiles, st);
    case Q3_K: return launch_grouped_codec<Q3_K, 2>(out_half, a, aligned, max_tiles, st);
    case Q4_K: return launch_grouped_codec<Q4_K, 16>(out_half, a, aligned, max_tiles, st);
    case Q5_K: return launch_grouped_codec<Q5_K, 16>(out_half, a, aligned, max_tiles, st);
    case Q6_K: return launch_grouped_codec<Q6_K, 2>(out_half, a, aligned, max_tiles, st);
    case Q4_0: return launch_grouped_codec<Q4_0, 2>(out_half, a, aligned, max_tiles, st);
    case Q8_0: return launch_grouped_codec<Q8_0, 2>(out_half, a, aligned, max_tiles, st);
    case IQ4_NL: return launch_grouped_codec<IQ4_NL, 2>(out_half, a, aligned, max_tiles, st);
    case IQ4_XS: return launch_grouped_codec<IQ4_XS, 8>(out_half, a, aligned, max_tiles, st);
    case IQ2_XXS: return launch_grouped_codec<IQ2_XXS, 2>(out_half, a, aligned, max_tiles, st);
    case Q4_1: return launch_grouped_codec<Q4_1, 4>(out_half, a, aligned, max_tiles, st);
    case Q5_0: return launch_grouped_codec<Q5_0, 2>(out_half, a, aligned, max_tiles, st);
    case Q5_1: return launch_grouped_codec<Q5_1, 8>(out_half, a, aligned, max_tiles, st);
    case IQ3_XXS: return launch_grouped_codec<IQ3_XXS, 2>(out_half, a, aligned, max_tiles, st);
    case IQ3_S: return launch_grouped_codec<IQ3_S, 2>(out_half, a, aligned, max_tiles, st);
    case IQ2_XS: return launch_grouped_codec<IQ2_XS, 2>(out_half, a, aligned, max_tiles, st);
    case IQ2_S: return launch_grouped_codec<IQ2_S, 2>(out_half, a, aligned, max_tiles, st);
    case IQ1_S: return launch_grouped_codec<IQ1_S, 2>(out_half, a, aligned, max_tiles, st);
    case IQ1_M: return launch_grouped_codec<IQ1_M, 8>(out_half, a, aligned, max_tiles, st);
    case MXFP4: return launch_grouped_codec<MXFP4, 1>(out_half, a, aligned, max_tiles, st);
    case NVFP4: return launch_grouped_codec<NVFP4, 4>(out_half, a, aligned, max_tiles, st);
  }
  return cudaErrorInvalidValue;
}

// Device address of the error word of the current device, for kernels of other translation units.
int* device_error_word() {
  static int* addr[16] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return nullptr;
  if (addr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_kq_device_error) != cudaSuccess) return nullptr;
    addr[dev] = static_cast<int*>(p);
  }
  return addr[dev];
}

// Flags raised by kernels that gave up on a bounded wait (0 = none). Synchronises the device.
cudaError_t read_device_error(int* out, bool clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_kq_device_error, sizeof(int));
  if (e == cudaSuccess && clear && *out != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_kq_device_error, &zero, sizeof(int));
  }
  return e;
}

}  // namespace kq
