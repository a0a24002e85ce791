// Two to sixteen dense activation rows of q4_k, q5_k, q6_k, iq4_xs: the products of kq_rows_unit.cuh (the integers as matrix
// operands, no weight rounded), each warp with a ring of its own.
//
// The kernel before (kq_rows.cu, which keeps the gathered rows) brought stages of all rows through producer warps with
// sixteen-byte copies and handed them to consumers over barriers: of its 8.7 million warp instructions for [14336, 4096] x 8
// q4_k less than half were products, and its 24 warps had 80 registers each. Here the sixteen warps of a CTA are all
// consumers. The units (tile of sixteen weight rows, superblock) are shared out evenly; a thread of the warp fetches a unit
// as one TMA box, several ahead; box rows are odd multiples of sixteen bytes, so four-byte and sixteen-byte reads of eight
// rows lie in different banks. (Rows of iq4_xs that are no whole sixteens come by sixteen-byte asynchronous copies of the
// same warp.) Activations are staged once per CTA, all of K, and with them the sums over sub-blocks that the offset and the
// mins need; where they do not fit, two CTAs share a row block, half of K each, and meet over distributed shared memory.
// Measured on B200, the kernels before and this one: q4_k [14336, 4096] x 4 15.5 -> 13.5 us, x 8 16.7 -> 14.1, x 16 21.5 ->
// 19.0; [28672, 8192] x 4 45.9 -> 35.5 (3.7 TB/s); q6_k [14336, 4096] x 8 22.3 -> 18.2; iq4_xs [28672, 8192] x 4 70.1 ->
// 38.8, in bf16 93 -> 38.8. What bounds it: short of bandwidth by staging (2.5 us) and one CTA per SM, whose prologue does
// not run beside the kernel before; the products of eight columns take 60 % of the issue slots of iq4_xs.
// Nothing is read ahead of griddepcontrol.wait: the weights may have been written by the kernel before.
#include <cuda.h>

#include <algorithm>
#include <cstdlib>

#include "kq_launch.h"
#include "kq_rows_unit.cuh"
#include "kq_tma_map.h"

namespace kq {

namespace {

constexpr int kFwWarps = 16, kFwThreads = 32 * kFwWarps, kFwSlots = 4;
constexpr int kFwSmem = 226 * 1024 - 256;
// bytes of a row in a slot: the superblock or the aligned window around it
__host__ __device__ constexpr int fw_pitch(int c) { return c == Q5_K ? 176 : (c == Q6_K ? 240 : 144); }

struct FewPlan {
  int R, n_blocks;          // weight rows of a row block, row blocks
  int rt;                   // row tiles of sixteen
  int D, share;             // slots of a warp, units of a warp at most
  int S;                    // CTAs of a cluster, a part of K each
  int red_pitch;
  // for the CTAs of a cluster and the row tiles: the first warp with units of the tile, the last (<< 8), and whether the
  // first has some of the tile before too (<< 16)
  int span[2][kFwWarps];
  int x_pitch, x_off, sum_off, red_off, smem;
};

// iq4_xs: a byte of quants is the levels of weights i and i + 16 of its sub-block. The 256 pairs, as 16-bit floats (small
// integers: exact in both types), stand in shared memory once per lane, 256 bytes apart, so that one byte permute makes an
// address - the byte above four times the lane - and a read has a bank of its own: 8 instructions for the operands of
// sixteen weights of a lane where byte permutes out of two tables took 40.
constexpr int kFwTable = 256 * 256;
template <typename XT>
__device__ __forceinline__ void fw_fill_table(uint8_t* tab) {
  static_assert(kFwThreads == 512, "two threads to an entry");
  // the levels plus 127, four to a word: a byte permute by the nibble
  constexpr uint32_t kL[4] = {0x3e2c1700u, 0x75695c4eu, 0xa5988c80u, 0xf0d8c4b4u};
  const uint32_t byte = threadIdx.x >> 1;
  auto level = [&](uint32_t nib) {
    const uint32_t v = __byte_perm(nib & 8 ? kL[2] : kL[0], nib & 8 ? kL[3] : kL[1], nib & 7) & 0xffu;
    return (float)(int)v - 127.f;
  };
  const float lo = level(byte & 15), hi = level(byte >> 4);
  uint32_t v;
  if constexpr (std::is_same<XT, __half>::value) {
    const __half2 h = __floats2half2_rn(lo, hi);
    v = *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    v = *reinterpret_cast<const uint32_t*>(&h);
  }
  uint4* out = reinterpret_cast<uint4*>(tab + byte * 256 + 64 * (threadIdx.x & 1));
#pragma unroll
  for (int i = 0; i < 4; i++) out[i] = make_uint4(v, v, v, v);
}
// RowsUnit::run of iq4_xs by that table (src/kquant_cpu_decode.cpp:557-584): weights 4 t .. 4 t + 3 and those 16 further
template <typename XT, int NT>
__device__ __forceinline__ void fw_run_iq4(float (&y)[NT][4], const uint8_t* r0, const uint8_t* r1, const uint8_t* (&xb)[NT],
                                           const uint8_t* tab, uint32_t lane4, int t) {
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
  auto pair = [&](uint32_t w, int i) {
    return *reinterpret_cast<const uint32_t*>(tab + __byte_perm(w, lane4, 0x5504u | (i << 4)));
  };
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const uint32_t wa = rw_lds(r0 + 8 + 16 * j + 4 * t), wb = rw_lds(r1 + 8 + 16 * j + 4 * t);
    uint32_t a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = pair(wa, i), b[i] = pair(wb, i);
    float c[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) {
      const uint2 v0 = *reinterpret_cast<const uint2*>(xb[n] + 64 * j + 8 * t);
      const uint2 v1 = *reinterpret_cast<const uint2*>(xb[n] + 64 * j + 32 + 8 * t);
      rw_mma0(c[n], a[0], b[0], a[1], b[1], __byte_perm(v0.x, v1.x, 0x5410), __byte_perm(v0.x, v1.x, 0x7632), XT());
      rw_mma(c[n], a[2], b[2], a[3], b[3], __byte_perm(v0.y, v1.y, 0x5410), __byte_perm(v0.y, v1.y, 0x7632), XT());
    }
    RowsUnit<IQ4_XS, XT, NT>::scale_add(acc, c, rw_byte(s0[j & 1], j >> 1, 8388640.f), rw_byte(s1[j & 1], j >> 1, 8388640.f));
  }
  RowsUnit<IQ4_XS, XT, NT>::finish(y, acc, __half2float(__ushort_as_half((unsigned short)h0.x)),
                                   __half2float(__ushort_as_half((unsigned short)h1.x)));
}

__device__ __forceinline__ void fw_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ float fw_ld_peer(const float* p, int rank) {
  uint32_t at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
  return v;
}

// TMA: the wire rows are whole sixteens
template <int C, typename XT, int NT, bool TMA, int S>
__global__ void __launch_bounds__(kFwThreads, 1)
few_kernel(const GemvArgs a, const FewPlan pl, const __grid_constant__ CUtensorMap map, int* __restrict__ error_word) {
  constexpr int BPB = bpb_of(C), kPitch = fw_pitch(C), kSlot = 16 * kPitch;
  constexpr bool kBf = std::is_same<XT, __nv_bfloat16>::value;
  constexpr bool kSums = rw_sums<C, kBf>();
  constexpr int kSumWords = NT * 8 * rw_sum_pitch(C);  // of a superblock
  extern __shared__ __align__(128) uint8_t fw_dyn[];
  __shared__ uint64_t full[kFwWarps][kFwSlots];
  __shared__ int abort_s;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int D = pl.D, M = a.M, red_pitch = pl.red_pitch;
  // this CTA's superblocks
  const int rank = (int)blockIdx.x % S, cluster = (int)blockIdx.x / S, clusters = (int)gridDim.x / S;
  auto first_sb = [&](int r) { return r * (a.K >> 8) / S; };
  const int sb0 = first_sb(rank), nsb = first_sb(rank + 1) - sb0;
  if (threadIdx.x == 0) abort_s = 0;
  if (TMA && lane == 0) {
    for (int d = 0; d < D; d++) mbar_init(&full[warp][d], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  volatile int* abort_flag = &abort_s;
  constexpr int kTab = C == IQ4_XS ? kFwTable : 0;  // (at the start: its addresses are constants)
  uint8_t* ring = fw_dyn + kTab + warp * D * kSlot;
  if constexpr (C == IQ4_XS) fw_fill_table<XT>(fw_dyn);
  // The units (tile, superblock) of a row block in equal contiguous shares: a warp's share touches two tiles at most.
  const int all = pl.rt * nsb, u0 = (warp * all) >> 4, u1 = ((warp + 1) * all) >> 4;
  const int my_blocks = (pl.n_blocks - 1 - cluster) / clusters + 1;
  const int units = (u1 - u0) * my_blocks;
  const uint8_t* wend = a.w + (long long)a.N * a.row_bytes;
  int is_u = 0, is_d = 0, is_blk = cluster, is_tile = u0 / nsb, is_sb = u0 - is_tile * nsb, is_left = u1 - u0;
  auto issue = [&]() {  // the next unit of this warp's share (of the next row block's)
    if (is_u < units) {
      const int row0 = is_blk * pl.R;
      uint8_t* slot = ring + is_d * kSlot;
      if constexpr (TMA) {
        if (lane == 0) {
          mbar_expect_tx(&full[warp][is_d], kSlot);
          fw_load(smem_u32(slot), &map, ((sb0 + is_sb) * BPB) & ~15, row0 + 16 * is_tile, &full[warp][is_d]);
        }
      } else {
        constexpr int P = kPitch / 16;
#pragma unroll
        for (int i = 0; i < (16 * P + 31) / 32; i++) {
          const int j = lane + 32 * i, r = j / P, piece = j - r * P;
          if (r >= 16) continue;
          const int row = min(row0 + 16 * is_tile + r, a.N - 1);
          const uint8_t* src = reinterpret_cast<const uint8_t*>(
                                   reinterpret_cast<uintptr_t>(a.w + (long long)row * a.row_bytes + (sb0 + is_sb) * BPB) & ~(uintptr_t)15) +
                               16 * piece;
          const long long left = wend - src;
          if (left >= 16) rw_cp16(smem_u32(slot + 16 * j), src);
          else if (left > 0) rw_cp16_upto(smem_u32(slot + 16 * j), src, (int)left);
        }
      }
      is_u++;
      if (++is_d == D) is_d = 0;
      if (++is_sb == nsb) is_sb = 0, is_tile++;
      if (--is_left == 0) is_blk += clusters, is_tile = u0 / nsb, is_sb = u0 - is_tile * nsb, is_left = u1 - u0;
    }
    if constexpr (!TMA) asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  uint8_t* const xs = fw_dyn + pl.x_off;
  {
    const int per_row = 32 * nsb;  // pieces of sixteen bytes
    const uint32_t dst = smem_u32(xs);
    const XT* src = static_cast<const XT*>(a.x) + 256 * sb0;
    for (int m = 0; m < M; m++)
      for (int c = threadIdx.x; c < per_row; c += kFwThreads) rw_cp16(dst + m * pl.x_pitch + 16 * c, src + m * a.x_row_stride + 8 * c);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  // (after the activations, which would wait behind them: [14336, 4096] x 4 15.1 us the other way, 14.5 so)
  for (int d = 0; d < D; d++) issue();  // (ragged rows: a group of copies each)
  // this thread's first output: its place in the row block, its column
  const int places = pl.rt * 16, e0 = (int)threadIdx.x + kFwThreads * rank;
  const int c0 = e0 / places, place0 = e0 - c0 * places;
  const int c_step = kFwThreads * S / places, place_step = kFwThreads * S - c_step * places;
  if constexpr (TMA) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  else if (D == 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  else if (D == 2) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
  else if (D == 3) asm volatile("cp.async.wait_group 3;\n" ::: "memory");
  else asm volatile("cp.async.wait_group 4;\n" ::: "memory");
  __syncthreads();  // the activations have landed
  float* sums = reinterpret_cast<float*>(fw_dyn + pl.sum_off);
  if constexpr (kSums) {
    for (int e = warp; e < nsb * NT; e += kFwWarps) {
      const int k = e / NT, n = e % NT;
      if (8 * n < M)
        rows_sums<C, XT>(xs + min(8 * n + g, M - 1) * pl.x_pitch + 512 * k, sums + (k * NT + n) * 8 * rw_sum_pitch(C), lane);
    }
    __syncthreads();
  }

  float* red = reinterpret_cast<float*>(fw_dyn + pl.red_off);  // [warp][its first tile, its second][16][red_pitch]
  auto meet = [&]() {
    if (S == 1) __syncthreads();
    else
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  };
  int d = 0;
  uint32_t par = 0;
  bool ok = true;
  for (int b = 0; b < my_blocks; b++) {
    const int row0 = (cluster + b * clusters) * pl.R, rows = min(pl.R, a.N - row0);
    float y[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) y[n][0] = y[n][1] = y[n][2] = y[n][3] = 0.f;
    int tile = u0 / nsb, sb = u0 - tile * nsb, second = 0;
    auto flush = [&]() {
      float* mine = red + ((2 * warp + second) * 16 + g) * red_pitch + 2 * t;
#pragma unroll
      for (int n = 0; n < NT; n++)
        if (8 * n + 2 * t < M) {
          *reinterpret_cast<float2*>(mine + 8 * n) = make_float2(y[n][0], y[n][1]);
          *reinterpret_cast<float2*>(mine + 8 * red_pitch + 8 * n) = make_float2(y[n][2], y[n][3]);
        }
    };
    for (int u = u0; u < u1; u++) {
      if constexpr (TMA) {
        if (ok) ok = mbar_wait_err(&full[warp][d], par, abort_flag, 0x400, error_word);
      } else {  // this unit's group: D - 1 younger ones
        if (D == 1) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        else if (D == 2) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else if (D == 3) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 3;\n" ::: "memory");
        __syncwarp();
      }
      if (ok) {
        const uint8_t* slot = ring + d * kSlot;
        int p0 = 0, p1 = 0;  // places of the superblock in the rows' windows
        if constexpr (!rw_al16(C)) {
          if constexpr (TMA) {
            p0 = p1 = ((sb0 + sb) * BPB) & 15;
          } else {
            p0 = (int)(((long long)(row0 + 16 * tile + g) * a.row_bytes + (long long)(sb0 + sb) * BPB) & 15);
            p1 = (int)(((long long)(row0 + 16 * tile + g + 8) * a.row_bytes + (long long)(sb0 + sb) * BPB) & 15);
          }
        }
        const uint8_t* xb[NT];
#pragma unroll
        for (int n = 0; n < NT; n++) xb[n] = xs + min(8 * n + g, M - 1) * pl.x_pitch + 512 * sb;
        const uint8_t *r0 = slot + g * kPitch + p0, *r1 = slot + (g + 8) * kPitch + p1;
        if constexpr (C == IQ4_XS) fw_run_iq4<XT, NT>(y, r0, r1, xb, fw_dyn, 4 * lane, t);
        else RowsUnit<C, XT, NT>::run(y, r0, r1, xb, sums + sb * kSumWords, g, t);
      }
      __syncwarp();  // the slot has been read
      issue();
      if (++d == D) d = 0, par ^= 1;
      if (++sb == nsb && u + 1 < u1) {
        flush();
        sb = 0, tile++, second = 1;
#pragma unroll
        for (int n = 0; n < NT; n++) y[n][0] = y[n][1] = y[n][2] = y[n][3] = 0.f;
      }
    }
    flush();
    meet();
    // the shares of a tile meet in a fixed order, in one of the cluster's CTAs
    if (abort_s == 0) {
      for (int place = place0, c = c0; c < M;) {
        const int tl = place >> 4, r = place, at_place = place & 15, at_c = c;
        place += place_step, c += c_step;
        if (place >= places) place -= places, c++;
        if (r >= rows) continue;
        float v = 0.f;
        for (int q = 0; q < S; q++) {
          const int sp = pl.span[q][tl], to = (sp >> 8) & 0xff;
          const float* at = red + ((2 * (sp & 0xff) + (sp >> 16)) * 16 + at_place) * red_pitch + at_c;
          for (int w = sp & 0xff; w <= to; w++) {
            // (a warp without a unit has left zeros)
            v += S == 1 ? *at : fw_ld_peer(at, q);
            at = red + ((2 * w + 2) * 16 + at_place) * red_pitch + at_c;
          }
        }
        if (!(fabsf(v) < INFINITY))
          v = rows_plain<C, XT>(a.w + (long long)(row0 + r) * a.row_bytes, static_cast<const XT*>(a.x) + at_c * a.x_row_stride,
                                a.K >> 8);
        if (a.row_scale != nullptr) v *= a.row_scale[at_c];
        const long long o = (long long)at_c * a.y_row_stride + row0 + r;
        if (kBf || a.out_bf16) static_cast<__nv_bfloat16*>(a.y)[o] = __float2bfloat16_rn(v);
        else static_cast<__half*>(a.y)[o] = __float2half_rn(v);
      }
    }
    if (S > 1 || b + 1 < my_blocks) meet();
  }
  if constexpr (TMA) {
    if (abort_s != 0) {  // given up: what is in flight lands long before this
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 1000000ull) {
      }
    }
  } else {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  }
}

int fw_sm_count() {
  static int sms[16] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 0;
  if (sms[dev] == 0 && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  return sms[dev];
}

// Row blocks as even as the SM count allows, one per SM and pass; false where the activations, their sums and a slot a warp
// do not fit.
template <int C, bool BF, int NT>
bool few_plan(const GemvArgs& a, int S, FewPlan& p) {
  const int sms = fw_sm_count(), clusters = sms / S;
  if (clusters <= 0 || (a.K >> 8) < S) return false;
  const int nsb = ((a.K >> 8) + S - 1) / S;
  const int passes = (a.N + clusters * 16 * kFwWarps - 1) / (clusters * 16 * kFwWarps);
  p.S = S;
  p.R = std::max(8, (a.N + clusters * passes - 1) / (clusters * passes));
  p.n_blocks = (a.N + p.R - 1) / p.R;
  p.rt = (p.R + 15) / 16;
  p.x_pitch = nsb * 512 + (rw_al16(C) ? 64 : 32);  // 16- and 8-byte reads of the B operand in different banks
  p.red_pitch = ((a.M + 1) & ~1) + 2;
  const int table = C == IQ4_XS ? kFwTable : 0, red = kFwWarps * 2 * 16 * p.red_pitch * 4;
  const int x = (a.M * p.x_pitch + 127) & ~127, sum = rw_sums<C, BF>() ? nsb * NT * 8 * rw_sum_pitch(C) * 4 : 0;
  p.share = ((p.rt * nsb + kFwWarps - 1) / kFwWarps) * ((p.n_blocks + clusters - 1) / clusters);
  const int room = kFwSmem - table - x - sum - red, slots = kFwWarps * 16 * fw_pitch(C);
  if (room < slots) return false;
  p.D = std::min({kFwSlots, p.share, room / slots});
  p.x_off = table + p.D * slots;
  p.sum_off = p.x_off + x;
  p.red_off = p.sum_off + sum;
  p.smem = p.red_off + red;
  for (int q = 0; q < S; q++)
    for (int t = 0; t < p.rt; t++) {
      const int n = (q + 1) * (a.K >> 8) / S - q * (a.K >> 8) / S, of = p.rt * n;
      const int from = ((t * n + 1) * kFwWarps - 1) / of, to = ((t + 1) * n * kFwWarps - 1) / of;
      p.span[q][t] = from | (to << 8) | ((from * of) / kFwWarps < t * n ? 1 << 16 : 0);
    }
  return true;
}

template <int C, typename XT, int NT, bool TMA, int S>
cudaError_t launch_few_t(const GemvArgs& a, const FewPlan& p, cudaStream_t st) {
  auto kern = few_kernel<C, XT, NT, TMA, S>;
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwSmem);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  int* err = device_error_word();
  if (err == nullptr) return cudaErrorUnknown;
  alignas(64) CUtensorMap map{};
  if (TMA) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (enc == nullptr) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)a.row_bytes, (cuuint64_t)a.N};
    const cuuint64_t strides[1] = {(cuuint64_t)a.row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)fw_pitch(C), 16u};
    const cuuint32_t estr[2] = {1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(a.w), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.S * std::min(p.n_blocks, fw_sm_count() / p.S));
  cfg.blockDim = dim3(kFwThreads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.S, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
  cfg.numAttrs = p.S > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, a, p, map, err);
}

template <int C, typename XT, int NT>
cudaError_t launch_few_nt(const GemvArgs& a, cudaStream_t st) {
  constexpr bool kBf = std::is_same<XT, __nv_bfloat16>::value;
  FewPlan p;
  // One CTA to a row block where it keeps enough units in flight, and the longer units of q6_k want a third with long K:
  // [4096, 14336] x 2 20.9 us with two slots, 18.2 as a pair of CTAs with four; q5_k [8192, 8192] x 8 19.4 with one slot,
  // 17.4 as a pair. A pair costs 1 to 2.5 us in staging and in the meeting (q4_k [4096, 4096] x 2, x 8); with two column
  // tiles one slot is enough (q4_k [4096, 4096] x 16 12.3 -> 9.6), and a pair pays from K of 8192 on (q4_k x 16 [8192, 8192]
  // 23.5 -> 22.0; [5120, 5120] 13.1 against 15.4), with iq4_xs always.
  const bool one = few_plan<C, kBf, NT>(a, 1, p) &&
                   (NT > 1 || p.D >= std::min(p.share, C == Q6_K && a.K >= 8192 ? 3 : 2));
  if (!one && (!few_plan<C, kBf, NT>(a, 2, p) || (NT > 1 && C != IQ4_XS && a.K < 8192)))
    return cudaErrorNotSupported;  // (nothing launched)
  if constexpr (C == IQ4_XS)
    if ((a.row_bytes & 15) != 0)
      return p.S == 1 ? launch_few_t<C, XT, NT, false, 1>(a, p, st) : launch_few_t<C, XT, NT, false, 2>(a, p, st);
  return p.S == 1 ? launch_few_t<C, XT, NT, true, 1>(a, p, st) : launch_few_t<C, XT, NT, true, 2>(a, p, st);
}

template <int C, typename XT>
cudaError_t launch_few_c(const GemvArgs& a, cudaStream_t st) {
  return a.M <= 8 ? launch_few_nt<C, XT, 1>(a, st) : launch_few_nt<C, XT, 2>(a, st);
}
template <typename XT>
cudaError_t launch_few_x(int codec, const GemvArgs& a, cudaStream_t st) {
  switch (codec) {
    case Q4_K: return launch_few_c<Q4_K, XT>(a, st);
    case Q5_K: return launch_few_c<Q5_K, XT>(a, st);
    case Q6_K: return launch_few_c<Q6_K, XT>(a, st);
    case IQ4_XS: return launch_few_c<IQ4_XS, XT>(a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

bool gemv_few_supported(int codec, int x_dtype, const GemvArgs& a) {
  if (codec != Q4_K && codec != Q5_K && codec != Q6_K && codec != IQ4_XS) return false;
  // (half of a longer row would not fit into shared memory, and few_plan counts bytes in int)
  if (!(x_dtype == F16 || x_dtype == BF16) || a.tasks != nullptr || a.bias != nullptr || a.M < 1 || a.M > 16 || a.N < 8 ||
      a.K < 256 || a.K > (1 << 18) || (a.K & 255) != 0 || a.w_align16 == 0 || a.row_bytes != (long long)(a.K >> 8) * bpb_of(codec))
    return false;
  if ((reinterpret_cast<uintptr_t>(a.x) & 15) != 0 || (a.x_row_stride & 7) != 0) return false;
  const long long size = (long long)a.N * a.K;
  // iq4_xs, against the table kernel with its K split and, up to 4 M weights, kq_rows.cu: one row [28672, 8192] 50 -> 38 us,
  // [1024, 4096] 4.0 -> 3.9, [1536, 2048] 3.2 against 3.8; sixteen rows [4096, 2048] 13 -> 7, [1024, 4096] 7.2 against 8.9.
  if (codec == IQ4_XS) return size > (4ll << 20) || (a.K >= 4096 && a.M <= 8);
  // The others, against kq_rows.cu (one row: kq_gemv_one.cu). Every CTA stages all activations and clears its sums, which
  // short rows do not pay for: q4_k x 8 [1024, 4096] 5.6 -> 5.3, [4096, 2048] 5.1 and 5.1, [3072, 3072] 6.0 against 6.4;
  // with many of them [40000, 1024] 15.4 -> 14.3.
  if (a.M < 2 || (a.row_bytes & 15) != 0 || !(a.K >= 4096 || (a.K >= 1024 && size >= (36ll << 20)))) return false;
  // and the row block has to fill its tiles, for the codec with the least bytes: [5120, 5120] x 8 10.1 against 10.3
  const int sms = fw_sm_count(), R = sms > 0 ? (a.N + sms - 1) / sms : 0;
  return codec != Q4_K || R <= 16 || R >= 64 || 4 * R >= 3 * ((R + 15) & ~15);
}

cudaError_t launch_gemv_few(int codec, int x_dtype, const GemvArgs& a, cudaStream_t st) {
  return x_dtype == F16 ? launch_few_x<__half>(codec, a, st) : launch_few_x<__nv_bfloat16>(codec, a, st);
}

}  // namespace kq
