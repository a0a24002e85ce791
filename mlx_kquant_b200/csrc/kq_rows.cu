// Decode product of a few activation rows: y[M, N] = x[M, K] . dequant(W)^T for 1 <= M <= 16, on mma.sync with the
// quantized integers themselves as the A operand (sixteen weight rows x sixteen weights an instruction; the products are in
// kq_rows_unit.cuh), the
// activations in their own 16-bit type as the B operand, float32 accumulation. Reference: qmv_fused_rows,
// src/kquant_cpu_decode.cpp:1032-1065.
//
// What bounds it: a tile product is a chain of shared-memory loads, permutes and matrix instructions some 2500 cycles
// long, with 16 warps on an SM to hide it (without any weight copy [28672, 8192] x 1 row takes 40 of 48 us; without any
// product 26), half of the issue slots and half of the ALU pipe (byte permutes) busy; HBM is the next bound. Measured
// q5_k [14336, 4096] x 16 fp16 rows 22.1 us, q4_k [3072, 3072] x 8 6.0, q6_k [5120, 5120] x 8 16.8. Most dense products with
// K from 4096 on are in kq_few.cu, which says why; here are shorter rows, q6_k in rows that are no whole sixteens,
// activations that do not fit there, and all gathered rows. (The products are in kq_rows_unit.cuh.) What it is built around:
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
#include "kq_launch.h"
#include "kq_rows_unit.cuh"
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

// gather_qmm: entry i multiplies activation row lhs[i] by matrix rhs[i]; grid.y counts the matrices, or (by_entry,
// fewer entries than matrices) the entries, of which the first of every matrix does the work for all. Routing may be
// uneven: a CTA makes at most `deep` passes over its matrix, and CTAs of y >= units take what is left (rows_left_over).
struct RowsGather {
  const uint32_t *lhs, *rhs;
  int n_entries, n_experts, by_entry;
  long long x_batch, expert_stride;
  int units, deep;
  int early;  // the weights of a CTA's first stages are fetched while it looks for its entries
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
  auto row_block = [&](int pass) { return ((int)blockIdx.x + (G ? 0 : pass * (int)gridDim.x)) * pl.R; };
  // A row's pieces of sixteen bytes go to neighbouring threads (a power of two of them, 1 << wlog: pl.wlog, pl.xlog),
  // every thread walks down the rows: two additions a piece (numbering the pieces of a stage and
  // stepping by the thread count instead: q6_k [4096, 14336] x 8 32 us against 24).
  const int tid = (warp - NW - kRwHelpers) * 32 + lane;  // of the producers
  constexpr int kThreads = 32 * kRwProducers;
  int pass_w = 0, st_w = 0, slot_w = 0;
  auto copy_w = [&]() {
    const int row0 = row_block(pass_w), rows = min(pl.R, a.N - row0), len = min(pl.cs, nsb - st_w * pl.cs) * BPB;
    const int step = kThreads >> pl.wlog, r0 = tid >> pl.wlog;
    const uint8_t* wend = wmat + (long long)a.N * a.row_bytes;
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
  int early = 0;  // stages whose weights are on their way already
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
    wmat += (long long)e * ga.expert_stride;
    if (ga.early && !left_over) {  // (between the loads of the indices and their use: q6_k 0.6 us slower)
      early = min(S, nst);
      if (warp >= NW + kRwHelpers)
        for (int i = 0; i < early; i++) copy_w();
    }
    if (threadIdx.x == 0) walk_s = make_int2(pass0, pass_step);
    const bool shared = ga.by_entry || share > 1 || left_over;
    const int total_m = collect_entries<TH>(ga.rhs, ga.lhs, ga.n_entries, ga.x_batch, e, list, &count_s,
                                            shared ? 0 : (more ? 8 * NT * base : ga.n_entries), [] {});
    if (total_m == 0 || (ga.by_entry && !left_over && list[0].y != (int)blockIdx.y)) {
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      return;
    }
    passes = ((total_m + 8 * NT - 1) / (8 * NT) - pass0 + pass_step - 1) / pass_step;
    if (more) passes = min(passes, ga.deep);
    if (passes <= 0) {
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      return;
    }
  } else {
    passes = (pl.n_blocks - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;
  }
  auto entry0 = [&](int pass) { return 8 * NT * (walk_s.x + pass * walk_s.y); };  // of the pass (gather)
  auto rows_of_x = [&](int pass) { return G ? min(8 * NT, count_s - entry0(pass)) : a.M; };
  volatile int* abort_flag = &abort_s;
  auto wait = [&](uint64_t* bar, int parity) { return mbar_wait_err(bar, parity, abort_flag, 0x100, error_word); };

  if (warp >= NW + kRwHelpers) {
    // ================= producers =================
    const int total = passes * nst;
    int pass_x = 0, st_x = 0, slot_x = 0;
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
    for (int i = early; i < first; i++) copy_w();
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
  // 64 matrices [128, 512] of q6_k, eight entries each 7.6 -> 7.2 us, q4_k 5.9 -> 5.4 (with fewer entries a matrix some have
  // none, whose weights would be fetched for nothing)
  gl.early = !ga.by_entry && ga.n_entries >= 4 * ga.n_experts ? 1 : 0;
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
  // iq4_xs: the permutes for its levels (23 instructions for eight weights against 7 of the others) bound it on large
  // matrices: [1000, 1280] x 2 rows 10.3 -> 3.6 us, but [14336, 4096] 22.7 against 28.9 (kq_few.cu has them from a table)
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
