// quantized_matmul with transpose == 0: W is [K, N / weights_per_block * bytes_per_block], every one of its
// K rows a quantized vector of N weights, and y[m, n] = sum_k x[m, k] * dequant(W)[k, n]
// (src/kquant_ops.cpp:140-155; the reference's qvm / qmm_n Metal kernels, src/kquant_matmul.cpp:705-751, and on
// the CPU dequantize-then-GEMM, src/kquant_cpu_decode.cpp:1299-1352). A rarely used orientation (the layers
// of the reference's own models keep [N, K] weights), served by one streaming CUDA-core kernel:
// a CTA owns 256 output columns and a slice of K; its eight warps take the slice's rows in turn, lane j
// decodes the eight weights 8 j .. 8 j + 7 of the row's 256-column chunk in fp32 (decode8, the dequantize
// kernel's arithmetic) and multiplies them by up to four activations x[m, k]; warps meet in shared memory,
// K slices (a cluster of up to 8 CTAs) through distributed shared memory. More than four rows are
// further passes over the weights (grid.z): correct for any M, efficient for decode-sized M only.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_launch.h"

namespace cg = cooperative_groups;

namespace kq {

namespace {

constexpr int kWarps = 8, kThreads = 256, kMT = 4, kMaxSplit = 8, kCols = 256;

struct QvmGather {
  const uint32_t* lhs;
  const uint32_t* rhs;   // nullptr = dense call
  long long entry0, x_batch, expert_stride;
  int n_experts, m_tiles;
};

template <typename XT>
__device__ __forceinline__ float load_x(const XT* p) {
  if constexpr (std::is_same<XT, __half>::value) return __half2float(*p);
  else if constexpr (std::is_same<XT, __nv_bfloat16>::value) return __bfloat162float(*p);
  else return __bfloat162float(__float2bfloat16_rn(*p));  // float rows are rounded to bf16 first, as the op does
}

template <int C, int A, typename XT>
__global__ void __launch_bounds__(kThreads)
qvm_kernel(const XT* __restrict__ x, long long x_row_stride, void* __restrict__ y, long long y_row_stride,
           const uint8_t* __restrict__ w, long long row_bytes, int M, int N, int K, QvmGather gq) {
  using OT = typename std::conditional<std::is_same<XT, __half>::value, __half, __nv_bfloat16>::type;
  constexpr int WPB = wpb_of(C), BPB = bpb_of(C);
  __shared__ float red[kWarps][kMT][kCols];
  __shared__ float part[kMT][kCols];
  __shared__ __align__(16) uint8_t s_tabs[(C == IQ4_NL || C == IQ4_XS || C == IQ2_XXS) ? kIqSmemBytes : 16];
  cg::cluster_group cluster = cg::this_cluster();
  IqTables tabs = global_iq_tables();
  if constexpr (C == IQ4_NL || C == IQ4_XS || C == IQ2_XXS) {
    tabs = stage_iq_tables(s_tabs, threadIdx.x, kThreads);
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int S = gridDim.y, slice = blockIdx.y;
  const int c0 = blockIdx.x * kCols + 8 * lane;  // this lane's eight output columns
  int mtile = blockIdx.z;
  if (gq.rhs != nullptr) {
    // gather form: grid.z = entries x row tiles; entry e multiplies x[lhs[e]] ([M, K]) by matrix rhs[e] into y[e].
    // An index out of range leaves the entry's rows unwritten (uniform over the cluster, which spans grid.y only).
    const long long e = gq.entry0 + blockIdx.z / gq.m_tiles;
    mtile = blockIdx.z % gq.m_tiles;
    const uint32_t l = gq.lhs[e], r = gq.rhs[e];
    if (r >= (uint32_t)gq.n_experts || (long long)l >= gq.x_batch) return;
    x += (long long)l * M * x_row_stride;
    w += (long long)r * gq.expert_stride;
    y = static_cast<OT*>(y) + e * M * y_row_stride;
  }
  const int m0 = mtile * kMT, m = min(kMT, M - m0);
  const int per = (K + S - 1) / S;
  const int k0 = min(slice * per, K), k1 = min(k0 + per, K);

  float acc[kMT][8];
#pragma unroll
  for (int t = 0; t < kMT; t++)
#pragma unroll
    for (int i = 0; i < 8; i++) acc[t][i] = 0.f;
  // this lane's eight columns: 256 blockIdx.x + 8 lane .. + 7
  const long long blk_off = block_of<C>(256ll * blockIdx.x + 8 * lane) * BPB;
  const int oct = octet_of<C>(8 * lane);
  if (c0 < N) {
    for (int k = k0 + warp; k < k1; k += kWarps) {
      float v[8];
      decode8<C, A>(w + (long long)k * row_bytes + blk_off, oct, v, tabs);
#pragma unroll
      for (int t = 0; t < kMT; t++) {
        if (t < m) {
          const float xv = load_x<XT>(x + (long long)(m0 + t) * x_row_stride + k);
#pragma unroll
          for (int i = 0; i < 8; i++) acc[t][i] = fmaf(xv, v[i], acc[t][i]);
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < kMT; t++)
#pragma unroll
    for (int i = 0; i < 8; i++) red[warp][t][8 * lane + i] = acc[t][i];
  __syncthreads();
  for (int idx = threadIdx.x; idx < kMT * kCols; idx += kThreads) {
    const int t = idx / kCols, c = idx % kCols;
    float s = 0.f;
#pragma unroll
    for (int wv = 0; wv < kWarps; wv++) s += red[wv][t][c];
    part[t][c] = s;
  }
  cluster.sync();  // every K slice's partial sums are in its shared memory
  const float* peer[kMaxSplit];
#pragma unroll
  for (int s = 0; s < kMaxSplit; s++) peer[s] = s < S ? cluster.map_shared_rank(&part[0][0], s) : &part[0][0];
  for (int idx = slice + S * threadIdx.x; idx < kMT * kCols; idx += S * kThreads) {
    const int t = idx / kCols, c = blockIdx.x * kCols + idx % kCols;
    if (t < m && c < N) {
      float sum = 0.f;
#pragma unroll
      for (int s = 0; s < kMaxSplit; s++)
        if (s < S) sum += peer[s][idx];
      OT* out = static_cast<OT*>(y) + (long long)(m0 + t) * y_row_stride + c;
      if constexpr (std::is_same<OT, __half>::value) *out = __float2half_rn(sum);
      else *out = __float2bfloat16_rn(sum);
    }
  }
  cluster.sync();  // peers may still be reading this CTA's partial sums
}

// The gather form for calls whose entries share matrices (absorbed attention: every sequence multiplies by the head's
// matrix): a CTA owns one matrix and 128 output columns, collects the matrix's entries from the index arrays by itself
// and multiplies up to eight of them per pass over the weights, so a weight is decoded once for eight rows where the
// kernel above decodes it for each. Up to 256 rows of the weights are copied to shared memory as the aligned windows
// around their bytes while the entries are looked for and the activations come (decoded from global memory, they were
// waited for once more each four rows, and one byte at a time where a row is no whole sixteens). A warp's halves take two
// rows of W at a time, a lane eight columns; the partial sums meet by one shuffle and in shared memory. Bound by the
// decode arithmetic (a third of the issue slots) and the chain index - activation - product; 64 heads [128, 512] q6_k,
// eight rows each: 9.1 -> 7.05 us a launch (the kernel above 39.6), q8_0 7.9 -> 6.5, 8 heads [512, 2048] q6_k 20.7 -> 18.4.
constexpr int kRowCols = 128, kRowM = 8;
constexpr int kRowEntries = 512;  // every CTA looks through all entries
constexpr int kRowChunk = 256;    // rows of W in shared memory at once
constexpr int kRowXPitch = 12;    // floats of a row of x in shared memory, by columns: stores of 32 k in eight banks
// bytes of a row's blocks in shared memory: 128 columns' and the aligned window around them
__host__ __device__ constexpr int row_pitch(int c) { return (std::max(1, kRowCols / wpb_of(c)) * bpb_of(c) + 30) / 16 * 16; }
constexpr int kRowFixed = kRowChunk * kRowXPitch * 4 + kWarps * kRowM * kRowCols * 4 + kRowEntries * 8;
template <int C, int A, typename XT>
__global__ void __launch_bounds__(kThreads, 2)
qvm_rows_kernel(const XT* __restrict__ x, void* __restrict__ y, const uint8_t* __restrict__ w, long long row_bytes,
                int N, int K, QvmGather gq, int n_entries) {
  using OT = typename std::conditional<std::is_same<XT, __half>::value, __half, __nv_bfloat16>::type;
  constexpr int BPB = bpb_of(C), kPitch = row_pitch(C);
  constexpr bool kIq = (C == IQ4_NL || C == IQ4_XS || C == IQ2_XXS);
  extern __shared__ __align__(16) uint8_t qr_dyn[];
  float (*xs)[kRowXPitch] = reinterpret_cast<float (*)[kRowXPitch]>(qr_dyn);  // activations of a K chunk
  float (*red)[kRowM][kRowCols] = reinterpret_cast<float (*)[kRowM][kRowCols]>(qr_dyn + kRowChunk * kRowXPitch * 4);
  int2* list = reinterpret_cast<int2*>(qr_dyn + kRowFixed - kRowEntries * 8);  // (row of x, row of y)
  uint8_t* ws = qr_dyn + kRowFixed;
  __shared__ __align__(16) uint8_t s_tabs[kIq ? kIqSmemBytes : 16];
  __shared__ int count_s;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  IqTables tabs = global_iq_tables();
  if constexpr (kIq) tabs = stage_iq_tables(s_tabs, threadIdx.x, kThreads);
  if (threadIdx.x == 0) count_s = 0;
  __syncthreads();
  const uint32_t e = blockIdx.y;
  w += (long long)e * gq.expert_stride;
  const int first = (int)block_of<C>(blockIdx.x * kRowCols);  // block of the CTA's first column
  const int len = min(std::max(1, kRowCols / wpb_of(C)), N / wpb_of(C) - first) * BPB;
  const uint8_t* wcols = w + (long long)first * BPB;
  const uint32_t place = (uint32_t)reinterpret_cast<uintptr_t>(wcols);
  auto stage = [&](int kb, int kn) {
    const uint8_t* wend = w + (long long)K * row_bytes;
    constexpr int P = kPitch / 16;
    for (int i = threadIdx.x; i < kn * P; i += kThreads) {
      const int r = i / P, c = i - r * P;
      const uint8_t* p = wcols + (long long)(kb + r) * row_bytes;
      const int ph = (int)(reinterpret_cast<uintptr_t>(p) & 15);
      const uint8_t* q = p - ph + 16 * c;
      const long long left = wend - q;
      const int bytes = left < 16 ? (int)left : 16;
      if (16 * c < len + ph)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(ws + 16 * i)), "l"(q), "r"(bytes) : "memory");
    }
  };
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int count = collect_entries<kThreads>(gq.rhs, gq.lhs, n_entries, gq.x_batch, e, list, &count_s,
                                              gridDim.z > 1 ? 0 : n_entries, [&]() { stage(0, min(kRowChunk, K)); });
  if (count == 0) {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    return;
  }

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, oc = lane & 15;
  const int c0 = blockIdx.x * kRowCols + 8 * oc;
  const bool live = c0 < N;  // N is a whole number of blocks: eight columns exist or none
  const int blk_off = live ? ((int)block_of<C>(c0) - first) * BPB : 0;
  const int oct = octet_of<C>(live ? c0 : 0);
  int staged = 0;  // the chunk in shared memory
  for (int e0 = kRowM * blockIdx.z; e0 < count; e0 += kRowM * gridDim.z) {  // grid.z CTAs share the entries
    const int m = min(kRowM, count - e0);
    float acc[kRowM][8];
#pragma unroll
    for (int t = 0; t < kRowM; t++)
#pragma unroll
      for (int i = 0; i < 8; i++) acc[t][i] = 0.f;
    for (int kb = 0; kb < K; kb += kRowChunk) {
      const int kn = min(kRowChunk, K - kb);
      __syncthreads();  // the chunk before (and the sums of the pass before) have been read
      if (kb != staged) stage(kb, kn);
      staged = kb;
      static_assert(kRowM == kWarps, "a row of x to a warp");
      const XT* xr = x + (long long)list[e0 + min(warp, m - 1)].x * K + kb;
#pragma unroll 4
      for (int k = lane; k < kn; k += 32) xs[k][warp] = warp < m ? load_x<XT>(xr + k) : 0.f;
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();
#pragma unroll 4
      for (int k = 2 * warp + half; k < kn; k += 2 * kWarps) {
        float v[8];
        const int ph = (place + (uint32_t)(kb + k) * (uint32_t)row_bytes) & 15;
        decode8<C, A>(ws + k * kPitch + ph + blk_off, oct, v, tabs);
        const float4 x0 = *reinterpret_cast<const float4*>(&xs[k][0]), x1 = *reinterpret_cast<const float4*>(&xs[k][4]);
        const float xv[kRowM] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
        for (int t = 0; t < kRowM; t++)
#pragma unroll
          for (int i = 0; i < 8; i++) acc[t][i] = fmaf(xv[t], v[i], acc[t][i]);
      }
    }
#pragma unroll
    for (int t = 0; t < kRowM; t++) {
#pragma unroll
      for (int i = 0; i < 8; i++) acc[t][i] += __shfl_xor_sync(0xffffffffu, acc[t][i], 16);
      if (half == (t & 1)) {
        *reinterpret_cast<float4*>(&red[warp][t][8 * oc]) = make_float4(acc[t][0], acc[t][1], acc[t][2], acc[t][3]);
        *reinterpret_cast<float4*>(&red[warp][t][8 * oc + 4]) = make_float4(acc[t][4], acc[t][5], acc[t][6], acc[t][7]);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m * kRowCols; i += kThreads) {
      const int t = i / kRowCols, c = i % kRowCols;
      if (blockIdx.x * kRowCols + c >= N) continue;
      float s = 0.f;
#pragma unroll
      for (int v = 0; v < kWarps; v++) s += red[v][t][c];
      OT* out = static_cast<OT*>(y) + (long long)list[e0 + t].y * N + blockIdx.x * kRowCols + c;
      if constexpr (std::is_same<OT, __half>::value) *out = __float2half_rn(s);
      else *out = __float2bfloat16_rn(s);
    }
  }
}

// routing may be uneven: while the CTAs are hardly more than reside at once, several share a matrix's entries
int row_share(int N, int n_experts, long long entries) {
  const long long ctas = (long long)((N + kRowCols - 1) / kRowCols) * n_experts;
  return (int)std::max(1ll, std::min((entries + kRowM - 1) / kRowM, 3 * 148 / ctas));
}

// One row an entry, at least as many entries as matrices: the shared decode against the kernel above with K split S
// ways. Both take time by the rows of K a CTA walks (a third of it there, of 128 columns and eight entries; of 256
// columns and one entry here) and by the CTAs beyond those that reside at once. Within 1-2 % of the faster one on average
// over 780 calls of q4_k, q6_k, iq4_xs and q8_0, 1 to 128 matrices and 1 to 128 entries each. 64 heads [128, 512] q6_k,
// one entry each 11.9 -> 6.3 us, eight 39.6 -> 7.1; but one matrix [4096, 4096] with one entry 34 us above, 90 here, and
// eight [2048, 1024] with one each 24 and 57.
bool rows_pay(int N, int K, int S, int n_experts, long long entries) {
  const double share = row_share(N, n_experts, entries);
  const double ctas = (double)((N + kRowCols - 1) / kRowCols) * n_experts * share;
  const double above = (double)((N + kCols - 1) / kCols) * entries * S;
  const double rows = (double)((entries + n_experts - 1) / n_experts);
  const double passes = std::max(1.0, std::ceil(std::ceil(rows / kRowM) / share));
  return 0.35 * passes * S * std::max(1.0, ctas / (3 * 148)) < std::max(1.0, above / (2 * 148));
}

template <int C, int A, typename XT>
cudaError_t launch_rows(const void* x, void* y, const uint8_t* w, long long row_bytes, int N, int K, cudaStream_t st,
                        QvmGather gq, int n_entries) {
  // the kernel counts its entries from 0: a slice of a longer call starts at its own indices and outputs
  gq.lhs += gq.entry0;
  gq.rhs += gq.entry0;
  y = static_cast<uint16_t*>(y) + gq.entry0 * N;  // both output types have two bytes
  cudaLaunchConfig_t cfg = {};
  const int share = row_share(N, gq.n_experts, n_entries);
  cfg.gridDim = dim3((N + kRowCols - 1) / kRowCols, gq.n_experts, share);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kRowFixed + std::min(kRowChunk, K) * row_pitch(C);
  static bool attr_set[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    const cudaError_t err = cudaFuncSetAttribute(qvm_rows_kernel<C, A, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kRowFixed + kRowChunk * row_pitch(C));
    if (err != cudaSuccess) return err;
    attr_set[dev] = true;
  }
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, qvm_rows_kernel<C, A, XT>, static_cast<const XT*>(x), y, w, row_bytes, N, K, gq,
                            n_entries);
}

template <int C, int A, typename XT>
cudaError_t launch_one(const void* x, long long x_row_stride, void* y, long long y_row_stride, const uint8_t* w,
                       long long row_bytes, int M, int N, int K, cudaStream_t st, QvmGather gq = QvmGather{},
                       long long entries = 1) {
  const int col_ctas = (N + kCols - 1) / kCols, m_tiles = (M + kMT - 1) / kMT;
  int S = 1;
  while (S < kMaxSplit && (long long)col_ctas * m_tiles * entries * S < 2 * 148 && K / (S * 2) >= 4 * kWarps) S *= 2;
  if (gq.rhs != nullptr && M == 1 && entries >= gq.n_experts && entries <= kRowEntries && gq.n_experts <= 65535 &&
      rows_pay(N, K, S, gq.n_experts, entries))
    return launch_rows<C, A, XT>(x, y, w, row_bytes, N, K, st, gq, (int)entries);
  gq.m_tiles = m_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(col_ctas, S, (unsigned)(m_tiles * entries));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = S;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, qvm_kernel<C, A, XT>, static_cast<const XT*>(x), x_row_stride, y, y_row_stride, w,
                            row_bytes, M, N, K, gq);
}

template <int C, int NAT>
cudaError_t launch_codec(int x_dtype, const void* x, long long x_row_stride, void* y, long long y_row_stride,
                         const uint8_t* w, long long row_bytes, int M, int N, int K, cudaStream_t st,
                         QvmGather gq = QvmGather{}, long long entries = 1) {
  // what decode8 loads at once, of every block
  const bool aligned = ((reinterpret_cast<uintptr_t>(w) | row_bytes | gq.expert_stride) & (NAT - 1)) == 0;
#define KQ_QVM(XT)                                                                                                    \
  return aligned ? launch_one<C, NAT, XT>(x, x_row_stride, y, y_row_stride, w, row_bytes, M, N, K, st, gq, entries)  \
                 : launch_one<C, 1, XT>(x, x_row_stride, y, y_row_stride, w, row_bytes, M, N, K, st, gq, entries)
  if (x_dtype == F16) KQ_QVM(__half);
  if (x_dtype == BF16) KQ_QVM(__nv_bfloat16);
  KQ_QVM(float);
#undef KQ_QVM
}

}  // namespace

cudaError_t launch_qvm(int codec, int x_dtype, const void* x, long long x_row_stride, void* y, long long y_row_stride,
                       const uint8_t* w, long long row_bytes, int M, int N, int K, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
  if ((M + kMT - 1) / kMT > 65535) return cudaErrorInvalidConfiguration;
#define KQ_CASE(CODEC, NAT) \
  case CODEC: return launch_codec<CODEC, NAT>(x_dtype, x, x_row_stride, y, y_row_stride, w, row_bytes, M, N, K, st)
  switch (codec) {
    KQ_CASE(Q2_K, 4);
    KQ_CASE(Q3_K, 2);
    KQ_CASE(Q4_K, 16);
    KQ_CASE(Q5_K, 16);
    KQ_CASE(Q6_K, 2);
    KQ_CASE(Q4_0, 2);
    KQ_CASE(Q8_0, 2);
    KQ_CASE(IQ4_NL, 2);
    KQ_CASE(IQ4_XS, 8);
    KQ_CASE(IQ2_XXS, 2);
    KQ_CASE(Q4_1, 4);
    KQ_CASE(Q5_0, 2);
    KQ_CASE(Q5_1, 8);
    KQ_CASE(IQ3_XXS, 2);
    KQ_CASE(IQ3_S, 2);
    KQ_CASE(IQ2_XS, 2);
    KQ_CASE(IQ2_S, 2);
    KQ_CASE(IQ1_S, 2);
    KQ_CASE(IQ1_M, 8);
    KQ_CASE(MXFP4, 1);
    KQ_CASE(NVFP4, 4);
  }
#undef KQ_CASE
  return cudaErrorInvalidValue;
}

// gather form of the same kernel: entry e is x[lhs[e]] ([M, K]) @ dequant(w[rhs[e]]) ([K, N]) -> y[e] ([M, N])
cudaError_t launch_qvm_gather(int codec, int x_dtype, const void* x, long long x_batch, void* y, const uint8_t* w,
                              int n_experts, long long expert_stride, long long row_bytes, int M, int N, int K,
                              const uint32_t* lhs, const uint32_t* rhs, long long n_entries, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0 || n_entries <= 0) return cudaSuccess;
  const int m_tiles = (M + kMT - 1) / kMT;
  if (m_tiles > 65535) return cudaErrorInvalidConfiguration;
  const long long per_launch = 65535 / m_tiles;
  for (long long e0 = 0; e0 < n_entries; e0 += per_launch) {
    const long long cnt = n_entries - e0 < per_launch ? n_entries - e0 : per_launch;
    QvmGather gq{lhs, rhs, e0, x_batch, expert_stride, n_experts, m_tiles};
    cudaError_t err = cudaErrorInvalidValue;
#define KQ_CASE(CODEC, NAT) \
  case CODEC: err = launch_codec<CODEC, NAT>(x_dtype, x, K, y, N, w, row_bytes, M, N, K, st, gq, cnt); break
    switch (codec) {
      KQ_CASE(Q2_K, 4);
      KQ_CASE(Q3_K, 2);
      KQ_CASE(Q4_K, 16);
      KQ_CASE(Q5_K, 16);
      KQ_CASE(Q6_K, 2);
      KQ_CASE(Q4_0, 2);
      KQ_CASE(Q8_0, 2);
      KQ_CASE(IQ4_NL, 2);
      KQ_CASE(IQ4_XS, 8);
      KQ_CASE(IQ2_XXS, 2);
      KQ_CASE(Q4_1, 4);
      KQ_CASE(Q5_0, 2);
      KQ_CASE(Q5_1, 8);
      KQ_CASE(IQ3_XXS, 2);
      KQ_CASE(IQ3_S, 2);
      KQ_CASE(IQ2_XS, 2);
      KQ_CASE(IQ2_S, 2);
      KQ_CASE(IQ1_S, 2);
      KQ_CASE(IQ1_M, 8);
      KQ_CASE(MXFP4, 1);
      KQ_CASE(NVFP4, 4);
    }
#undef KQ_CASE
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

}  // namespace kq
