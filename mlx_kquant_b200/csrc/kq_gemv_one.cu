// One dense activation row against q4_k, q5_k, q6_k: y[N] = x[K] . dequant(W)^T on the integer dot-product pipe.
// Reference: qmv_fused_rows, src/kquant_cpu_decode.cpp:1032-1065; decode src/kquant_cpu_decode.cpp:177-280.
//
// The arithmetic is that of kq_gemv_dp4a.cuh - activations as 16-bit integers with a scale per 32 of them, in two byte
// planes, exact integer sums per sub-block, scales in float32 - but what bounded that kernel on these codecs was not the
// products: of its 5.4 instructions a weight (q6_k [4096, 14336]: 29 us, issue slots a third busy) more than half moved wire
// bytes, in pieces of sixteen with an address each, and read them back word by word. Here one thread of a warp fetches a
// superblock of the warp's rows as one TMA box, and a thread reads its row's part in 16-byte words (box rows are odd
// multiples of sixteen bytes: no bank conflicts).
// One CTA per SM owns N / SM count rows, in blocks of at most 32 (a thread a row), sixteen blocks at most (beyond 75 776 rows
// there are more CTAs than SMs); its warps take the (block, superblock)
// units in turn, several in flight each, and meet in shared memory. Measured, one bf16 row, back to back in a graph, before
// and after: q6_k [4096, 14336] 29.0 -> 13.4 us, [28672, 8192] 65.8 -> 35.6 (5.4 TB/s), q5_k [8192, 8192] 21.9 -> 12.3, q4_k
// [28672, 8192] 39.1 -> 25.6 (5.2 TB/s), [14336, 4096] 10.5 -> 9.3. Bound by HBM on large matrices, by the start of a launch
// (fetching and quantizing the row) and its end on small ones.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_launch.h"
#include "kq_tcgen05.cuh"
#include "kq_tma_map.h"

namespace kq {

namespace {

constexpr int kOneWarps = 12, kOneThreads = 32 * kOneWarps, kOneSlots = 4, kOneBlocks = 16;
constexpr int kOneMaxK = 16384, kOneSmem = 222 * 1024;
// the least maximum that a scale is made for: 32767 / amax stays finite
constexpr float kOneLeast = 0x1p-112f;
// bytes of a box row: the superblock, for q6_k the aligned window around it
__host__ __device__ constexpr int one_pitch(int c) { return c == Q4_K ? 144 : (c == Q5_K ? 176 : 240); }
// XH [K] | XL [K] | scale per 32 [K / 32] | integer sums per 16 [K / 16] | float sums per 32 [K / 32]
__host__ __device__ constexpr int one_x_bytes(int K) { return 2 * K + K / 8 + K / 4 + K / 8; }

struct OnePlan {
  int R, blocks;         // rows of a block, blocks of a CTA
  int D, slot, x_off, red_off;  // slots of a warp, bytes of one, offsets of the activations and of the warps' sums
};

// activations of a superblock
struct OneX {
  const uint4 *xh, *xl;  // sixteen each: sixteen activations a piece
  const float* sg;       // 8
  const int* xi16;       // 16
  const float* xs;       // 8
};

__device__ __forceinline__ float one_byte(uint32_t v, int j) {  // byte j as a float (mantissa of 2^23)
  return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u + j)) - 8388608.f;
}
__device__ __forceinline__ void dot4(uint32_t q, uint32_t xh, uint32_t xl, int& hi, int& lo) {
  asm("dp4a.u32.s32 %0, %1, %2, %0;\n" : "+r"(hi) : "r"(q), "r"(xh));
  asm("dp4a.u32.u32 %0, %1, %2, %0;\n" : "+r"(lo) : "r"(q), "r"(xl));
}

// q4_k / q5_k: 32 quant bytes hold sub-blocks 2 p (low nibbles) and 2 p + 1 (high ones).
// MID (q4_k, fp16 rows of large matrices): the integers multiply quants less 8, eight times the activations' float sum makes up for it. An
// activation is off by its rounding to an integer, and quants, half their range on average, are twice the weights that they
// stand for. Errors beyond the output's rounding, [28672, 8192], 5.1e-5 -> 2.2e-5 of the outputs' size: not above the 2.7e-5
// of the fp16 matrix kernel that had matrices beyond 60 M weights (32.9 us; 25.7 -> 26.5 here). Smaller ones had 16-bit integers
// with a scale per 256 of them (6.3e-5) and are spared the 2 to 3 %.
template <int C, bool MID>
__device__ __forceinline__ float one_dot_k4(const uint8_t* blk, const OneX& X) {
  const uint4* b = reinterpret_cast<const uint4*>(blk);
  const uint4 hdr = b[0];
  const uint32_t sc[2] = {hdr.y & 0x3f3f3f3fu, (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u)};
  const uint32_t mn[2] = {hdr.z & 0x3f3f3f3fu, ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u)};
  uint4 u[2] = {};
  if constexpr (C == Q5_K) u[0] = b[1], u[1] = b[2];
  const uint32_t uw[8] = {u[0].x, u[0].y, u[0].z, u[0].w, u[1].x, u[1].y, u[1].z, u[1].w};
  float prod = 0.f, mins = 0.f, mids = 0.f;
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const uint4 q0 = b[(C == Q5_K ? 3 : 1) + 2 * p], q1 = b[(C == Q5_K ? 4 : 2) + 2 * p];
    const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
      const int j = 2 * p + hh;
      int hi = 0, lo = 0;
#pragma unroll
      for (int s = 0; s < 2; s++) {
        const uint4 xh = X.xh[2 * j + s], xl = X.xl[2 * j + s];
        const uint32_t h[4] = {xh.x, xh.y, xh.z, xh.w}, l[4] = {xl.x, xl.y, xl.z, xl.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
          uint32_t q;
          if constexpr (C == Q4_K) {
            q = w[4 * s + i] & (hh ? 0xf0f0f0f0u : 0x0f0f0f0fu);  // (the high ones stay in place: 16 q)
          } else {
            const uint32_t v = uw[4 * s + i];
            q = ((hh ? w[4 * s + i] >> 4 : w[4 * s + i]) & 0x0f0f0f0fu) | ((j <= 4 ? v << (4 - j) : v >> (j - 4)) & 0x10101010u);
          }
          dot4(q, h[i], l[i], hi, lo);
        }
      }
      const float scale = one_byte(sc[j >> 2], j & 3), s = scale * X.sg[j];
      int dot = hi * 256 + lo;
      if constexpr (MID) {
        const int2 xi = *reinterpret_cast<const int2*>(X.xi16 + 2 * j);
        dot -= (hh ? 128 : 8) * (xi.x + xi.y);
        mids = fmaf(scale, X.xs[j], mids);
      }
      prod = fmaf(C == Q4_K && hh ? s * 0.0625f : s, (float)dot, prod);
      mins = fmaf(one_byte(mn[j >> 2], j & 3), X.xs[j], mins);
    }
  }
  const float2 dd = __half22float2(*reinterpret_cast<const __half2*>(&hdr.x));
  if constexpr (MID) prod = fmaf(8.f, mids, prod);
  return dd.x * prod - dd.y * mins;
}

// q6_k: half hf of the superblock is four quarters of 32 weights over the same 64 ql and 32 qh bytes; scales per sixteen
template <int W>
__device__ __forceinline__ float one_dot_q6_at(const uint8_t* win, uint32_t odd_bits, const OneX& X) {
  float prod = 0.f;
#pragma unroll 1  // four variants of this run side by side: unrolled they outgrow the instruction cache
  for (int hf = 0; hf < 2; hf++) {
    uint32_t sc[2];
    {
      const uint32_t* s = reinterpret_cast<const uint32_t*>(win + 192 + 8 * hf + 4 * W);
      const uint32_t v0 = s[0], v1 = s[1], v2 = s[2];
      sc[0] = __funnelshift_r(v0, v1, odd_bits) ^ 0x80808080u, sc[1] = __funnelshift_r(v1, v2, odd_bits) ^ 0x80808080u;  // biased by 128
    }
    uint32_t H[8];
    window_words<W, 8>(win + 128 + 32 * hf, odd_bits, H);
#pragma unroll
    for (int a = 0; a < 2; a++) {
      uint32_t L[8];
      window_words<W, 8>(win + 64 * hf + 32 * a, odd_bits, L);
#pragma unroll
      for (int up = 0; up < 2; up++) {
        const int qd = 2 * up + a;
#pragma unroll
        for (int s = 0; s < 2; s++) {
          const int g = 8 * hf + 2 * qd + s;
          const uint4 xh = X.xh[g], xl = X.xl[g];
          const uint32_t h[4] = {xh.x, xh.y, xh.z, xh.w}, l[4] = {xl.x, xl.y, xl.z, xl.w};
          int hi = 0, lo = 0;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const uint32_t hv = H[4 * s + i];
            const uint32_t hb = qd == 0 ? hv << 4 : (qd == 1 ? hv << 2 : (qd == 2 ? hv : hv >> 2));
            const uint32_t q = ((up ? L[4 * s + i] >> 4 : L[4 * s + i]) & 0x0f0f0f0fu) | (hb & 0x30303030u);
            dot4(q, h[i], l[i], hi, lo);
          }
          const int dot = hi * 256 + lo - 32 * X.xi16[g];
          prod = fmaf((one_byte(sc[up], 2 * a + s) - 128.f) * X.sg[g >> 1], (float)dot, prod);
        }
      }
    }
  }
  return prod * __half2float(*reinterpret_cast<const __half*>(win + 4 * W + (odd_bits >> 3) + 208));
}

__device__ __forceinline__ void one_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

template <int C, typename XT, bool MID>
__global__ void __launch_bounds__(kOneThreads, 1)
gemv_one_kernel(const GemvArgs a, const OnePlan pl, const __grid_constant__ CUtensorMap map, int* __restrict__ error_word) {
  using OT = typename std::conditional<std::is_same<XT, __half>::value, __half, __nv_bfloat16>::type;
  constexpr int kPitch = one_pitch(C), kBlk = bpb_of(C);
  extern __shared__ __align__(128) uint8_t one_dyn[];
  __shared__ uint64_t full[kOneWarps][kOneSlots];
  __shared__ int abort_s;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = a.K, nsb = K >> 8, D = pl.D;
  const int row0 = (int)blockIdx.x * pl.R * pl.blocks;
  const int blocks = min(pl.blocks, (a.N - row0 + pl.R - 1) / pl.R), units = blocks * nsb;
  if (lane == 0) {
    for (int d = 0; d < D; d++) mbar_init(&full[warp][d], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (threadIdx.x == 0) abort_s = 0;
  __syncwarp();
  uint8_t* ring = one_dyn + warp * D * pl.slot;
  float(*red)[kOneWarps][32] = reinterpret_cast<float(*)[kOneWarps][32]>(one_dyn + pl.red_off);  // [block]
  // unit u: block u / nsb, superblock u % nsb
  auto issue = [&](int u, int d) {
    const int b = u / nsb, sb = u - b * nsb;
    mbar_expect_tx(&full[warp][d], pl.R * kPitch);
    one_load(smem_u32(ring + d * pl.slot), &map, (sb * kBlk) & ~15, row0 + b * pl.R, &full[warp][d]);
  };
  if (lane == 0)
    for (int d = 0; d < D; d++)
      if (warp + d * kOneWarps < units) issue(warp + d * kOneWarps, d);
  __syncwarp();
  for (int i = threadIdx.x; i < blocks * kOneWarps * 32; i += kOneThreads) (&red[0][0][0])[i] = 0.f;
  __syncthreads();
  asm volatile("griddepcontrol.wait;\n" ::: "memory");  // activations may come from the kernel before this one

  // ---- the row as integers: eight activations a thread and step, four threads to a scale
  uint8_t* xb = one_dyn + pl.x_off;
  uint32_t* XH = reinterpret_cast<uint32_t*>(xb);
  uint32_t* XL = XH + K / 4;
  float* SG = reinterpret_cast<float*>(XL + K / 4);
  int* XI = reinterpret_cast<int*>(SG + K / 32);
  float* XS = reinterpret_cast<float*>(XI + K / 16);
  const XT* xrow = static_cast<const XT*>(a.x);
  for (int c0 = 0; c0 < K / 8; c0 += 4 * kOneThreads) {
    uint4 in[4], in2[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int c = c0 + threadIdx.x + i * kOneThreads;
      if (c < K / 8) {
        if constexpr (sizeof(XT) == 4) {
          in[i] = __ldcg(reinterpret_cast<const uint4*>(xrow + 8 * c));
          in2[i] = __ldcg(reinterpret_cast<const uint4*>(xrow + 8 * c) + 1);
        } else {
          in[i] = __ldcg(reinterpret_cast<const uint4*>(xrow + 8 * c));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int c = c0 + threadIdx.x + i * kOneThreads;
      if (c >= K / 8) continue;  // (K / 8 is a multiple of 32: whole warps)
      float v[8];
      if constexpr (sizeof(XT) == 4) {
        const uint32_t f[8] = {in[i].x, in[i].y, in[i].z, in[i].w, in2[i].x, in2[i].y, in2[i].z, in2[i].w};
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = __bfloat162float(__float2bfloat16_rn(__uint_as_float(f[e])));
      } else {
        const uint32_t w4[4] = {in[i].x, in[i].y, in[i].z, in[i].w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          float2 f;
          if constexpr (std::is_same<XT, __half>::value) f = __half22float2(*reinterpret_cast<const __half2*>(&w4[e]));
          else f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w4[e]));
          v[2 * e] = f.x, v[2 * e + 1] = f.y;
        }
      }
      // the largest magnitude as bits: infinities and NaNs, which order above all numbers, survive it
      uint32_t top = 0;
      float sum = 0.f;
#pragma unroll
      for (int e = 0; e < 8; e++) {
        top = max(top, __float_as_uint(v[e]) & 0x7fffffffu);
        sum += v[e];
      }
      top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      const bool finite = top > 0 && top < 0x7f800000u;
      const float amax = finite ? fmaxf(__uint_as_float(top), kOneLeast) : __uint_as_float(top);
      const float inv = finite ? 32767.f * __frcp_rn(amax) : 0.f;
      int xi[8], isum = 0;
      uint32_t h[2], l[2];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        xi[e] = __float2int_rn(v[e] * inv);
        isum += xi[e];
      }
#pragma unroll
      for (int e = 0; e < 2; e++) {  // bytes 0 and 1 of four integers
        const uint32_t p0 = __byte_perm(xi[4 * e], xi[4 * e + 1], 0x5140), p1 = __byte_perm(xi[4 * e + 2], xi[4 * e + 3], 0x5140);
        l[e] = __byte_perm(p0, p1, 0x5410);
        h[e] = __byte_perm(p0, p1, 0x7632);
      }
      isum += __shfl_xor_sync(0xffffffffu, isum, 1);
      *reinterpret_cast<uint2*>(XH + 2 * c) = make_uint2(h[0], h[1]);
      *reinterpret_cast<uint2*>(XL + 2 * c) = make_uint2(l[0], l[1]);
      if ((c & 1) == 0) XI[c >> 1] = isum;
      if ((c & 3) == 0) {
        XS[c >> 2] = sum;
        // a group holding inf / nan: its integers are zeros, and zero times the scale makes every output a NaN, which is
        // computed again below
        SG[c >> 2] = finite ? amax * (1.f / 32767.f) : amax;
      }
    }
  }
  __syncthreads();

  volatile int* abort_flag = &abort_s;
  float y = 0.f;
  int blk = 0, d = 0;
  uint32_t ph = 0;
  for (int u = warp; u < units; u += kOneWarps) {
    const int b = u / nsb, sb = u - b * nsb;
    if (b != blk) {
      red[blk][warp][lane] = y;
      y = 0.f;
      blk = b;
    }
    if (!mbar_wait_err(&full[warp][d], ph, abort_flag, 0x200, error_word)) break;
    const uint8_t* row = ring + d * pl.slot + min(lane, pl.R - 1) * kPitch;
    const OneX X{reinterpret_cast<const uint4*>(XH) + 16 * sb, reinterpret_cast<const uint4*>(XL) + 16 * sb, SG + 8 * sb,
                 XI + 16 * sb, XS + 8 * sb};
    if constexpr (C == Q6_K) {
      const int phase = (sb * kBlk) & 15;  // the same for all rows
      const uint32_t odd = 8u * (phase & 2);
      switch (phase >> 2) {
        case 0: y += one_dot_q6_at<0>(row, odd, X); break;
        case 1: y += one_dot_q6_at<1>(row, odd, X); break;
        case 2: y += one_dot_q6_at<2>(row, odd, X); break;
        default: y += one_dot_q6_at<3>(row, odd, X); break;
      }
    } else {
      y += one_dot_k4<C, MID>(row, X);
    }
    __syncwarp();  // the slot has been read
    if (lane == 0 && u + D * kOneWarps < units) issue(u + D * kOneWarps, d);
    if (++d == D) d = 0, ph ^= 1;
  }
  red[blk][warp][lane] = y;
  __syncthreads();
  if (abort_s != 0) {  // given up: no outputs; what is in flight lands long before this
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) {
    }
    return;
  }
  for (int i = threadIdx.x; i < blocks * pl.R; i += kOneThreads) {
    const int b = i / pl.R, r = i - b * pl.R, n = row0 + i;
    if (n >= a.N) continue;
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kOneWarps; w++) sum += red[b][w][r];
    // Infinities and NaN among the activations; and the sums of 32 activations and the sub-blocks' scales come before the
    // superblock's scale, which is small, and can overflow for the largest of them.
    if (!(fabsf(sum) < INFINITY)) sum = plain_dot<C, C == Q6_K ? 2 : 16>(a.w + (long long)n * a.row_bytes, xrow, K);
    OT* out = static_cast<OT*>(a.y) + n;
    if constexpr (std::is_same<OT, __half>::value) *out = __float2half_rn(sum);
    else *out = __float2bfloat16_rn(sum);
  }
}

template <int C, typename XT, bool MID = false>
cudaError_t launch_one_t(const GemvArgs& a, cudaStream_t st) {
  auto kern = gemv_one_kernel<C, XT, MID>;
  static int sms[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (sms[dev] == 0) {
    int n = 0;
    cudaError_t e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneSmem);
    if (e != cudaSuccess) return e;
    sms[dev] = n;
  }
  int* err = device_error_word();
  EncodeTiledFn enc = encode_tiled_fn();
  if (err == nullptr || enc == nullptr) return cudaErrorNotSupported;
  OnePlan pl;
  const int per_sm = (a.N + sms[dev] - 1) / sms[dev];
  pl.blocks = std::min(kOneBlocks, (per_sm + 31) / 32);
  pl.R = std::min(32, (per_sm + pl.blocks - 1) / pl.blocks);
  pl.slot = (pl.R * one_pitch(C) + 127) & ~127;
  // Slots of a warp: two where a second CTA (that of the next launch, which then has its first weights before its turn
  // comes) fits beside, otherwise as many as shared memory holds. [14336, 4096] q4_k 9.3 us with two, 10.3 with four alone;
  // q6_k 13.2 with two alone, 16.1 with one beside another.
  const int turns = (pl.blocks * (a.K >> 8) + kOneWarps - 1) / kOneWarps;
  const int rest = ((one_x_bytes(a.K) + 127) & ~127) + pl.blocks * kOneWarps * 128;
  const int fit = std::min(kOneSlots, (kOneSmem - rest) / (kOneWarps * pl.slot));
  const int beside = (kOneSmem / 2 - 2048 - rest) / (kOneWarps * pl.slot);
  pl.D = std::max(1, std::min(turns, beside >= 2 ? std::min(beside, kOneSlots) : fit));
  pl.x_off = kOneWarps * pl.D * pl.slot;
  pl.red_off = pl.x_off + ((one_x_bytes(a.K) + 127) & ~127);
  alignas(64) CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)a.row_bytes, (cuuint64_t)a.N};
  const cuuint64_t strides[1] = {(cuuint64_t)a.row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)one_pitch(C), (cuuint32_t)pl.R};
  const cuuint32_t estr[2] = {1, 1};
  if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(a.w), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.N + pl.R * pl.blocks - 1) / (pl.R * pl.blocks));
  cfg.blockDim = dim3(kOneThreads);
  cfg.dynamicSmemBytes = pl.red_off + pl.blocks * kOneWarps * 128;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a, pl, map, err);
}

template <int C>
cudaError_t launch_one_c(int x_dtype, const GemvArgs& a, cudaStream_t st) {
  if (C == Q4_K && x_dtype == F16 && (long long)a.N * a.K > (60ll << 20)) return launch_one_t<C, __half, C == Q4_K>(a, st);
  if (x_dtype == F16) return launch_one_t<C, __half>(a, st);
  if (x_dtype == BF16) return launch_one_t<C, __nv_bfloat16>(a, st);
  return launch_one_t<C, float>(a, st);
}

}  // namespace

bool gemv_one_supported(int codec, const GemvArgs& a) {
  return (codec == Q4_K || codec == Q5_K || codec == Q6_K) && a.M == 1 && a.tasks == nullptr && a.bias == nullptr &&
         a.out_bf16 == 0 && a.row_scale == nullptr && a.w_align16 != 0 && (a.K & 255) == 0 && a.K <= kOneMaxK && a.N >= 8 &&
         (a.row_bytes & 15) == 0 && a.row_bytes == (long long)(a.K >> 8) * bpb_of(codec) &&
         (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;
}

cudaError_t launch_gemv_one(int codec, int x_dtype, const GemvArgs& a, cudaStream_t st) {
  switch (codec) {
    case Q4_K: return launch_one_c<Q4_K>(x_dtype, a, st);
    case Q5_K: return launch_one_c<Q5_K>(x_dtype, a, st);
    case Q6_K: return launch_one_c<Q6_K>(x_dtype, a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kq
