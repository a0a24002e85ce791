// dequantize: GGUF wire bytes -> f32 / f16 / bf16, bit-exact with the
// reference's CPU decoders (src/kquant_dequantize.cpp:59-91 ->
// src/kquant_cpu_decode.cpp:1136-1207).
//
// HBM-bound streaming kernel. A tile is kTileW consecutive weights: its wire bytes
// (tile_blocks * bytes_per_block, not a multiple of 16 for most codecs) are brought
// into shared memory by one bulk copy that starts at the 16-byte boundary below the
// tile, so global reads are contiguous whatever the block size; every thread then
// decodes eight consecutive weights at a time from shared memory and writes them with
// one or two 16-byte stores, consecutive threads writing consecutive chunks. For
// 16-bit outputs as many CTAs as fit the SMs walk the tiles through two buffers each,
// so that a tile's bytes are under way while the one before is decoded (a CTA per tile
// that loads, waits and decodes spends a third of its life on the load: [14336, 4096]
// -> fp16, q6_k 45 -> 31 us = 5.3 TB/s, q4_k 35 -> 29).
// Algorithmic bytes per weight: bytes_per_block / weights_per_block read plus
// sizeof(out type) written.
#include <algorithm>

#include "kq_common.cuh"
#include "kq_launch.h"
#include "kq_imma_q4k.cuh"
#include "kq_tcgen05.cuh"

namespace kq {

constexpr int kDqThreads = 256;
constexpr int kTileW = 8192;  // weights per tile
// Two buffers and as many CTAs as fit for 16-bit outputs; float32 outputs, bound by their stores, are faster with a
// CTA per tile in launch order (q4_k [14336, 4096] 53 us against 65; fp16 35 against 29).
template <typename T>
constexpr int dq_bufs() { return sizeof(T) == 4 ? 1 : 2; }

// The four bytes of q, minus 32, times d: the two float steps for two weights an instruction. Of the 295 instructions of 32
// weights these are 64, now 32: where the outputs stay in the cache [4096, 4096] q6_k -> bf16 14.9 -> 13.0 us, -> fp16 14.3 ->
// 12.3; [14336, 4096] is bound by its stores (31 us both ways).
__device__ __forceinline__ void dq_mul4(uint32_t q, float d, float* v) {
  unsigned long long two, off, dd;
  asm("mov.b64 %0, {%1, %1};" : "=l"(dd) : "f"(d));
  asm("mov.b64 %0, {%1, %1};" : "=l"(off) : "f"(-8388640.f));
#pragma unroll
  for (int i = 0; i < 2; i++) {
    asm("mov.b64 %0, {%1, %2};" : "=l"(two) : "r"(__byte_perm(q, 0x4B000000u, 0x7440u + 2 * i)), "r"(__byte_perm(q, 0x4B000000u, 0x7441u + 2 * i)));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(two) : "l"(off));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(two) : "l"(dd));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2 * i]), "=f"(v[2 * i + 1]) : "l"(two));
  }
}

template <typename T>
struct Pack8;
template <>
struct Pack8<float> {
  static __device__ __forceinline__ void store(float* o, const float (&v)[8], bool vec) {
    if (vec) {
      __stcs(reinterpret_cast<float4*>(o), make_float4(v[0], v[1], v[2], v[3]));
      __stcs(reinterpret_cast<float4*>(o) + 1, make_float4(v[4], v[5], v[6], v[7]));
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) o[i] = v[i];
    }
  }
};
template <>
struct Pack8<__half> {
  static __device__ __forceinline__ void store(__half* o, const float (&v)[8], bool vec) {
    if (vec) {
      __half2 h[4];
#pragma unroll
      for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
      *reinterpret_cast<uint4*>(o) = *reinterpret_cast<uint4*>(h);
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) o[i] = __float2half_rn(v[i]);
    }
  }
};
template <>
struct Pack8<__nv_bfloat16> {
  static __device__ __forceinline__ void store(__nv_bfloat16* o, const float (&v)[8], bool vec) {
    if (vec) {
      __nv_bfloat162 h[4];
#pragma unroll
      for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      *reinterpret_cast<uint4*>(o) = *reinterpret_cast<uint4*>(h);
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) o[i] = __float2bfloat16_rn(v[i]);
    }
  }
};

// A = alignment of every block start in SHARED memory, which equals the
// alignment of block starts in global memory because the staging copy keeps
// the address phase modulo 16.
template <int C, int A, typename T>
__global__ void __launch_bounds__(kDqThreads)
dequant_kernel(const uint8_t* __restrict__ w, T* __restrict__ out, long long n_blocks, int out_vec, int* error_word) {
  constexpr int WPB = wpb_of(C), BPB = bpb_of(C);
  constexpr int TB = kTileW / WPB;            // blocks per tile
  constexpr int OPB = WPB / 8;                // octets per block
  constexpr int kStage = TB * BPB + 32;       // tile bytes + phase + round-up
  constexpr int kBuf = (kStage + 15) & ~15, kBufs = dq_bufs<T>();
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint64_t full[2];
  __shared__ int abort_s;
  IqTables tabs = global_iq_tables();
  if constexpr (C == IQ4_NL || C == IQ4_XS || C == IQ2_XXS)
    tabs = stage_iq_tables(smem + kBufs * kBuf, threadIdx.x, kDqThreads);

  const long long tiles = (n_blocks + TB - 1) / TB;
  const uint8_t* w_end = w + n_blocks * BPB;
  // one bulk copy from the 16-byte boundary at or below the tile; the bytes past the last whole sixteen of the
  // wire buffer (its last tile only) are stored one by one, before the arrival
  auto fetch = [&](long long tile, int buf) {
    const long long b0 = tile * TB;
    const uint8_t* src = w + b0 * BPB;
    const uint8_t* end = w + min(b0 + TB, n_blocks) * BPB;
    const uint8_t* a0 = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15);
    uint32_t n = (uint32_t)((end - a0 + 15) & ~(long long)15);
    if (a0 + n > w_end) {
      n -= 16;
      for (const uint8_t* q = a0 + n; q < end; q++) smem[buf * kBuf + (q - a0)] = *q;
    }
    st_mbar_expect_tx(&full[buf], n);
    if (n > 0) st_bulk_g2s(smem + buf * kBuf, a0, n, &full[buf]);
  };
  constexpr bool kBulk = A >= 2 && kBufs > 1;
  if constexpr (kBulk) {
    if (threadIdx.x == 0) {
      abort_s = 0;
      st_mbar_init(&full[0], 1);
      st_mbar_init(&full[1], 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
      for (int i = 0; i < kBufs; i++)
        if (blockIdx.x + (long long)i * gridDim.x < tiles) fetch(blockIdx.x + (long long)i * gridDim.x, i);
    }
  }
  __syncthreads();
  int it = 0;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x, it++) {
    const long long b0 = tile * TB;
    const int nb = (int)min((long long)TB, n_blocks - b0);
    const int buf = it % kBufs;
    uint8_t* stage = smem + buf * kBuf;
    int phase;
    if constexpr (A >= 2) {
      phase = (int)(reinterpret_cast<uintptr_t>(w + b0 * BPB) & 15);
      if constexpr (kBufs == 1) {
        // one tile a CTA: sixteen-byte loads by all threads (a bulk copy here: q3_k -> float32 56 us against 49); a chunk
        // that would run past the end of the wire buffer is copied byte by byte
        const uint8_t* a0 = w + b0 * BPB - phase;
        const int nchunks = (phase + nb * BPB + 15) >> 4;
        for (int c = threadIdx.x; c < nchunks; c += kDqThreads) {
          const uint8_t* g = a0 + 16 * c;
          if (g + 16 <= w_end) {
            reinterpret_cast<uint4*>(stage)[c] = *reinterpret_cast<const uint4*>(g);
          } else {
            for (int i = 0; i < 16; i++)
              if (g + i < w_end) stage[16 * c + i] = g[i];
          }
        }
        __syncthreads();
      } else {
        if (!mbar_wait_err(&full[buf], (it / kBufs) & 1, &abort_s, 0x200, error_word)) return;
      }
    } else {
      phase = 0;
      const uint8_t* src = w + b0 * BPB;
      for (int i = threadIdx.x; i < nb * BPB; i += kDqThreads) stage[i] = src[i];
      __syncthreads();
    }

    const uint8_t* tile_s = stage + phase;
    T* out_t = out + b0 * WPB;
    const int n_oct = nb * OPB;
    if constexpr ((C == Q4_K || C == Q5_K) && A >= 4) {
      // The 6-bit scale / min pair of a sub-block serves 32 weights: unpack each pair once per tile
      // (one per thread: TB * 8 = 256 of them) instead of once per eight weights. Same arithmetic as
      // decode8<>: sc = d * scale, mn = dmin * min in fp32, v = sc * q - mn (sc * q is exact).
      float2* scmn = reinterpret_cast<float2*>(smem + kBufs * kBuf);
      for (int i = threadIdx.x; i < nb * 8; i += kDqThreads) {
        const uint8_t* blk = tile_s + (i >> 3) * BPB;
        const uint32_t h = ld32<A>(blk);
        const float d = __half2float(__ushort_as_half((unsigned short)(h & 0xffff)));
        const float dmin = __half2float(__ushort_as_half((unsigned short)(h >> 16)));
        uint32_t rsc, rmn;
        k4_scale_min(ld32<A>(blk + 4), ld32<A>(blk + 8), ld32<A>(blk + 12), i & 7, rsc, rmn);
        scmn[i] = make_float2(d * u2f(rsc), dmin * u2f(rmn));
      }
      __syncthreads();
      for (int o = threadIdx.x; o < n_oct; o += kDqThreads) {
        const int blk = o / OPB, j = o % OPB;
        const int sb = j >> 2, i0 = (j & 3) * 8;
        const float2 sm = scmn[blk * 8 + sb];
        const uint8_t* bp = tile_s + blk * BPB;
        const uint8_t* qs = bp + (C == Q4_K ? 16 : 48) + (sb >> 1) * 32 + i0;
        const int sh = (sb & 1) * 4;
        // four nibbles per word in the low halves of its bytes, then one conversion per byte
        uint32_t n0 = (ld32<A>(qs) >> sh) & 0x0f0f0f0fu, n1 = (ld32<A>(qs + 4) >> sh) & 0x0f0f0f0fu;
        if constexpr (C == Q5_K) {
          n0 |= ((ld32<A>(bp + 16 + i0) >> sb) & 0x01010101u) << 4;
          n1 |= ((ld32<A>(bp + 20 + i0) >> sb) & 0x01010101u) << 4;
        }
        float v[8];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          v[c] = sm.x * b2f(n0, c) - sm.y;
          v[c + 4] = sm.x * b2f(n1, c) - sm.y;
        }
        Pack8<T>::store(out_t + (size_t)o * 8, v, out_vec != 0);
      }
    } else if constexpr (C == Q6_K && A >= 2 && sizeof(T) == 2) {
      // Weights l, l + 32, l + 64, l + 96 of a half share bytes: a thread makes eight of each from one read of them
      // (two-byte loads: 14 for 32 weights instead of 40), 256 such units a tile. Same products as decode8<>, exact in
      // fp32 in any order. 16-bit outputs only: their 64-byte runs cost nothing, those of float32 a third.
      for (int o = threadIdx.x; o < nb * 8; o += kDqThreads) {
        const uint8_t* bp = tile_s + (o >> 3) * BPB;
        const int half = (o >> 2) & 1, l0 = (o & 3) * 8;
        const uint8_t *ql = bp + 64 * half + l0, *qh = bp + 128 + 32 * half + l0;
        const uint32_t l[2][2] = {{ld32<2>(ql), ld32<2>(ql + 4)}, {ld32<2>(ql + 32), ld32<2>(ql + 36)}};
        const uint32_t h[2] = {ld32<2>(qh), ld32<2>(qh + 4)};
        const float d = ldf16<2>(bp + 208);
        const uint8_t* sc = bp + 192 + 8 * half + (l0 >> 4);
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
          const float dsc = d * (float)(int)(int8_t)sc[2 * qd];
          float v[8];
#pragma unroll
          for (int p = 0; p < 2; p++) {
            const uint32_t q = ((l[qd & 1][p] >> (2 * (qd & 2))) & 0x0f0f0f0fu) | (((h[p] >> (2 * qd)) & 0x03030303u) << 4);
            dq_mul4(q, dsc, v + 4 * p);
          }
          Pack8<T>::store(out_t + (size_t)(o >> 3) * 256 + 128 * half + 32 * qd + l0, v, out_vec != 0);
        }
      }
    } else {
      for (int o = threadIdx.x; o < n_oct; o += kDqThreads) {
        const int blk = o / OPB, j = o % OPB;
        float v[8];
        decode8<C, A>(tile_s + blk * BPB, j, v, tabs);
        Pack8<T>::store(out_t + (size_t)o * 8, v, out_vec != 0);
      }
    }
    __syncthreads();  // the buffer has been read
    if constexpr (kBulk) {
      if (threadIdx.x == 0 && tile + (long long)kBufs * gridDim.x < tiles)
        fetch(tile + (long long)kBufs * gridDim.x, buf);
    }
  }
}

template <int C, int A, typename T>
static cudaError_t launch_one(const uint8_t* w, void* out, long long n_blocks, cudaStream_t st) {
  constexpr int WPB = wpb_of(C), BPB = bpb_of(C), TB = kTileW / WPB;
  const long long tiles = (n_blocks + TB - 1) / TB;
  if (tiles == 0) return cudaSuccess;
  static_assert(kIqSmemBytes >= (kTileW / 256) * 8 * 8, "the k-quant scale table shares the IQ table area");
  const int smem = dq_bufs<T>() * ((TB * BPB + 32 + 15) & ~15) + kIqSmemBytes;
  const int out_vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  static int resident[16] = {};  // CTAs that fit the device at once
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (resident[dev] == 0) {
    int per_sm = 0, sms = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dequant_kernel<C, A, T>, kDqThreads, smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    resident[dev] = std::max(1, per_sm * sms);
  }
  int* err = device_error_word();
  if (err == nullptr) return cudaErrorUnknown;
  dequant_kernel<C, A, T><<<(unsigned)(dq_bufs<T>() == 1 ? tiles : std::min<long long>(tiles, resident[dev])), kDqThreads, smem, st>>>(
      w, static_cast<T*>(out), n_blocks, out_vec, err);
  return cudaGetLastError();
}

template <int C, int NAT>
static cudaError_t launch_codec(const uint8_t* w, void* out, long long n_blocks, int dtype, cudaStream_t st) {
  // Natural block alignment holds when the wire base is 16-byte aligned
  // (cudaMalloc / torch allocations are); otherwise take the byte-wise variant.
  const bool aligned = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
#define KQ_DQ(T)                                                   \
  return aligned ? launch_one<C, NAT, T>(w, out, n_blocks, st)     \
                 : launch_one<C, 1, T>(w, out, n_blocks, st)
  switch (dtype) {
    case F32: KQ_DQ(float);
    case F16: KQ_DQ(__half);
    case BF16: KQ_DQ(__nv_bfloat16);
  }
#undef KQ_DQ
  return cudaErrorInvalidValue;
}

cudaError_t launch_dequantize(int codec, const uint8_t* w, long long n_blocks, int dtype, void* out,
                              cudaStream_t st) {
  switch (codec) {
    case Q2_K: return launch_codec<Q2_K, 4>(w, out, n_blocks, dtype, st);
    case Q3_K: return launch_codec<Q3_K, 2>(w, out, n_blocks, dtype, st);
    case Q4_K: return launch_codec<Q4_K, 16>(w, out, n_blocks, dtype, st);
    case Q5_K: return launch_codec<Q5_K, 16>(w, out, n_blocks, dtype, st);
    case Q6_K: return launch_codec<Q6_K, 2>(w, out, n_blocks, dtype, st);
    case Q4_0: return launch_codec<Q4_0, 2>(w, out, n_blocks, dtype, st);
    case Q8_0: return launch_codec<Q8_0, 2>(w, out, n_blocks, dtype, st);
    case IQ4_NL: return launch_codec<IQ4_NL, 2>(w, out, n_blocks, dtype, st);
    case IQ4_XS: return launch_codec<IQ4_XS, 8>(w, out, n_blocks, dtype, st);
    case IQ2_XXS: return launch_codec<IQ2_XXS, 2>(w, out, n_blocks, dtype, st);
    case Q4_1: return launch_codec<Q4_1, 4>(w, out, n_blocks, dtype, st);
    case Q5_0: return launch_codec<Q5_0, 2>(w, out, n_blocks, dtype, st);
    case Q5_1: return launch_codec<Q5_1, 8>(w, out, n_blocks, dtype, st);
    case IQ3_XXS: return launch_codec<IQ3_XXS, 2>(w, out, n_blocks, dtype, st);
    case IQ3_S: return launch_codec<IQ3_S, 2>(w, out, n_blocks, dtype, st);
    case IQ2_XS: return launch_codec<IQ2_XS, 2>(w, out, n_blocks, dtype, st);
    case IQ2_S: return launch_codec<IQ2_S, 2>(w, out, n_blocks, dtype, st);
    case IQ1_S: return launch_codec<IQ1_S, 2>(w, out, n_blocks, dtype, st);
    case IQ1_M: return launch_codec<IQ1_M, 8>(w, out, n_blocks, dtype, st);
    case MXFP4: return launch_codec<MXFP4, 1>(w, out, n_blocks, dtype, st);
    case NVFP4: return launch_codec<NVFP4, 4>(w, out, n_blocks, dtype, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kq
