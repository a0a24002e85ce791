// Fused mixture-of-experts decode kernels for q4_k expert stacks (the B200 counterparts of the reference's
// Metal-only ops moe_glu_gather_kq, gather_qmv_mix_ns_kq and moe_router_topk, src/kquant.h:335-357, 549-558,
// 560-585), for calls of a few tokens where every routed (token, expert) entry streams its own expert's rows:
//
//   moe_glu_kernel     h[entry, f] = act(x[token] . Wg[e][f]) * (x[token] . Wu[e][f])
//                      grid (F / 16, entries): one CTA multiplies 16 gate rows and the 16 up rows of the same
//                      features by one activation row (the two 16-row fragments share every activation
//                      fragment) and applies the activation before its single rounding.
//   moe_mix_kernel     y[token, n] = sum_s score[token, s] * (h[token, s] . Wd[e_s][n])
//                      grid (N / 16, tokens): warp w owns slot s = w, w + 8, ...: it quantizes that slot's
//                      activation row, multiplies the slot's expert rows, and the score-weighted float32 sum
//                      over the slots is taken in slot order before the single rounding.
//   router_topk_kernel one warp per token, the E scores in registers, top_k rounds of a warp arg-max with the
//                      lowest index winning ties.
//
// Both product kernels start their weight copies before griddepcontrol.wait, from the expert indices as they
// are in memory then; after the wait the indices are read again and a CTA whose expert changed copies again
// (its first copy has landed by then). The activations are only read after the wait.
// Arithmetic and shared-memory layout of the products: kq_imma_q4k.cuh / kq_gemv_stream.cu.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_imma_q4k.cuh"
#include "kq_launch.h"
#include "kq_rows_unit.cuh"
#include "kq_tma_map.h"

namespace kq {

namespace {

constexpr int kMdWarps = 8, kMdThreads = 32 * kMdWarps;

inline int md_group_stride(long long row_bytes) {
  const long long gb = 4 * row_bytes;
  return (int)(gb + ((32 - (gb & 127)) & 127));
}

__device__ __forceinline__ uint32_t md_ld_cg32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// bounded wait for a bulk-copy barrier; false (and a raised flag) after two seconds
__device__ __forceinline__ bool md_wait(uint64_t* bar, uint32_t parity, int* error_word) {
  if (st_mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = st_gtime();
  for (int spin = 0; !st_mbar_try_wait(bar, parity); spin++) {
    if ((spin & 63) == 63 && st_gtime() - t0 > 2000000000ull) {
      atomicOr(error_word, 0x100);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ float md_act(float g, float u, int act, float limit) {
  if (act == 1) {  // tanh-approximated gelu
    const float t = tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g));
    return (0.5f * g * (1.0f + t)) * u;
  }
  if (act == 2) {  // limited SwiGLU: gate clamped from above, up clamped on both sides
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
  }
  return (g / (1.0f + expf(-g))) * u;
}

template <typename T>
__device__ __forceinline__ void md_store(T* p, float v) {
  if constexpr (std::is_same<T, __half>::value) *p = __float2half_rn(v);
  else *p = __float2bfloat16_rn(v);
}

// copies of up to 16 rows of one matrix in groups of four (group i at dst + i * GS)
__device__ __forceinline__ void md_copy_tile(uint8_t* dst, const uint8_t* src, int rows, int RB, int GS, uint64_t* bar) {
  for (int r = 0; r < rows; r += 4) st_bulk_g2s(dst + (r >> 2) * GS, src + (long long)r * RB, (uint32_t)(min(4, rows - r) * RB), bar);
}

struct GluArgs {
  const void* x;            // [T, K]
  const uint8_t* wg;
  const uint8_t* wu;
  long long stride_g, stride_u;
  int row_bytes, K, F, R, n_entries, n_experts;
  const uint32_t* idx;      // [T * R]
  void* y;                  // [T * R, F]
  int act;
  float limit;
};

// shared memory: gate tile | up tile (4 groups each) | planes 2 K | XS K / 32 | SX K / 256 (padded) | red 8 x 32 | mbar
inline int glu_smem_bytes(int K, int row_bytes) {
  return 8 * md_group_stride(row_bytes) + 2 * K + (K / 32) * 4 + (((K / 256) + 3) & ~3) * 4 + kMdWarps * 32 * 4 + 16;
}

template <typename XT>
__global__ void __launch_bounds__(kMdThreads, 3) moe_glu_kernel(const GluArgs a, int* __restrict__ error_word) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  extern __shared__ __align__(128) uint8_t md_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int K = a.K, nchunks = K >> 8, RB = a.row_bytes;
  const int gb = 4 * RB, GS = gb + ((32 - (gb & 127)) & 127);
  uint8_t* wbuf = md_dyn;
  uint8_t* planes = wbuf + 8 * GS;
  float* XS = reinterpret_cast<float*>(planes + 2 * K);
  float* SX = XS + (K / 32);
  float* red = SX + ((nchunks + 3) & ~3);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(red + kMdWarps * 32);
  const int entry = blockIdx.y, f0 = blockIdx.x * 16;
  const int rows = min(16, a.F - f0);
  __shared__ int s_parity;

  // expert as it is now; the copies start before the preceding kernel has finished
  const uint32_t e0 = md_ld_cg32(a.idx + entry);
  const bool v0 = e0 < (uint32_t)a.n_experts;
  auto issue = [&](uint32_t e) {
    st_mbar_expect_tx(mbar, (uint32_t)(2 * rows * RB));
    md_copy_tile(wbuf, a.wg + (long long)e * a.stride_g + (long long)f0 * RB, rows, RB, GS, mbar);
    md_copy_tile(wbuf + 4 * GS, a.wu + (long long)e * a.stride_u + (long long)f0 * RB, rows, RB, GS, mbar);
  };
  if (threadIdx.x == 0) {
    st_mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    if (v0) issue(e0);
  }
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const uint32_t e = md_ld_cg32(a.idx + entry);
  const bool valid = e < (uint32_t)a.n_experts;
  if (threadIdx.x == 0) {
    int parity = 0;
    bool ok = true;
    if (v0 && e != e0) {  // the first copy must land before its buffer is reused or the CTA leaves
      ok = md_wait(mbar, 0, error_word);
      parity = 1;
      if (valid && ok) issue(e);
    } else if (!v0 && valid) {
      issue(e);
    }
    s_parity = ok ? parity : -1;
  }
  __syncthreads();
  const int parity = s_parity;
  if (!valid || parity < 0) return;

  const XT* x = static_cast<const XT*>(a.x) + (long long)(entry / a.R) * K;
  for (int sb = warp; sb < nchunks; sb += kMdWarps)
    st_quantize<XT>(st_ld_cg16(x + sb * 256 + lane * 8), sb, lane, K, planes, XS, SX);
  __syncwarp();
  if (!md_wait(mbar, (uint32_t)parity, error_word)) return;

  const uint8_t* bplane = planes + min(g, 1) * K + 8 * t;
  const int lrA = min(4 * (g & 3) + (g >> 2), rows - 1), lrB = min(4 * (g & 3) + (g >> 2) + 2, rows - 1);
  const uint8_t* base[4] = {wbuf + (lrA >> 2) * GS + (lrA & 3) * RB, wbuf + (lrB >> 2) * GS + (lrB & 3) * RB,
                            wbuf + (4 + (lrA >> 2)) * GS + (lrA & 3) * RB, wbuf + (4 + (lrB >> 2)) * GS + (lrB & 3) * RB};
  float y4[4] = {0.f, 0.f, 0.f, 0.f};
  for (int sb = warp; sb < nchunks; sb += kMdWarps) {
    const uint8_t* const blk[4] = {base[0] + sb * 144, base[1] + sb * 144, base[2] + sb * 144, base[3] + sb * 144};
    st_unit<2>(blk, bplane + sb * 256, XS + sb * 8, SX[sb], t, y4);
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    y4[r] += __shfl_xor_sync(0xffffffffu, y4[r], 1);
    y4[r] += __shfl_xor_sync(0xffffffffu, y4[r], 2);
  }
  if (t == 0) {
    const int rA = 4 * (g & 3) + (g >> 2), rB = rA + 2;   // unclamped: rows past the tile are never read back
    red[warp * 32 + rA] = y4[0];
    red[warp * 32 + rB] = y4[1];
    red[warp * 32 + 16 + rA] = y4[2];
    red[warp * 32 + 16 + rB] = y4[3];
  }
  __syncthreads();
  if (threadIdx.x < rows) {
    float gs = 0.f, us = 0.f;
#pragma unroll
    for (int w = 0; w < kMdWarps; w++) {
      gs += red[w * 32 + threadIdx.x];
      us += red[w * 32 + 16 + threadIdx.x];
    }
    md_store(static_cast<XT*>(a.y) + (long long)entry * a.F + f0 + threadIdx.x, md_act(gs, us, a.act, a.limit));
  }
}

struct MixArgs {
  const void* x;            // [T * S, K]
  const uint8_t* w;
  long long stride_w;
  int row_bytes, K, N, S, n_experts;
  const uint32_t* idx;      // [T * S]
  const float* scores;      // [T * S]
  void* y;                  // [T, N]
};

// shared memory per warp: one 16-row tile (4 groups) | planes 2 K | XS | SX; then red 8 x 16 | 8 mbarriers
inline int mix_warp_bytes(int K, int row_bytes) {
  return 4 * md_group_stride(row_bytes) + 2 * K + (K / 32) * 4 + (((K / 256) + 3) & ~3) * 4;
}
inline int mix_smem_bytes(int K, int row_bytes) { return kMdWarps * mix_warp_bytes(K, row_bytes) + kMdWarps * 16 * 4 + kMdWarps * 8; }

template <typename XT>
__global__ void __launch_bounds__(kMdThreads, 2) moe_mix_kernel(const MixArgs a, int* __restrict__ error_word) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  extern __shared__ __align__(128) uint8_t md_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int K = a.K, nchunks = K >> 8, RB = a.row_bytes;
  const int gb = 4 * RB, GS = gb + ((32 - (gb & 127)) & 127);
  const int wbytes = 4 * GS + 2 * K + (K / 32) * 4 + ((nchunks + 3) & ~3) * 4;
  uint8_t* wbuf = md_dyn + warp * wbytes;
  uint8_t* planes = wbuf + 4 * GS;
  float* XS = reinterpret_cast<float*>(planes + 2 * K);
  float* SX = XS + (K / 32);
  float* red = reinterpret_cast<float*>(md_dyn + kMdWarps * wbytes);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(red + kMdWarps * 16) + warp;
  const int token = blockIdx.y, n0 = blockIdx.x * 16;
  const int rows = min(16, a.N - n0);
  const int lrA = min(4 * (g & 3) + (g >> 2), rows - 1), lrB = min(4 * (g & 3) + (g >> 2) + 2, rows - 1);
  const uint8_t* bplane = planes + min(g, 1) * K + 8 * t;
  const long long slot0 = (long long)token * a.S;

  auto issue = [&](uint32_t e) {
    st_mbar_expect_tx(mbar, (uint32_t)(rows * RB));
    md_copy_tile(wbuf, a.w + (long long)e * a.stride_w + (long long)n0 * RB, rows, RB, GS, mbar);
  };
  // first slot of this warp: its copy starts before the preceding kernel has finished
  uint32_t e0 = 0xffffffffu;
  if (warp < a.S) e0 = md_ld_cg32(a.idx + slot0 + warp);
  bool v0 = e0 < (uint32_t)a.n_experts;
  if (lane == 0) {
    st_mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    if (v0) issue(e0);
  }
  __syncwarp();
  asm volatile("griddepcontrol.wait;\n" ::: "memory");

  float yA = 0.f, yB = 0.f;   // score-weighted sums of this warp's slots (rows lrA, lrB), complete in lanes t = 0
  uint32_t parity = 0;
  bool dead = false;
  for (int s = warp; s < a.S; s += kMdWarps) {
    const uint32_t e = md_ld_cg32(a.idx + slot0 + s);
    const bool valid = e < (uint32_t)a.n_experts;
    // copies: the first slot's may already be in flight for another expert
    if (lane == 0) {
      bool ok = true;
      if (s == warp) {
        if (v0 && e != e0) {
          ok = md_wait(mbar, 0, error_word);
          if (ok && valid) issue(e);
        } else if (!v0 && valid) {
          issue(e);
        }
      } else if (valid) {
        issue(e);
      }
      if (!ok) atomicOr(error_word, 0x100);
    }
    if (s == warp && v0 && e != e0) parity ^= 1;
    __syncwarp();
    if (valid) {
      const XT* x = static_cast<const XT*>(a.x) + (slot0 + s) * K;
      for (int sb = 0; sb < nchunks; sb++)
        st_quantize<XT>(st_ld_cg16(x + sb * 256 + lane * 8), sb, lane, K, planes, XS, SX);
      __syncwarp();
      if (!md_wait(mbar, parity, error_word)) {
        dead = true;
        break;
      }
      parity ^= 1;
      const uint8_t* pA = wbuf + (lrA >> 2) * GS + (lrA & 3) * RB;
      const uint8_t* pB = wbuf + (lrB >> 2) * GS + (lrB & 3) * RB;
      float y2[2] = {0.f, 0.f};
      for (int sb = 0; sb < nchunks; sb++) {
        const uint8_t* const blk[2] = {pA + sb * 144, pB + sb * 144};
        st_unit<1>(blk, bplane + sb * 256, XS + sb * 8, SX[sb], t, y2);
      }
      const float sc = a.scores[slot0 + s];
      yA = fmaf(sc, y2[0], yA);
      yB = fmaf(sc, y2[1], yB);
      __syncwarp();   // the tile and the planes are free for the next slot
    }
  }
  yA += __shfl_xor_sync(0xffffffffu, yA, 1);
  yA += __shfl_xor_sync(0xffffffffu, yA, 2);
  yB += __shfl_xor_sync(0xffffffffu, yB, 1);
  yB += __shfl_xor_sync(0xffffffffu, yB, 2);
  if (t == 0) {
    const int rA = 4 * (g & 3) + (g >> 2);
    red[warp * 16 + rA] = yA;
    red[warp * 16 + rA + 2] = yB;
  }
  (void)dead;   // every copy that was started has been waited for above (the stale one by lane 0)
  __syncthreads();
  if (threadIdx.x < rows) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kMdWarps; w++) sum += red[w * 16 + threadIdx.x];
    md_store(static_cast<XT*>(a.y) + (long long)token * a.N + n0 + threadIdx.x, sum);
  }
}

// ---------------------------------------------------------------------------------- grouped by expert
// From a few dozen routed entries on, entries that share an expert share its weight stream: the entries are
// grouped by expert on the device (kq_gather.cu) and cut into tasks of 8 NT entries. The products are those of the dense
// kernel for few rows (kq_few.cu): integers as matrix operands, sixteen warps with a ring of TMA boxes each.
// All tasks' 16-row tiles stand in one row, CTA c of one per SM takes an even part of it, and within a task the units
// (tile, superblock) are shared evenly by the warps. Tiles that a warp has whole leave from its registers, the others meet
// in shared memory. The gate and the up rows of the same features are a unit together, so that the activation function is
// applied to float32 sums. Boxes of the next task are on their way while a task's activations are staged.
// Measured on B200, 512 entries of 128 experts, K 2048, F 768 (226 MB and 113 MB of weights): gate | up 109 -> 74 us, down
// 51 -> 43 (before: tasks of sixteen entries, four at a time as byte planes in int8 operands, a CTA for 64 features, whose
// ten microseconds of serial latencies two CTAs an SM did not hide).
template <int NT>
struct Tasks {
  int expert, m;
  int ent[8 * NT];   // entry indices; slots past m repeat the last one
};

struct TaskArgs {
  const void* x;            // entry b's row is b / R
  int K, F, R;              // F: rows of a matrix (of gate and of up each)
  const uint8_t *wg, *wu;   // wu: nullptr in the form of one matrix
  long long stride_g, stride_u;
  int row_bytes;
  void* y;                  // [entries, F]
  int act;
  float limit;
  int D;                    // slots of a warp
  int x_pitch, x_off, sum_off, red_off;
};

constexpr int kTkWarps = 16, kTkThreads = 32 * kTkWarps, kTkMaxSlots = 4, kTkSlot = 16 * 144;
constexpr int kTkSmem = 226 * 1024 - 512;

__device__ __forceinline__ void tk_load(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

template <typename XT, int NT, bool GLU>
__global__ void __launch_bounds__(kTkThreads, 1)
moe_tasks_product_kernel(const TaskArgs a, const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_u,
                         const Tasks<NT>* tasks, const int* n_tasks, int* __restrict__ error_word) {
  // (tasks, n_tasks: not __restrict__, whose loads may be moved ahead of griddepcontrol.wait)
  constexpr int H = GLU ? 2 : 1;                       // matrices
  constexpr int kRedPitch = 8 * NT + (NT == 1 ? 2 : 0);
  constexpr int kSumWords = NT * 8 * rw_sum_pitch(Q4_K);
  extern __shared__ __align__(128) uint8_t tk_dyn[];
  __shared__ uint64_t full[kTkWarps][kTkMaxSlots];
  __shared__ int abort_s, ent_s[8 * NT];
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nsb = a.K >> 8, D = a.D, nt = (a.F + 15) >> 4;
  if (threadIdx.x == 0) abort_s = 0;
  if (lane == 0) {
    for (int d = 0; d < D; d++) mbar_init(&full[warp][d], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  volatile int* abort_flag = &abort_s;
  uint8_t* const ring = tk_dyn + warp * D * kTkSlot;
  uint8_t* const xs = tk_dyn + a.x_off;
  float* const sums = reinterpret_cast<float*>(tk_dyn + a.sum_off);
  float* const red = reinterpret_cast<float*>(tk_dyn + a.red_off);  // [warp][first tile, last][matrix][16][kRedPitch]
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const long long total = (long long)*n_tasks * nt;
  const int t0 = (int)(total * blockIdx.x / gridDim.x), t1 = (int)(total * (blockIdx.x + 1) / gridDim.x);  // this CTA's tiles
  auto end_of = [&](int from) { return min(t1, (from / nt + 1) * nt); };  // of the tiles of a task

  // boxes: the next one of this warp's share
  int is_from = t0, is_d = 0, is_row = 0, is_sb = 0, is_half = 0, is_left = 0, is_expert = 0;
  auto open = [&]() {  // the share in the tasks from is_from on
    while (is_left == 0 && is_from < t1) {
      const int end = end_of(is_from), all = (end - is_from) * nsb, u0 = (warp * all) >> 4, u1 = ((warp + 1) * all) >> 4;
      if (u1 > u0) {
        const int tile = u0 / nsb, task = is_from / nt;
        is_row = 16 * (is_from - task * nt + tile);
        is_sb = u0 - tile * nsb;
        is_left = u1 - u0;
        is_expert = tasks[task].expert;
      }
      is_from = end;
    }
  };
  auto issue = [&]() {
    if (is_left == 0) return;
    if (lane == 0) {
      mbar_expect_tx(&full[warp][is_d], kTkSlot);
      tk_load(smem_u32(ring + is_d * kTkSlot), GLU && is_half ? &map_u : &map_g, 144 * is_sb, is_row, is_expert, &full[warp][is_d]);
    }
    if (++is_d == D) is_d = 0;
    if (GLU && is_half == 0) {
      is_half = 1;
      return;
    }
    is_half = 0;
    if (++is_sb == nsb) is_sb = 0, is_row += 16;
    if (--is_left == 0) open();
  };

  int d = 0;
  uint32_t par = 0;
  bool ok = true, begun = false;
  for (int from = t0, end; from < t1; from = end) {
    end = end_of(from);
    const int task = from / nt, tile0 = from - task * nt, expert = tasks[task].expert, m = tasks[task].m;
    const int all = (end - from) * nsb;
    auto cut = [&](int w) { return (w * all) >> 4; };  // the first unit of warp w
    __syncthreads();  // the activations and the partial sums of the task before have been read
    if (threadIdx.x < 8 * NT) ent_s[threadIdx.x] = tasks[task].ent[threadIdx.x];
    for (int i = warp; i < m; i += kTkWarps) {
      const XT* src = static_cast<const XT*>(a.x) + (long long)(tasks[task].ent[i] / a.R) * a.K;
      const uint32_t dst = smem_u32(xs + i * a.x_pitch);
      for (int c = lane; c < 32 * nsb; c += 32) rw_cp16(dst + 16 * c, src + 8 * c);
    }
    if (!begun) {
      begun = true;
      open();
      for (int i = 0; i < D; i++) issue();
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    for (int e = warp; e < nsb * NT; e += kTkWarps) {
      const int k = e / NT, n = e % NT;
      if (8 * n < m)
        rows_sums<Q4_K, XT>(xs + min(8 * n + g, m - 1) * a.x_pitch + 512 * k, sums + (k * NT + n) * 8 * rw_sum_pitch(Q4_K), lane);
    }
    __syncthreads();

    auto finish = [&](int row, int c, float vg, float vu) {  // row of the matrix, activation row of the task
      if (row >= a.F || c >= m) return;
      const int entry = ent_s[c];
      if (!(fabsf(vg) < INFINITY) || (GLU && !(fabsf(vu) < INFINITY))) {
        const XT* xr = static_cast<const XT*>(a.x) + (long long)(entry / a.R) * a.K;
        vg = rows_plain<Q4_K, XT>(a.wg + (long long)expert * a.stride_g + (long long)row * a.row_bytes, xr, nsb);
        if (GLU) vu = rows_plain<Q4_K, XT>(a.wu + (long long)expert * a.stride_u + (long long)row * a.row_bytes, xr, nsb);
      }
      md_store(static_cast<XT*>(a.y) + (long long)entry * a.F + row, GLU ? md_act(vg, vu, a.act, a.limit) : vg);
    };

    const int u0 = cut(warp), u1 = cut(warp + 1);
    float y[H][NT][4];
#pragma unroll
    for (int h = 0; h < H; h++)
#pragma unroll
      for (int n = 0; n < NT; n++) y[h][n][0] = y[h][n][1] = y[h][n][2] = y[h][n][3] = 0.f;
    int tile = u0 / nsb, sb = u0 - tile * nsb, second = 0;
    bool whole = sb == 0;
    for (int u = u0; u < u1; u++) {
      const uint8_t* xb[NT];
#pragma unroll
      for (int n = 0; n < NT; n++) xb[n] = xs + min(8 * n + g, m - 1) * a.x_pitch + 512 * sb;
#pragma unroll
      for (int h = 0; h < H; h++) {
        if (ok) ok = mbar_wait_err(&full[warp][d], par, abort_flag, 0x500, error_word);
        if (ok) {
          const uint8_t* r0 = ring + d * kTkSlot + g * 144;
          if (NT == 1 || m > 8) {
            RowsUnit<Q4_K, XT, NT>::run(y[h], r0, r0 + 8 * 144, xb, sums + sb * kSumWords, g, t);
          } else {
            const uint8_t* xb1[1] = {xb[0]};
            float y1[1][4] = {{y[h][0][0], y[h][0][1], y[h][0][2], y[h][0][3]}};
            RowsUnit<Q4_K, XT, 1>::run(y1, r0, r0 + 8 * 144, xb1, sums + sb * kSumWords, g, t);
            y[h][0][0] = y1[0][0], y[h][0][1] = y1[0][1], y[h][0][2] = y1[0][2], y[h][0][3] = y1[0][3];
          }
        }
        __syncwarp();  // the slot has been read
        issue();
        if (++d == D) d = 0, par ^= 1;
      }
      if (++sb < nsb && u + 1 < u1) continue;
      if (whole && sb == nsb) {
        if (ok) {
          const int row = 16 * (tile0 + tile) + g;
#pragma unroll
          for (int n = 0; n < NT; n++)
#pragma unroll
            for (int i = 0; i < 4; i++)
              finish(row + (i >> 1) * 8, 8 * n + 2 * t + (i & 1), y[0][n][i], y[H - 1][n][i]);
        }
      } else {
#pragma unroll
        for (int h = 0; h < H; h++) {
          float* mine = red + (((2 * warp + second) * H + h) * 16 + g) * kRedPitch + 2 * t;
#pragma unroll
          for (int n = 0; n < NT; n++) {
            *reinterpret_cast<float2*>(mine + 8 * n) = make_float2(y[h][n][0], y[h][n][1]);
            *reinterpret_cast<float2*>(mine + 8 * kRedPitch + 8 * n) = make_float2(y[h][n][2], y[h][n][3]);
          }
        }
      }
      sb = 0, tile++, second = 1, whole = true;
#pragma unroll
      for (int h = 0; h < H; h++)
#pragma unroll
        for (int n = 0; n < NT; n++) y[h][n][0] = y[h][n][1] = y[h][n][2] = y[h][n][3] = 0.f;
    }
    __syncthreads();
    // tiles that a cut between two warps goes through, the parts in order
    if (abort_s == 0) {
      for (int i = threadIdx.x; i < (kTkWarps - 1) * 16 * m; i += kTkThreads) {
        const int w = 1 + i / (16 * m), at = i - (w - 1) * 16 * m, place = at & 15, c = at >> 4;
        const int tl = cut(w) / nsb, u = tl * nsb;
        if (cut(w) == u || cut(w - 1) > u) continue;  // no tile is cut here, or it was cut before
        float v[2] = {0.f, 0.f};
        for (int q = w - 1; q < kTkWarps && cut(q) < u + nsb; q++) {
          if (cut(q + 1) <= u || cut(q + 1) == cut(q)) continue;
          const float* part = red + ((2 * q + (cut(q) / nsb == tl ? 0 : 1)) * H * 16 + place) * kRedPitch + c;
          v[0] += part[0];
          if (GLU) v[1] += part[16 * kRedPitch];
        }
        finish(16 * (tile0 + tl) + place, c, v[0], v[1]);
      }
    }
  }
  if (abort_s != 0) {  // given up: what is in flight lands long before this
    const unsigned long long since = globaltimer_ns();
    while (globaltimer_ns() - since < 1000000ull) {
    }
  }
}

// ------------------------------------------------------------------------------------------------ router
struct RouterArgs {
  const void* logits;       // [T, E + shared]
  int dtype, T, E, top_k, norm, shared, scoring;
  const float* pes;         // per-expert scale [E] or nullptr
  const float* bias;        // selection bias [E] or nullptr
  float scale;
  uint32_t* indices;        // [T, top_k]
  float* scores;            // [T, top_k + shared]
};

__device__ __forceinline__ float md_logit(const void* p, int dtype, long long i) {
  if (dtype == F32) return static_cast<const float*>(p)[i];
  if (dtype == F16) return __half2float(static_cast<const __half*>(p)[i]);
  return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}

// One warp per token; lane l holds experts l, l + 32, ... (E <= 32 NI: at most NI per lane). With arrays of 32 whatever
// E, the arg-max rounds over 128 experts spent seven of eight comparisons on places that hold none (4096 tokens, top 8:
// 21 us).
template <int NI>
__global__ void __launch_bounds__(256) router_topk_kernel(const RouterArgs a) {
  // the kernel that consumes the indices may start its prologue now; it reads them again after this grid is done
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= a.T) return;
  const long long row = (long long)token * (a.E + a.shared);
  float p[NI], rk[NI];
  float gsum = 1.f;
  if (a.scoring == 1) {   // sqrt(softplus(x)), softplus in its overflow-free form
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int e = lane + 32 * i;
      float v = -INFINITY;
      if (e < a.E) {
        const float x = md_logit(a.logits, a.dtype, row + e);
        v = sqrtf(fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))));
      }
      p[i] = v;
    }
  } else {
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int e = lane + 32 * i;
      p[i] = e < a.E ? md_logit(a.logits, a.dtype, row + e) : -INFINITY;
      m = fmaxf(m, p[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int e = lane + 32 * i;
      const float v = e < a.E ? expf(p[i] - m) : 0.f;
      p[i] = e < a.E ? v : -INFINITY;
      s += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    gsum = s;
  }
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int e = lane + 32 * i;
    rk[i] = (a.bias != nullptr && e < a.E) ? p[i] + a.bias[e] : p[i];
  }
  float win_v = 0.f;        // lane r keeps the r-th winner
  uint32_t win_i = 0;
  float psum = 0.f;
  for (int r = 0; r < a.top_k; r++) {
    float bv = -INFINITY;
    uint32_t bi = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < NI; i++) {   // ascending expert index within the lane: '>' keeps the lowest on ties
      if (rk[i] > bv) {
        bv = rk[i];
        bi = (uint32_t)(lane + 32 * i);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) {
        bv = ov;
        bi = oi;
      }
    }
    // the emitted score is the unbiased one; its owner lane removes the expert from the ranking
    float pv = 0.f;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      if ((uint32_t)(lane + 32 * i) == bi) {
        pv = p[i];
        rk[i] = -INFINITY;
      }
    }
    pv = __shfl_sync(0xffffffffu, pv, bi & 31);
    psum += pv;
    if (lane == r) {
      win_v = pv;
      win_i = bi;
    }
  }
  const float denom = a.norm ? (a.scoring == 1 ? psum + 1e-20f : psum) : gsum;
  if (lane < a.top_k) {
    float sv = win_v / denom;
    if (a.pes != nullptr && win_i < (uint32_t)a.E) sv *= a.pes[win_i];
    a.indices[(long long)token * a.top_k + lane] = win_i;
    a.scores[(long long)token * (a.top_k + a.shared) + lane] = sv * a.scale;
  }
  if (a.shared && lane == 0)
    a.scores[(long long)token * (a.top_k + 1) + a.top_k] = 1.f / (1.f + expf(-md_logit(a.logits, a.dtype, row + a.E)));
}

template <typename KernelT>
cudaError_t md_set_smem(KernelT kern, int bytes, bool (&done)[16]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
  if (!done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    done[dev] = true;
  }
  return cudaSuccess;
}

constexpr int kMdMaxSmem = 200 * 1024;

template <typename KernelT, typename ArgsT>
cudaError_t md_launch(KernelT kern, dim3 grid, int smem, const ArgsT& a, cudaStream_t st) {
  int* err = device_error_word();
  if (err == nullptr) return cudaErrorUnknown;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kMdThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  static const bool no_pdl = std::getenv("KQ_NO_PDL") != nullptr;  // A/B lever
  cfg.numAttrs = no_pdl ? 0 : 1;
  return cudaLaunchKernelEx(&cfg, kern, a, err);
}

}  // namespace

// ---- grouped forms: scratch = grouping arrays + task list (+ the per-entry products of the down stage)
struct MoeWs {
  size_t counts, cursor, offsets, task_base, n_tasks, order, tasks, d, total;
  long long max_tasks;
};
static MoeWs moe_ws_layout(long long n_entries, int n_experts, long long d_bytes) {
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  MoeWs L{};
  const size_t e1 = (size_t)(n_experts + 1) * 4;
  L.counts = 0;
  L.cursor = e1;
  L.offsets = 2 * e1;
  L.task_base = 3 * e1;
  L.n_tasks = 4 * e1;
  L.order = up(4 * e1 + 4);
  L.max_tasks = n_entries / 16 + n_experts + 1;
  L.tasks = up(L.order + (size_t)n_entries * 4);
  L.d = up(L.tasks + (size_t)L.max_tasks * sizeof(Tasks<2>));
  L.total = up(L.d + (size_t)d_bytes);
  return L;
}

size_t moe_grouped_workspace_bytes(long long n_entries, int n_experts, long long d_bytes) {
  return moe_ws_layout(n_entries, n_experts, d_bytes).total;
}

// Tasks of eight entries where experts have few, of sixteen where a good part of them has more than eight. (Those of eight
// fit into the room of the others: 40 (n / 8 + E) <= 72 (n / 16 + E).) Both products of a call see the same sizes here.
static bool moe_small_tasks(long long n_entries, int n_experts) { return n_entries <= 5ll * n_experts; }

static cudaError_t moe_build_tasks(const uint32_t* idx, long long n_entries, int n_experts, uint8_t* ws, const MoeWs& L,
                                   cudaStream_t st) {
  return launch_group_by_expert(idx, n_entries, n_experts, moe_small_tasks(n_entries, n_experts) ? 8 : 16,
                                reinterpret_cast<int*>(ws + L.counts), reinterpret_cast<int*>(ws + L.cursor),
                                reinterpret_cast<int*>(ws + L.offsets), reinterpret_cast<int*>(ws + L.task_base),
                                reinterpret_cast<int*>(ws + L.n_tasks), reinterpret_cast<int*>(ws + L.order),
                                reinterpret_cast<int*>(ws + L.tasks), st);
}

// all experts' rows of one matrix
static cudaError_t md_map(CUtensorMap* map, const uint8_t* w, long long row_bytes, int F, int n_experts, long long stride) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (enc == nullptr) return cudaErrorNotSupported;
  const cuuint64_t dims[3] = {(cuuint64_t)row_bytes, (cuuint64_t)F, (cuuint64_t)n_experts};
  const cuuint64_t strides[2] = {(cuuint64_t)row_bytes, (cuuint64_t)stride};
  const cuuint32_t box[3] = {144u, 16u, 1u}, estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(w), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// shared memory: rings | activations | their sums | partial sums; false where a slot of a matrix and one more do not fit
template <int NT, bool GLU>
static bool md_plan(TaskArgs& a, int& smem) {
  const int nsb = a.K >> 8;
  a.x_pitch = 2 * a.K + 64;
  const int x = 8 * NT * a.x_pitch, sum = nsb * NT * 8 * rw_sum_pitch(Q4_K) * 4;
  const int red = kTkWarps * 2 * (GLU ? 2 : 1) * 16 * (8 * NT + (NT == 1 ? 2 : 0)) * 4;
  a.D = std::min(kTkMaxSlots, (kTkSmem - x - sum - red) / (kTkWarps * kTkSlot));
  if (kTkSmem - x - sum - red < 0 || a.D < 2) return false;
  a.x_off = a.D * kTkWarps * kTkSlot;
  a.sum_off = a.x_off + x;
  a.red_off = a.sum_off + sum;
  smem = a.red_off + red;
  return true;
}

template <typename XT, int NT, bool GLU>
static cudaError_t md_launch_product(TaskArgs a, int n_experts, const void* tasks, const int* n_tasks, cudaStream_t st) {
  int smem = 0;
  if (!md_plan<NT, GLU>(a, smem)) return cudaErrorInvalidConfiguration;  // (not reached: moe_grouped_supported)
  int* err = device_error_word();
  if (err == nullptr) return cudaErrorUnknown;
  static bool done[16] = {};
  cudaError_t e = md_set_smem(moe_tasks_product_kernel<XT, NT, GLU>, kTkSmem, done);
  if (e != cudaSuccess) return e;
  alignas(64) CUtensorMap mg{}, mu{};
  if ((e = md_map(&mg, a.wg, a.row_bytes, a.F, n_experts, a.stride_g)) != cudaSuccess) return e;
  if (GLU && (e = md_map(&mu, a.wu, a.row_bytes, a.F, n_experts, a.stride_u)) != cudaSuccess) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms);
  cfg.blockDim = dim3(kTkThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, moe_tasks_product_kernel<XT, NT, GLU>, a, mg, mu, static_cast<const Tasks<NT>*>(tasks), n_tasks, err);
}
template <bool GLU>
static cudaError_t md_launch_products(int x_dtype, const TaskArgs& a, long long n_entries, int n_experts, const void* tasks,
                                      const int* n_tasks, cudaStream_t st) {
  if (moe_small_tasks(n_entries, n_experts))
    return x_dtype == F16 ? md_launch_product<__half, 1, GLU>(a, n_experts, tasks, n_tasks, st)
                          : md_launch_product<__nv_bfloat16, 1, GLU>(a, n_experts, tasks, n_tasks, st);
  return x_dtype == F16 ? md_launch_product<__half, 2, GLU>(a, n_experts, tasks, n_tasks, st)
                        : md_launch_product<__nv_bfloat16, 2, GLU>(a, n_experts, tasks, n_tasks, st);
}

// the grouping alone (for a caller whose own grouped kernel does not apply but whose workspace is handed on)
cudaError_t launch_moe_grouping_only(const uint32_t* idx, long long n_entries, int n_experts, void* workspace,
                                     cudaStream_t st) {
  const MoeWs L = moe_ws_layout(n_entries, n_experts, 0);
  return moe_build_tasks(idx, n_entries, n_experts, static_cast<uint8_t*>(workspace), L, st);
}

// The limits of the kernels before these, whose rows and tiles had to fit twice into shared memory; md_plan has room for longer
// rows, and the grouped mix is the faster one there too (512 entries of 128 experts, K 1536: 377 us entry by entry, 81 grouped;
// 32 experts, K 2048, 256 entries: 712 and 77). But it rounds every slot's product to 16 bits before the weighted sum, which the
// other form does not, so that calls that have had one rounding keep it.
bool moe_grouped_supported(int K, bool rows_kernel) {
  return K <= (rows_kernel ? 1280 : 2304);
}

cudaError_t launch_moe_glu_grouped(int x_dtype, const void* x, int K, const uint8_t* wg, long long stride_g,
                                   const uint8_t* wu, long long stride_u, long long row_bytes, int F, int n_experts,
                                   const uint32_t* idx, long long n_entries, int R, int act, float limit, void* y,
                                   void* workspace, cudaStream_t st) {
  if (n_entries <= 0 || F <= 0) return cudaSuccess;
  const MoeWs L = moe_ws_layout(n_entries, n_experts, 0);
  if (L.max_tasks > 65535) return cudaErrorInvalidConfiguration;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  cudaError_t e = moe_build_tasks(idx, n_entries, n_experts, ws, L, st);
  if (e != cudaSuccess) return e;
  TaskArgs a{};
  a.x = x, a.K = K, a.F = F, a.R = R;
  a.wg = wg, a.wu = wu, a.stride_g = stride_g, a.stride_u = stride_u, a.row_bytes = (int)row_bytes;
  a.y = y, a.act = act, a.limit = limit;
  return md_launch_products<true>(x_dtype, a, n_entries, n_experts, ws + L.tasks, reinterpret_cast<const int*>(ws + L.n_tasks), st);
}

// d[b] = x[b] . W[idx[b]]^T for every entry b (entries grouped by expert), then y[t] = sum_s scores[t, s] d[t S + s]
cudaError_t launch_moe_mix_grouped(int x_dtype, const void* x, int K, const uint8_t* w, long long stride_w,
                                   long long row_bytes, int N, int n_experts, const uint32_t* idx, const float* scores,
                                   long long T, int S, void* y, void* workspace, bool reuse_grouping,
                                   cudaStream_t st) {
  const long long n_entries = T * S;
  if (n_entries <= 0 || N <= 0) return cudaSuccess;
  const MoeWs L = moe_ws_layout(n_entries, n_experts, n_entries * (long long)N * 2);
  if (L.max_tasks > 65535) return cudaErrorInvalidConfiguration;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  cudaError_t e = cudaSuccess;
  // reuse_grouping: the workspace still holds the task list that launch_moe_glu_grouped built from these indices
  if (!reuse_grouping && (e = moe_build_tasks(idx, n_entries, n_experts, ws, L, st)) != cudaSuccess) return e;
  TaskArgs a{};
  a.x = x, a.K = K, a.F = N, a.R = 1;
  a.wg = w, a.stride_g = stride_w, a.row_bytes = (int)row_bytes;
  a.y = ws + L.d;
  e = md_launch_products<false>(x_dtype, a, n_entries, n_experts, ws + L.tasks, reinterpret_cast<const int*>(ws + L.n_tasks), st);
  if (e != cudaSuccess) return e;
  // entries of experts out of range get no task: the weighted sum does not read their d rows (with rows of zeros instead, the
  // memset between the two products kept them apart)
  return launch_moe_combine(x_dtype, ws + L.d, scores, T, S, N, y, false, st, idx, (uint32_t)n_experts);
}

bool moe_decode_supported(int codec, int x_dtype, int K, long long row_bytes, const void* x, const void* w0,
                          long long stride0, const void* w1, long long stride1) {
  if (codec != Q4_K || (x_dtype != F16 && x_dtype != BF16)) return false;
  if (K < 256 || (K & 255) != 0 || row_bytes != (long long)(K >> 8) * 144) return false;
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return false;
  if ((reinterpret_cast<uintptr_t>(w0) & 15) != 0 || (stride0 & 15) != 0) return false;
  if (w1 != nullptr && ((reinterpret_cast<uintptr_t>(w1) & 15) != 0 || (stride1 & 15) != 0)) return false;
  return glu_smem_bytes(K, (int)row_bytes) <= kMdMaxSmem && mix_smem_bytes(K, (int)row_bytes) <= kMdMaxSmem;
}

cudaError_t launch_moe_glu(int x_dtype, const void* x, int K, const uint8_t* wg, long long stride_g, const uint8_t* wu,
                           long long stride_u, long long row_bytes, int F, int n_experts, const uint32_t* idx,
                           long long n_entries, int R, int act, float limit, void* y, cudaStream_t st) {
  if (n_entries <= 0 || F <= 0) return cudaSuccess;
  if (n_entries > 65535) return cudaErrorInvalidConfiguration;
  GluArgs a{x, wg, wu, stride_g, stride_u, (int)row_bytes, K, F, R, (int)n_entries, n_experts, idx, y, act, limit};
  const int smem = glu_smem_bytes(K, (int)row_bytes);
  const dim3 grid((F + 15) / 16, (unsigned)n_entries, 1);
  static bool done_h[16] = {}, done_b[16] = {};
  cudaError_t e;
  if (x_dtype == F16) {
    if ((e = md_set_smem(moe_glu_kernel<__half>, kMdMaxSmem, done_h)) != cudaSuccess) return e;
    return md_launch(moe_glu_kernel<__half>, grid, smem, a, st);
  }
  if ((e = md_set_smem(moe_glu_kernel<__nv_bfloat16>, kMdMaxSmem, done_b)) != cudaSuccess) return e;
  return md_launch(moe_glu_kernel<__nv_bfloat16>, grid, smem, a, st);
}

cudaError_t launch_moe_mix(int x_dtype, const void* x, int K, const uint8_t* w, long long stride_w, long long row_bytes,
                           int N, int n_experts, const uint32_t* idx, const float* scores, long long T, int S, void* y,
                           cudaStream_t st) {
  if (T <= 0 || N <= 0) return cudaSuccess;
  if (T > 65535) return cudaErrorInvalidConfiguration;
  MixArgs a{x, w, stride_w, (int)row_bytes, K, N, S, n_experts, idx, scores, y};
  const int smem = mix_smem_bytes(K, (int)row_bytes);
  const dim3 grid((N + 15) / 16, (unsigned)T, 1);
  static bool done_h[16] = {}, done_b[16] = {};
  cudaError_t e;
  if (x_dtype == F16) {
    if ((e = md_set_smem(moe_mix_kernel<__half>, kMdMaxSmem, done_h)) != cudaSuccess) return e;
    return md_launch(moe_mix_kernel<__half>, grid, smem, a, st);
  }
  if ((e = md_set_smem(moe_mix_kernel<__nv_bfloat16>, kMdMaxSmem, done_b)) != cudaSuccess) return e;
  return md_launch(moe_mix_kernel<__nv_bfloat16>, grid, smem, a, st);
}

cudaError_t launch_router_topk(const void* logits, int dtype, int T, int E, int top_k, int norm, int shared, int scoring,
                               const float* pes, const float* bias, float scale, uint32_t* indices, float* scores,
                               cudaStream_t st) {
  if (T <= 0) return cudaSuccess;
  RouterArgs a{logits, dtype, T, E, top_k, norm, shared, scoring, pes, bias, scale, indices, scores};
  const int warps = T <= 4 * 148 ? 2 : 8;  // few tokens: spread over the SMs
  auto kern = E <= 128 ? router_topk_kernel<4> : E <= 256 ? router_topk_kernel<8> : router_topk_kernel<32>;
  kern<<<(T + warps - 1) / warps, 32 * warps, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace kq
