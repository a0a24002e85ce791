// The integer dot-product decode kernels (kq_gemv_dp4a.cuh): which calls take them, and those of the K-quants.
#include "kq_gemv_dp4a.cuh"

namespace kq {

bool gemv_dp4a_supported(int codec, int x_dtype, const GemvArgs& a) {
  if (codec > Q5_1) return false;   // the codecs added after the integer kernels were written use the generic path
  if (!a.w_align16 || (a.K & 255) != 0 || a.K > kMaxK) return false;
  if ((a.row_bytes & 15) != 0 && (a.tasks != nullptr || !ragged_rows(codec) || (a.row_bytes & 1) != 0)) return false;
  if ((a.row_bytes & 15) == 0 && a.row_bytes < 16 * 17) return false;
  if (a.tasks != nullptr) {
    // task lists (gather_qmm): rows in slices of four. q4_k with fp16 rows and the two table codecs keep
    // their tensor-core kernels, which take sixteen rows per pass over the weights.
    if ((codec == Q4_K && x_dtype == F16) || codec == IQ4_XS || codec == IQ2_XXS) return false;
    if (a.n_tasks > 65535) return false;
    // measured on a 128-expert block: a win at ~4 rows per expert, a loss at 16 (every four-row slice
    // streams the expert's weights again)
    if (a.avg_rows > 4) return false;
    return 4 * x_bytes(a.K) <= 96 * 1024;
  }
  if (codec == Q4_K) return false;  // dense q4_k has its own kernels (kq_gemv.cu)
  if (codec > Q5_1) return false;   // the codecs added after the integer kernels were written use the generic path
  if (a.M < 1 || a.M > 4) return false;
  // measured: with more than one row the table-driven tensor-core kernels of kq_gemv.cu win for these two,
  // and so they do for iq2_xxs matrices too small to hide the lattice lookups
  if ((codec == IQ4_XS || codec == IQ2_XXS) && a.M > 1) return false;
  if (codec == IQ2_XXS && (long long)a.N * a.K < (48ll << 20)) return false;
  // the activations of all rows are staged whole: 2.6 bytes per activation
  const int mt = a.M == 3 ? 4 : a.M;
  return mt * x_bytes(a.K) <= 96 * 1024;
}

cudaError_t launch_gemv_dp4a_blocks(int codec, int x_dtype, const GemvArgs& a, cudaStream_t st);  // the other codecs

cudaError_t launch_gemv_dp4a(int codec, int x_dtype, const GemvArgs& a, cudaStream_t st) {
  switch (codec) {
    case Q2_K: return launch_codec<Q2_K>(x_dtype, a, st);
    case Q3_K: return launch_codec<Q3_K>(x_dtype, a, st);
    case Q4_K: return launch_codec<Q4_K>(x_dtype, a, st);
    case Q5_K: return launch_codec<Q5_K>(x_dtype, a, st);
    case Q6_K: return launch_codec<Q6_K>(x_dtype, a, st);
  }
  return launch_gemv_dp4a_blocks(codec, x_dtype, a, st);
}

}  // namespace kq
