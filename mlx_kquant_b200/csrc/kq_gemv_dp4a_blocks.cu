// The integer dot-product decode kernels (kq_gemv_dp4a.cuh) of the codecs with blocks of 32 and of the table codecs.
#include "kq_gemv_dp4a.cuh"

namespace kq {

cudaError_t launch_gemv_dp4a_blocks(int codec, int x_dtype, const GemvArgs& a, cudaStream_t st) {
  switch (codec) {
    case Q4_0: return launch_codec<Q4_0>(x_dtype, a, st);
    case Q8_0: return launch_codec<Q8_0>(x_dtype, a, st);
    case IQ4_NL: return launch_codec<IQ4_NL>(x_dtype, a, st);
    case IQ4_XS: return launch_codec<IQ4_XS>(x_dtype, a, st);
    case IQ2_XXS: return launch_codec<IQ2_XXS>(x_dtype, a, st);
    case Q4_1: return launch_codec<Q4_1>(x_dtype, a, st);
    case Q5_0: return launch_codec<Q5_0>(x_dtype, a, st);
    case Q5_1: return launch_codec<Q5_1>(x_dtype, a, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kq
