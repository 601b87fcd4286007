// Streaming GEMV kernels of Q5_K, IQ4_NL (krk_gemv_stream.cuh).
#include "krk_gemv_stream.cuh"

namespace krk_cuda {
namespace stream {
KRK_STREAM_FORMAT(, KRK_CUDA_Q5_K)
KRK_STREAM_FORMAT(, KRK_CUDA_IQ4_NL)
} // namespace stream
} // namespace krk_cuda
