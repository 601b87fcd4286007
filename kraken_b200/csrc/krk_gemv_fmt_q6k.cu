// Streaming GEMV kernels of Q6_K (krk_gemv_stream.cuh).
#include "krk_gemv_stream.cuh"

namespace krk_cuda {
namespace stream {
KRK_STREAM_FORMAT(, KRK_CUDA_Q6_K)
} // namespace stream
} // namespace krk_cuda
