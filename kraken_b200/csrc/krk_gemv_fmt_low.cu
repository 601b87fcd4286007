// Streaming GEMV kernels of Q2_K (krk_gemv_stream.cuh).
#include "krk_gemv_stream.cuh"

namespace krk_cuda {
namespace stream {
KRK_STREAM_FORMAT(, KRK_CUDA_Q2_K)
} // namespace stream
} // namespace krk_cuda
