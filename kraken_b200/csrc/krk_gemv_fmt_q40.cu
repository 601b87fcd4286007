// Streaming GEMV kernels of Q4_0, Q5_0 (krk_gemv_stream.cuh).
#include "krk_gemv_stream.cuh"

namespace krk_cuda {
namespace stream {
KRK_STREAM_FORMAT(, KRK_CUDA_Q4_0)
KRK_STREAM_FORMAT(, KRK_CUDA_Q5_0)
} // namespace stream
} // namespace krk_cuda
