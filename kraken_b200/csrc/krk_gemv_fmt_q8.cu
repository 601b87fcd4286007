// Streaming GEMV kernels of Q8_0, Q5_1 (krk_gemv_stream.cuh).
#include "krk_gemv_stream.cuh"

namespace krk_cuda {
namespace stream {
KRK_STREAM_FORMAT(, KRK_CUDA_Q8_0)
KRK_STREAM_FORMAT(, KRK_CUDA_Q5_1)
} // namespace stream
} // namespace krk_cuda
