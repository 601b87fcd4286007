// Entry points of the streaming decode GEMV (krk_gemv_stream.cuh): dispatch by weight type.
#include "krk_gemv_stream.cuh"

namespace krk_cuda {

namespace stream {
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q4_K)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q6_K)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q8_0)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q4_0)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q5_K)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q2_K)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q3_K)
KRK_STREAM_FORMAT(extern, KRK_CUDA_IQ4_NL)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q5_0)
KRK_STREAM_FORMAT(extern, KRK_CUDA_Q5_1)
} // namespace stream

// One warp: lane q waits (bounded) until flag[q] has reached `epoch`, i.e. until peer q has stored its
// slice of the row into this GPU's buffer. A wait that gives up raises the device status word.
static __global__ void __launch_bounds__(32) flag_wait_kernel(const int *flags, int n, int epoch, int *status) {
    const int q = threadIdx.x;
    if (q < n) {
        const long long t0 = clock64();
        while (*reinterpret_cast<const volatile int *>(flags + q) < epoch) {
            __nanosleep(200);
            if (clock64() - t0 > stream::kWaitCycles) {
                atomicExch(status, KRK_CUDA_ETIMEOUT);
                break;
            }
        }
    }
    __threadfence_system();
}

// Activation rows whose limbs leave no room for a ring, K a multiple of 256: half of them at a time, or half of those, with four
// limbs: 30 bits below the largest activation of a warp's slices, sums of activations (formats with a minimum) in eighths of the
// 22nd. The warp-per-row kernel, which had these shapes, multiplies in f32: it keeps 24 bits of every activation, however small, but
// adds up in more steps, and its results are no nearer the f64 sums (530 weight rows, normal activations and with every 97th 300
// times as large, worst of twelve: 12544 values, six rows 0.7e-7 to 1.2e-7 here, 1.4e-7 to 1.7e-7 there; 21504, three rows 0.9e-7 to
// 1.4e-7, 1.5e-7 to 1.9e-7; 22 bits 2.6e-7 and eight times that. Q2_K, whose sums are of 16 values, up to 24576 values: beyond, 40960 with
// two rows 2.3e-7 against 1.9e-7).
// 4096 x 11264: Q4_K at six and eight rows 97 -> 30, 117 -> 51 us, Q6_K 101 -> 35, 122 -> 61; 16384 x 9984 at eight rows 404 -> 77, 425 -> 109.
// A shape that has room for some rows has it for fewer: no part is refused after one that was launched.
static int launch_parts(const GemvMat *mats, int n_mat, int64_t n_in, int rows, int accumulate, int silu_pair, cudaStream_t st) {
    int rc = 0;
    if (rows <= 4) KRK_DISPATCH_WT(mats[0].wt, rc = stream::launch_fmt<WT>(mats, n_mat, n_in, rows, accumulate, silu_pair, true, st));
    if (rc != 0 || rows == 1) return rc;
    GemvMat part[KRK_CUDA_MAX_GROUP];
    for (int m = 0; m < n_mat; m++) part[m] = mats[m];
    const int first = (rows + 1) / 2;
    rc = launch_parts(part, n_mat, n_in, first, accumulate, silu_pair, st);
    if (rc != 1) return rc;
    for (int m = 0; m < n_mat; m++) {
        part[m].x += first * n_in;
        part[m].y += first * mats[m].n_out;
    }
    return launch_parts(part, n_mat, n_in, rows - first, accumulate, silu_pair, st);
}

int launch_gemv_stream(const GemvMat *mats, int n_mat, int64_t n_in, int rows, int accumulate, int silu_pair,
                       cudaStream_t st) {
    if (n_mat < 1 || rows < 1 || rows > KRK_CUDA_MAX_ROWS) return 0;
    const int wt = mats[0].wt;
    for (int m = 1; m < n_mat; m++)
        if (mats[m].wt != wt) return 0;
    int64_t out = 0;
    for (int m = 0; m < n_mat; m++) out += mats[m].n_out;
    // K not a multiple of 256. Short rows leave little to stream beside the preparation of the activation, and matrices that
    // fill few SMs with rows little to gain: the warp-per-row kernel (one row, 1024 weight rows, streaming against it: K = 288
    // Q8_0 4.0 against 2.6 us, Q5_0 5.7 against 2.5; K = 544 3.3 against 2.8 and 5.1 against 2.7; K = 1056 3.9 against 4.2 and
    // 4.1 against 3.8, Q5_1 at three rows 7.6 against 5.9; K = 2080 4.9 against 5.7 and 4.8 against 5.2). Below 512
    // weight rows either is a matter of a few microseconds.
    const bool odd_k = n_in % 256 != 0, few_rows = out < 8 * sm_count();
    if (odd_k && out >= 512 && (n_in < 1024 || (wt == KRK_CUDA_Q5_1 && n_in < 2048 && few_rows))) return 0;
    int rc = 0;
    KRK_DISPATCH_WT(wt, rc = stream::launch_fmt<WT>(mats, n_mat, n_in, rows, accumulate, silu_pair, false, st));
    // (few rows of Q5_1, whose units are the longest: 256 x 11264 at six rows 43.8 and 45.9 us)
    if (rc == 0 && rows > 1 && !odd_k && n_mat <= KRK_CUDA_MAX_GROUP && (wt != KRK_CUDA_Q5_1 || out >= 512) && (wt != KRK_CUDA_Q2_K || n_in <= 24576))
        return launch_parts(mats, n_mat, n_in, rows, accumulate, silu_pair, st);
    // Activation rows whose four limbs leave no room for a ring go in two launches: the weights twice through the ring are
    // quicker than the warp-per-row kernel once (8 rows of K = 11232, 2048 weight rows: Q8_0 50 against 81 us, Q5_1 70 against
    // 75), but for matrices that do not fill the SMs with rows in the formats with the longer units (512 weight rows: Q4_0
    // 57 against 52, Q5_1 70 against 53; Q8_0 48 against 55; six rows of Q4_0 37 against 42).
    const bool halve = !few_rows || wt == KRK_CUDA_Q8_0 || wt == KRK_CUDA_IQ4_NL || (wt != KRK_CUDA_Q5_1 && rows <= 6);
    if (rc == 0 && rows > 1 && odd_k && halve && n_mat <= KRK_CUDA_MAX_GROUP) {
        GemvMat part[KRK_CUDA_MAX_GROUP];
        for (int m = 0; m < n_mat; m++) part[m] = mats[m];
        const int first = (rows + 1) / 2;
        rc = launch_gemv_stream(part, n_mat, n_in, first, accumulate, silu_pair, st);
        if (rc != 1) return rc;
        for (int m = 0; m < n_mat; m++) {
            part[m].x += first * n_in;
            part[m].y += first * mats[m].n_out;
        }
        rc = launch_gemv_stream(part, n_mat, n_in, rows - first, accumulate, silu_pair, st);
    }
    return rc;
}

int launch_gemv_stream_table(const StreamTable *table, const int32_t *x_rows, int wt, int64_t n_out, int64_t n_in, int rows, int silu_pair,
                             const StreamBanks *banks, cudaStream_t st) {
    int rc = 0;
    KRK_DISPATCH_WT(wt, rc = stream::launch_table_fmt<WT>(table, x_rows, n_out, n_in, rows, silu_pair, banks, st));
    return rc;
}

int launch_gemv_stream_peers(const GemvMat &mat, int64_t n_in, int rows, const PeerScatter &ps, cudaStream_t st) {
    int rc = 0;
    KRK_DISPATCH_WT(mat.wt, rc = stream::launch_peers_fmt<WT>(mat, n_in, rows, ps, st));
    return rc;
}

int launch_flag_wait(const int *flags, int n, int epoch, cudaStream_t st) {
    int *status = device_status_word();
    if (!status) return KRK_CUDA_EDEVICE;
    flag_wait_kernel<<<1, 32, 0, st>>>(flags, n, epoch, status);
    note_launch();
    return check_launch();
}

bool stream_takes(int wt, int64_t n_in, int rows) {
    bool ok = false;
    KRK_DISPATCH_WT(wt, ok = stream::takes_fmt<WT>(n_in, rows));
    return ok;
}

} // namespace krk_cuda
