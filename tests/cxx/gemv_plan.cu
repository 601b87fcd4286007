// The decode GEMV's plan and shared-memory layout (setup_format and what it counts with), on the host: no device is needed.
#include <cstdio>

#include "krk_gemv_stream.cuh"

using namespace krk_cuda;
using namespace krk_cuda::stream;

static int bad = 0, checked = 0;
static void check(bool ok, const char *what, int wt, int64_t n_in, int rows, int a, int b) {
    checked++;
    if (ok) return;
    if (bad++ < 20) std::printf("%s: format %d, K %lld, %d rows: %d, %d\n", what, wt, (long long)n_in, rows, a, b);
}

template <int WT>
static void check_format() {
    for (int rows = 1; rows <= KRK_CUDA_MAX_ROWS; rows++)
        for (int64_t n_in = 256; n_in <= 20480; n_in += block_size(WT))
            for (int tma = 0; tma < 2; tma++) {
                StreamParams p;
                size_t smem = 0;
                if (!setup_format<WT>(p, n_in, rows, 0, &smem, tma != 0)) continue;
                const int tile_stages = (p.units + kConsumerWarps - 1) / kConsumerWarps;
                check(smem <= (size_t)kSmemWhole && p.n_stages >= 2, "room", WT, n_in, rows, (int)smem, p.n_stages);
                // a tile's stages in turn: where the ring is short of two tiles, but a stage is on its way beside the two in use or
                // there is one tile only
                const bool short_ring = WT == KRK_CUDA_Q6_K && p.ragged && p.groups == 2 && tile_stages > 3 && p.n_stages < 2 * tile_stages;
                check(p.by_stage == (short_ring && p.n_stages >= 3), "stages in turn", WT, n_in, rows, p.n_stages, tile_stages);
                check(stages_in_turn<WT>(p, true) == short_ring, "stages of one tile in turn", WT, n_in, rows, p.n_stages, tile_stages);
            }
}

int main() {
    check_format<KRK_CUDA_Q4_0>();
    check_format<KRK_CUDA_Q5_0>();
    check_format<KRK_CUDA_Q5_1>();
    check_format<KRK_CUDA_Q8_0>();
    check_format<KRK_CUDA_IQ4_NL>();
    check_format<KRK_CUDA_Q2_K>();
    check_format<KRK_CUDA_Q3_K>();
    check_format<KRK_CUDA_Q4_K>();
    check_format<KRK_CUDA_Q5_K>();
    check_format<KRK_CUDA_Q6_K>();
    std::printf("%d of %d checks failed\n", bad, checked);
    return bad != 0;
}
