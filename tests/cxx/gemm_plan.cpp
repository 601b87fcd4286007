// plan_gemm over products and devices: every tile is computed once, and no cluster size that the device does not hold
// (count 0) is chosen.
#include <cstdio>
#include <initializer_list>

#include "krk_gemm_plan.h"

using namespace krk_cuda;

static int check(int64_t n_out, int64_t n_in, int64_t rows, int sms, const int *counts) {
    const GemmPlan g = plan_gemm(n_out, n_in, rows, sms, counts);
    const long long tiles = (long long)g.n_tiles_n * g.n_tiles_m, left = tiles - g.n_full;
    bool ok = g.tile_m >= 16 && g.tile_m <= kMaxTileM && g.tile_m % 16 == 0 && (long long)g.n_tiles_n * kTileN >= n_out &&
              (long long)g.n_tiles_m * g.tile_m >= rows && (g.n_tiles_m == 1 || g.tile_m % kYChunk == 0);
    if (g.split == 1) {
        ok = ok && left == 0 && g.grid >= 1 && g.grid <= sms && g.grid <= tiles;
    } else {
        const long long clusters = g.grid / g.split;
        ok = ok && g.split <= kMaxSplit && g.split <= n_in / 256 && counts[g.split] > 0 && g.grid % g.split == 0 && clusters <= counts[g.split] &&
             left >= 1 && left <= clusters && g.n_full % g.grid == 0;
    }
    if (!ok)
        std::printf("%lld x %lld, %lld rows, %d SMs: tile_m %d, %d x %d tiles, split %d, %d whole, grid %d\n", (long long)n_out, (long long)n_in,
                    (long long)rows, sms, g.tile_m, g.n_tiles_n, g.n_tiles_m, g.split, g.n_full, g.grid);
    return ok ? 0 : 1;
}

int main() {
    const int whole[kMaxSplit + 1] = {0, 148, 74, 46, 37, 26, 24, 18, 18}, none[kMaxSplit + 1] = {0, 148}, some[kMaxSplit + 1] = {0, 148, 74, 0, 37, 0, 0, 0, 18};
    const int small[kMaxSplit + 1] = {0, 10, 5, 0, 2, 0, 1, 0, 1}, one[kMaxSplit + 1] = {0, 1};
    int bad = 0, n = 0;
    for (int64_t n_out : {1, 100, 512, 4096, 11008, 14336, 128256})
        for (int64_t n_in : {256, 512, 2048, 4096, 11008})
            for (int64_t rows : {1, 9, 16, 37, 128, 300, 512, 1000, 4097}) {
                bad += check(n_out, n_in, rows, 148, whole) + check(n_out, n_in, rows, 148, none) + check(n_out, n_in, rows, 148, some) +
                       check(n_out, n_in, rows, 10, small) + check(n_out, n_in, rows, 1, one);
                n += 5;
            }
    std::printf("%d of %d plans wrong\n", bad, n);
    return bad != 0;
}
