// Tile and split plan of the dense prefill GEMM (krk_gemm_tc.cu): host arithmetic alone, apart from the kernel so that it can
// be tested without a device.
#pragma once

#include <cstdint>

namespace krk_cuda {

constexpr int kTileN = 128;            // weight rows per tile (MMA M)
constexpr int kMaxTileM = 256;         // tokens per tile (MMA N)
constexpr int kYChunk = 32;            // tokens per TMA store of the read-out
constexpr int kMaxSplit = 8;           // CTAs of a cluster that share a tile

// How a dense product is cut. One tile is 128 weight rows x tile_m tokens; whole waves of tiles go to the CTAs one by
// one, and clusters of `split` CTAs share what is left of them, if that is at most one tile for every cluster (Q3_K
// 11008 x 4096, M = 300: 172 tiles of 160 tokens are a wave of 148 and 24 more; 53 -> 43 us). The model below (clocks)
// picks the pair of both that ends first: narrow tiles are bound by the decode, wide ones by MMA and power, a tile costs
// some fixed clocks for its pipeline fill and read-out, and a cluster some more to add its pieces, with its size. Over 60
// products drawn from 512..14336 rows, K of 1024..11264 and 9..2048 tokens, every pair timed, its choice takes 1.02 of the
// best pair's time on average, 1.18 at worst.
struct GemmPlan {
    int tile_m, n_tiles_n, n_tiles_m, split, n_full, grid;
};
constexpr double kFullStart = 4000.0;   // a launch on more than half of the SMs starts on some only when the one before it ends
constexpr double kStepMin = 350.0, kStepBase = 200.0, kStepToken = 2.7;
constexpr int kFixedCycles = 4000;

inline GemmPlan plan_gemm(int64_t n_out, int64_t n_in, int64_t rows, int sms, const int *clusters) {
    GemmPlan g;
    g.n_tiles_n = (int)((n_out + kTileN - 1) / kTileN);
    const int k_blocks = (int)(n_in / 256), m_max = (int)(rows >= kMaxTileM ? kMaxTileM : (rows + 15) / 16 * 16);
    double best = 0.0;
    g.tile_m = 0;
    for (int tm = m_max; tm >= 16; tm -= 16) {
        const int nm = (int)((rows + tm - 1) / tm);
        if (nm > 1 && (tm & (kYChunk - 1)) != 0) continue;   // whole chunks: a store must not reach into the next tile's tokens
        const long long tiles = (long long)g.n_tiles_n * nm;
        const double wide = kStepBase + kStepToken * tm, step = wide > kStepMin ? wide : kStepMin;
        for (int s = 1; s <= kMaxSplit && s <= k_blocks; s++) {
            if (s > 1 && clusters[s] < 1) continue;   // the device holds none of this size
            const long long ctas = s > 1 ? (long long)s * clusters[s] : sms, waves = tiles / ctas, left = tiles - waves * ctas;
            if (s > 1 && (left == 0 || left > clusters[s])) continue;
            double t = waves * (4.0 * k_blocks * step + tm * 20.0) + kFixedCycles;
            if (left > 0) t += 4.0 * ((k_blocks + s - 1) / s) * step + tm * 20.0 + (s > 1 ? 1500.0 + tm * 8.0 + s * 300.0 : 0.0);
            const long long busy = waves > 0 ? ctas : left * s;
            if (busy > sms / 2) t += kFullStart * (double)(busy - sms / 2) / (sms / 2);
            if (g.tile_m == 0 || t < best * 0.98) {   // a smaller tile or more pieces have to pay
                best = t;
                g.tile_m = tm;
                g.n_tiles_m = nm;
                g.split = s;
                g.n_full = (int)(s > 1 ? waves * ctas : tiles);
                g.grid = (int)busy;
            }
        }
    }
    return g;
}

} // namespace krk_cuda
