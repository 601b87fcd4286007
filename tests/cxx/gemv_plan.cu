// The decode GEMV's plan and shared-memory layout (setup_format and what it counts with), on the host: no device is needed.
#include <algorithm>
#include <cstdio>
#include <vector>

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
                // the ring is as deep, and as much of the SM left, as beside chunk sums that lie next to each other
                const int held = (int)smem - p.n_stages * p.stage_bytes;
                const int close = held - p.tps * (chunk_sum_bytes<WT>(p.n_in, rows, p.spread_sums) - chunk_sum_bytes<WT>(p.n_in, rows, 0));
                int fit = p.groups == 1 ? (kSmemLimit - close) / p.stage_bytes : 0;
                const bool half = fit >= 3;
                if (!half) fit = (kSmemWhole - close) / p.stage_bytes;
                const int most = p.groups == 1 ? kMaxHalfStages : kMaxStages;
                check(p.n_stages == (fit < most ? fit : most) && (!half || smem <= (size_t)kSmemLimit), "ring", WT, n_in, rows, p.n_stages, fit);
                // a tile's stages in turn: where the ring is short of two tiles, but a stage is on its way beside the two in use or
                // there is one tile only
                const bool short_ring = WT == KRK_CUDA_Q6_K && p.ragged && p.groups == 2 && tile_stages > 3 && p.n_stages < 2 * tile_stages;
                check(p.by_stage == (short_ring && p.n_stages >= 3), "stages in turn", WT, n_in, rows, p.n_stages, tile_stages);
                check(stages_in_turn<WT>(p, true) == short_ring, "stages of one tile in turn", WT, n_in, rows, p.n_stages, tile_stages);
            }
}

// How often the fullest bank of shared memory is met when the columns of a B fragment are read: `bytes` a lane, four lanes a
// column, 128 bytes at a time; equal addresses count once.
template <int WT, int NG, bool FOLD, bool FINE>
static int wavefronts(int n_in, int rows, int mg, int bytes) {
    const int per_pass = 128 / (4 * bytes);
    int worst = 0;
    for (int g0 = 0; g0 < 8; g0 += per_pass) {
        int words[32][8], count[32] = {};
        for (int g = g0; g < g0 + per_pass; g++) {
            const Column c = column_of<NG, FOLD, FINE>(mg, g);
            const int at = plane_at<WT>(n_in, rows, c.row < rows ? c.row : rows - 1, c.limb);
            for (int w = at / 4; w < at / 4 + bytes; w++) {
                int i = 0;
                while (i < count[w % 32] && words[w % 32][i] != w) i++;
                if (i == count[w % 32]) words[w % 32][count[w % 32]++] = w;
            }
        }
        for (int b = 0; b < 32; b++) worst = count[b] > worst ? count[b] : worst;
    }
    return worst;
}

template <int WT, int NG, bool FINE>
static void check_banks(int n_in, int rows) {
    constexpr bool kFold = block_size(WT) == 256 && NG > 1;
    if (WT == KRK_CUDA_Q5_0 || WT == KRK_CUDA_Q5_1) return;   // (32 bytes between planes, see plane_at)
    for (int mg = 0; mg < (kFold ? kFoldGroups<NG> : kMmaGroups<NG, FINE>); mg++) {
        const int n = wavefronts<WT, NG, kFold, FINE>(n_in, rows, mg, kWidePlanes<WT> ? 8 : 4);
        check(n <= (rows <= 4 ? 1 : 2), "bank conflicts", WT, n_in, rows, mg, n);
    }
}

template <int WT>
static void check_planes() {
    for (int rows = 1; rows <= KRK_CUDA_MAX_ROWS; rows++)
        for (int n_in = 256; n_in <= 20480; n_in += block_size(WT)) {
            const bool fine = fine_limbs<WT>(n_in);
            // planes lie apart, 16-byte aligned (32 in the formats that load 8 bytes), inside their room, which is that of planes of n_in + 32
            std::vector<int> at;
            for (int r = 0; r < rows; r++)
                for (int l = 0; l < (fine ? 4 : 3); l++) at.push_back(plane_at<WT>(n_in, rows, r, l));
            std::sort(at.begin(), at.end());
            for (size_t i = 0; i < at.size(); i++)
                check(at[i] % 16 == 0 && at[i] >= 0 && at[i] + n_in <= (i + 1 < at.size() ? at[i + 1] : plane_bytes<WT>(n_in, rows)), "planes", WT, n_in,
                      rows, (int)i, at[i]);
            check(plane_bytes<WT>(n_in, rows) <= align_up((int)at.size() * (n_in + 32), 128), "planes' room", WT, n_in, rows, plane_bytes<WT>(n_in, rows), 0);
            if constexpr (block_size(WT) == 32) {
                if (fine && rows <= 2) check_banks<WT, 1, true>(n_in, rows);
                else if (fine && rows <= 4) check_banks<WT, 2, true>(n_in, rows);
                else if (fine) check_banks<WT, 4, true>(n_in, rows);
            }
            if (!fine && rows <= 2) check_banks<WT, 1, false>(n_in, rows);
            else if (!fine && rows <= 4) check_banks<WT, 2, false>(n_in, rows);
            else if (!fine) check_banks<WT, 4, false>(n_in, rows);
        }
}

// The plans that a launch may ask for: one consumer group where two are usual, two groups that take a tile's stages in turn at one and two
// rows, four limbs.
template <int WT>
static void check_plan(int64_t n_in, int rows, bool tma, bool one_group, bool whole_sm, bool wide) {
    StreamParams p;
    size_t smem = 0;
    if (!setup_format<WT>(p, n_in, rows, 0, &smem, tma, one_group, whole_sm, wide)) return;
    const int tile_stages = (p.units + kConsumerWarps - 1) / kConsumerWarps;
    check(smem <= (size_t)kSmemWhole && p.n_stages >= 2, "room", WT, n_in, rows, (int)smem, p.n_stages);
    // the ring is as deep, and as much of the SM left, as beside chunk sums that lie next to each other
    const int held = (int)smem - p.n_stages * p.stage_bytes;
    const int close = held - p.tps * (chunk_sum_bytes<WT>(p.n_in, rows, p.spread_sums) - chunk_sum_bytes<WT>(p.n_in, rows, 0));
    int fit = p.groups == 1 ? (kSmemLimit - close) / p.stage_bytes : 0;
    const bool half = fit >= 3;
    if (!half) fit = (kSmemWhole - close) / p.stage_bytes;
    const int most = p.groups == 1 ? kMaxHalfStages : kMaxStages;
    check(p.n_stages == (fit < most ? fit : most) && (!half || smem <= (size_t)kSmemLimit), "ring", WT, n_in, rows, p.n_stages, fit);
    // what lies before the ring: the block's own words, planes and chunk sums of every stacked tile
    const bool pair = rows <= 2 && !(wide && block_size(WT) == 256);
    const size_t own = pair ? (p.groups == 1 ? sizeof(Smem<1>) : sizeof(Smem<1, 2>)) : one_group ? sizeof(Smem<2, 1>) : rows <= 4 ? sizeof(Smem<2>) : sizeof(Smem<4>);
    check(held >= align_up((int)own, 128) + p.tps * (plane_bytes<WT>(p.n_in, rows, wide) + chunk_sum_bytes<WT>(p.n_in, rows, p.spread_sums)), "before the ring", WT, n_in,
          rows, held, (int)own);
    // a tile's stages in turn: where the ring is short of two tiles, but a stage is on its way beside the two in use or
    // there is one tile only
    const bool short_ring = WT == KRK_CUDA_Q6_K && p.ragged && p.groups == 2 && tile_stages > 3 && p.n_stages < 2 * tile_stages;
    check(p.by_stage == (short_ring && p.n_stages >= 3), "stages in turn", WT, n_in, rows, p.n_stages, tile_stages);
    check(stages_in_turn<WT>(p, true) == short_ring, "stages of one tile in turn", WT, n_in, rows, p.n_stages, tile_stages);
    if (p.ragged) {   // a slot holds a row's part from the 16-byte boundary below it to the word and the boundary above it
        const int part = (p.units < kConsumerWarps ? p.units : kConsumerWarps) * Fmt<WT>::unit_bytes;
        check(p.row_stride >= align_up(14 + part, 16) && p.row_stride % 16 == 0, "slot", WT, n_in, rows, p.row_stride, part);
        check((p.row_bytes * p.ragged) % 16 == 0 && (p.ragged == 2 || (p.row_bytes * (p.ragged / 2)) % 16 != 0), "phases", WT, n_in, rows, p.row_bytes, p.ragged);
    }
    check(p.n_stages * p.stage_bytes >= p.n_stages * kTileRows * p.tps * (p.use_tma == 1 ? 1 : p.row_stride) && p.stage_bytes >= p.box_bytes && p.stage_bytes % 128 == 0,
          "stage", WT, n_in, rows, p.stage_bytes, p.box_bytes);
}

// Planes lie apart, 16-byte aligned, inside their room, which is that of planes of n_in + 32.
template <int WT>
static void check_apart(int n_in, int rows, bool wide) {
    std::vector<int> at;
    for (int r = 0; r < rows; r++)
        for (int l = 0; l < (wide || fine_limbs<WT>(n_in) ? 4 : 3); l++) at.push_back(plane_at<WT>(n_in, rows, r, l, wide));
    std::sort(at.begin(), at.end());
    for (size_t i = 0; i < at.size(); i++)
        check(at[i] % 16 == 0 && at[i] >= 0 && at[i] + n_in <= (i + 1 < at.size() ? at[i + 1] : plane_bytes<WT>(n_in, rows, wide)), "planes", WT, n_in, rows, (int)i, at[i]);
    check(plane_bytes<WT>(n_in, rows, wide) <= align_up((int)at.size() * (n_in + 32), 128), "planes' room", WT, n_in, rows, plane_bytes<WT>(n_in, rows, wide), wide);
}

template <int WT>
static void check_plans() {
    for (int rows = 1; rows <= KRK_CUDA_MAX_ROWS; rows++)
        for (int64_t n_in = 256; n_in <= 20480; n_in += block_size(WT)) {
            for (int tma = 0; tma < 2; tma++) {
                check_plan<WT>(n_in, rows, tma, false, false, false);
                if (rows <= 2) check_plan<WT>(n_in, rows, tma, false, true, false);
                if (rows <= 4 && n_in % 256 == 0) check_plan<WT>(n_in, rows, tma, false, false, true);
                if (rows <= 4 && rows > 2 && WT == KRK_CUDA_Q8_0 && n_in % 256 == 0) check_plan<WT>(n_in, rows, tma, true, false, false);
            }
            // (the kernel of four limbs passes `wide` for K that is not a multiple of 256 too)
            if (fine_limbs<WT>(n_in) || rows <= 4) check_apart<WT>(n_in, rows, true);
        }
    // Fewer rows have room where more do: parts of a call that are launched one after the other are taken or refused alike (wide: of at
    // most four rows; beyond 65,536 values no format has room).
    for (int64_t n_in = 256; n_in <= 66560; n_in += block_size(WT))
        for (int wide = 0; wide <= (n_in % 256 == 0 ? 1 : 0); wide++)
            for (int tma = 0; tma < 2; tma++) {
                bool more = false;
                for (int rows = wide ? 4 : KRK_CUDA_MAX_ROWS; rows >= 1; rows--) {
                    StreamParams p;
                    size_t smem = 0;
                    const bool takes = setup_format<WT>(p, n_in, rows, 0, &smem, tma, false, false, wide);
                    check(takes || !more, "fewer rows", WT, n_in, rows, tma, wide);
                    more = takes;
                }
            }
}

// Tiles of ragged rows (TilePlace): every row in one tile, none of more rows than a stage holds, and the same tiles from whichever
// granule a CTA starts; as many granules as the rows fill, and rows dealt to more.
static void check_phases() {
    StreamParams p = {};
    for (p.ragged = 2; p.ragged <= 8; p.ragged *= 2)
        for (int gran = kTileRows; gran <= kTileRows * kMaxStack; gran *= 2)
            for (int n_out = 1; n_out <= 2600; n_out += n_out < 160 ? 1 : 53) {
                p.gran = (short)gran;
                const int fill = (int)granules(p, n_out);
                for (int all : {fill, 148}) {
                    if (all < fill || (all > fill && all > n_out)) continue;
                    std::vector<int> at(all), count(all), seen(n_out, 0);
                    TilePlace tile(p, 0, all);
                    for (int i = 0; i < all; i++, tile.next()) {
                        tile.look(p, all, n_out);
                        at[i] = tile.phase + p.ragged * tile.first_row();
                        count[i] = tile.count();
                        check(tile.phase < p.ragged && count[i] >= 0 && count[i] <= gran, "rows of a tile", p.ragged, n_out, all, i, count[i]);
                        for (int r = 0; r < count[i]; r++) {
                            const int row = at[i] + p.ragged * r;
                            check(row < n_out, "row", p.ragged, n_out, all, i, row);
                            if (row < n_out) seen[row]++;
                        }
                    }
                    for (int r = 0; r < n_out; r++) check(seen[r] == 1, "a row's tiles", p.ragged, n_out, all, r, seen[r]);
                    for (int first = 1; first < all; first += 1 + all / 7) {
                        TilePlace from(p, first, all);
                        for (int i = first; i < all && i < first + 3; i++, from.next()) {
                            from.look(p, all, n_out);
                            check(from.phase + p.ragged * from.first_row() == at[i] && from.count() == count[i], "start", p.ragged, n_out, all, first, i);
                        }
                    }
                }
            }
}

int main() {
    check_format<KRK_CUDA_Q4_0>();
    check_planes<KRK_CUDA_Q4_0>();
    check_format<KRK_CUDA_Q5_0>();
    check_planes<KRK_CUDA_Q5_0>();
    check_format<KRK_CUDA_Q5_1>();
    check_planes<KRK_CUDA_Q5_1>();
    check_format<KRK_CUDA_Q8_0>();
    check_planes<KRK_CUDA_Q8_0>();
    check_format<KRK_CUDA_IQ4_NL>();
    check_planes<KRK_CUDA_IQ4_NL>();
    check_format<KRK_CUDA_Q2_K>();
    check_planes<KRK_CUDA_Q2_K>();
    check_format<KRK_CUDA_Q3_K>();
    check_planes<KRK_CUDA_Q3_K>();
    check_format<KRK_CUDA_Q4_K>();
    check_planes<KRK_CUDA_Q4_K>();
    check_format<KRK_CUDA_Q5_K>();
    check_planes<KRK_CUDA_Q5_K>();
    check_format<KRK_CUDA_Q6_K>();
    check_planes<KRK_CUDA_Q6_K>();
    check_phases();
    check_plans<KRK_CUDA_Q4_0>();
    check_plans<KRK_CUDA_Q5_0>();
    check_plans<KRK_CUDA_Q5_1>();
    check_plans<KRK_CUDA_Q8_0>();
    check_plans<KRK_CUDA_IQ4_NL>();
    check_plans<KRK_CUDA_Q2_K>();
    check_plans<KRK_CUDA_Q3_K>();
    check_plans<KRK_CUDA_Q4_K>();
    check_plans<KRK_CUDA_Q5_K>();
    check_plans<KRK_CUDA_Q6_K>();
    std::printf("%d of %d checks failed\n", bad, checked);
    return bad != 0;
}
