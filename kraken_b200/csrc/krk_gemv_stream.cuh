// Streaming decode GEMV for sm_100a: weights in any of the ten block formats (Q4_K, Q6_K, Q8_0, Q4_0, Q5_K, Q5_0,
// Q5_1, IQ4_NL, Q2_K, Q3_K), K a multiple of 256 (of 32 for the formats of 32-value blocks), 1..8 activation rows, up to 16
// matrices per launch.
//
// Design (B200-first, not the reference's one-warp-per-row walk of src/hip/kernels/gemm.hpp:76):
//
//  * One persistent CTA per SM owns a contiguous range of output rows. A producer warp streams
//    that range through a ring of shared-memory stages, one tensor copy a stage wherever a map can describe it (a copy takes 82
//    clocks to issue whatever its size; else one bulk copy per weight row), laid out without bank conflicts and signalled
//    on mbarriers; 8 consumer warps never touch global memory for weights. The ring keeps
//    50-90 KB of HBM reads in flight per SM without spending registers on it.
//
//  * A CTA takes HALF an SM (320 threads, <= 113 KB of shared memory), so the CTA of the NEXT launch
//    in the stream becomes resident (programmatic dependent launch) while this one is still
//    streaming: it sets itself up and fills its ring with weights, which no kernel in flight
//    writes, and only then waits for this grid to complete before it reads activations. The gap
//    between two launches is then a CTA start, not a CTA start plus a pipeline fill.
//
//  * At 8 TB/s a B200 SM must retire ~40 four-bit weights per clock: unpacking each one to f32
//    and issuing an FMA for it does not fit the issue budget. So the dot products run on the
//    tensor cores as EXACT integer arithmetic: the quants are fed as s8 fragments straight from
//    the packed bytes (one AND per four nibbles) to mma.sync m16n8k32 / m16n8k16 (s8 x s8 -> s32),
//    16 output rows at a time, and the activation is held as three signed 8-bit limbs of a
//    23-bit fixed-point number (x ~ s * (l0*65536 + l1*256 + l2), |X| < 2^22), one limb per MMA column
//    (four limbs where K is not a multiple of 256, see fine_limbs, and where rows go in parts, see launch_parts).
//    The products and sums are exact; the only rounding is the 23-bit quantisation of x
//    (relative to max|x|, i.e. f32-mantissa sized) and the final f32 scale arithmetic, so the
//    result sits well inside the 1e-4 * ||w_row|| * ||x|| bound. Sub-block scales are applied
//    to the s32 partial sums in integer arithmetic, block scales in f32.
//
//  * Because a dot product does not care about the order of its terms, each lane takes the
//    bytes that are cheapest to load and the activation limbs are laid out in the matching
//    order once per CTA.
//
// Every wait on an mbarrier is bounded; a wait that gives up raises the device status word
// and the CTA drains without touching memory it does not own.
#pragma once

#include <cuda.h>

#include <cfloat>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "krk_chunk.cuh"

namespace krk_cuda {

// The streaming GEMV itself; every format's kernels are instantiated in one of the krk_gemv_fmt_*.cu files, so that they
// compile side by side. krk_gemv_stream.cu holds the entry points.
namespace stream {

constexpr int kConsumerWarps = 8;
constexpr int kConsumerThreads = kConsumerWarps * 32;
// One or two groups of consumer warps per CTA. One or two activation rows: one group in half an SM, or, of many stages, two groups in a
// whole SM that take a tile's stages in turn (see stages_halve). More rows: two groups in a whole SM that share one prepared activation
// and take tiles in turn (one group per SM, all that its registers allowed before the accumulators were folded, left the schedulers
// waiting half of the time); one group and two CTAs per SM in some launches of Q8_0 (see setup_launch).
__host__ __device__ constexpr int consumer_groups(int ng) { return ng == 1 ? 1 : 2; }
__host__ __device__ constexpr int cta_threads(int groups) { return groups * kConsumerThreads + 64; }   // warp 0: producer, then the consumers, then the epilogue
// Tiles whose partial sums may wait for the epilogue warp (fewer when more activation rows make a slot larger).
__host__ __device__ constexpr int red_slots(int ng, int groups = 2) { return ng == 1 ? 4 / groups : ng == 2 ? 2 : 1; }   // of each consumer group
constexpr int kMaxRedSlots = 4;
constexpr int kMaxMaps = 24;      // of a launch: three matrices of ragged rows (with 16, a kilobyte of parameters less, every other launch takes as long)
constexpr int kMaxStack = 4;      // 16-row tiles per stage at most
constexpr int kTileRows = 16;                     // the M of the MMA
constexpr int kMaxStages = 8;                    // of a whole-SM CTA
constexpr int kMaxHalfStages = 4;                // of a half-SM one. Measured: four stages in flight per CTA stream a large Q4_K matrix at
                                                 // 0.89 of the copy bandwidth, five (all that fit) at 0.86, three at 0.86
constexpr int kSmemLimit = 113 * 1024;           // two CTAs per SM (228 KB, 1 KB reserved per CTA)
constexpr int kSmemWhole = 227 * 1024;
constexpr float kFixedOne = 4194303.0f;           // 2^22 - 1: every limb stays in s8 and X = rint(x / s) is one FMA against
                                                  // the bits of 1.5 * 2^23 (no conversion instruction)
constexpr long long kWaitCycles = 4000000000LL;   // ~2 s at boost clock, then give up
constexpr uint32_t kWaitHalfMs = (uint32_t)(kWaitCycles >> 20);

template <int WT> struct Fmt;
// tma: how a stage can arrive as ONE tiled tensor copy. 1: a unit is a whole number of 16-byte granules (Q4_K's
// 144 bytes): box {unit bytes, rows, units}, laid out [unit][row][unit bytes]. 2: eight units of a row are (Q6_K:
// 8 x 210 = 1680 bytes, as 210 64-bit elements): box {8 units, rows}, laid out [row][8 units], which is the
// layout of the per-row copies with a 1680-byte pitch. 3: a stage's part of a row is, but rows at that pitch would meet on the same
// banks (see box_pitch): box {that and up to 16 bytes more, rows} over the row bytes as 64-bit elements.
template <> struct Fmt<KRK_CUDA_Q4_K> { static constexpr int unit_values = 256, unit_bytes = 144, stride_mod = 32, tma = 1; };
template <> struct Fmt<KRK_CUDA_Q6_K> { static constexpr int unit_values = 256, unit_bytes = 210, stride_mod = 16, tma = 2; };
template <> struct Fmt<KRK_CUDA_Q8_0> { static constexpr int unit_values = 128, unit_bytes = 136, stride_mod = 16, tma = 3; };
// Q5_K: Q4_K's header and nibbles with 32 bytes of fifth bits between them (src/quant.cpp:462-489).
template <> struct Fmt<KRK_CUDA_Q5_K> { static constexpr int unit_values = 256, unit_bytes = 176, stride_mod = 32, tma = 1; };
// Q4_0: eight 18-byte blocks are 144 bytes, the size of a Q4_K unit, so the stages are laid out the same way.
template <> struct Fmt<KRK_CUDA_Q4_0> { static constexpr int unit_values = 256, unit_bytes = 144, stride_mod = 16, tma = 1; };
// Q5_0: eight 22-byte blocks are 176 bytes, the size of a Q5_K unit (rows of a fragment load 44 words apart: no
// bank is met twice). Q5_1: eight 24-byte blocks are 192 bytes, a pitch that would put rows g and g + 2 on the
// same banks, so its stages have a padded pitch.
template <> struct Fmt<KRK_CUDA_Q5_0> { static constexpr int unit_values = 256, unit_bytes = 176, stride_mod = 16, tma = 1; };
// Q2_K (84 bytes) and Q3_K (110 bytes): rows that are not 16-byte multiples go the ragged way.
template <> struct Fmt<KRK_CUDA_Q2_K> { static constexpr int unit_values = 256, unit_bytes = 84, stride_mod = 16, tma = 3; };
template <> struct Fmt<KRK_CUDA_Q3_K> { static constexpr int unit_values = 256, unit_bytes = 110, stride_mod = 16, tma = 3; };
// IQ4_NL: Q4_0's block with grid indices in place of quants.
template <> struct Fmt<KRK_CUDA_IQ4_NL> { static constexpr int unit_values = 256, unit_bytes = 144, stride_mod = 16, tma = 1; };
template <> struct Fmt<KRK_CUDA_Q5_1> { static constexpr int unit_values = 256, unit_bytes = 192, stride_mod = 16, tma = 3; };

// Parameters arrive cold in every launch, a 64-byte line at a time (some 700 clocks each): what every warp reads before its
// first load stands in the first line, the rest of what a launch of one matrix needs in the second, and the first matrices from
// the fourth on.
struct StreamParams {
    int n_entries;        // matrices, or gate/up pairs when silu_pair
    int step;             // matrices per entry (2 for gate/up pairs)
    int rows;             // activation rows
    int units;            // n_in / unit_values
    int n_in;
    int gran_q, gran_r;   // granules in all = grid * gran_q + gran_r
    const StreamTable *dev_table;   // when set, the matrices come from device memory
    const int32_t *table_rows;      // table launches: [entries][rows], see launch_gemv_stream_table
    short gran;           // rows per granule: 1, or 8 when rows are not 16-byte multiples
    short spread_sums;    // 1: planes of chunk sums lie an odd multiple of their load apart, see sum_pitch
    int tps;              // 16-row tiles stacked in one stage (> 1 when a row has so few K units that one
                          // tile would leave most consumer warps idle: warp w takes unit w % units of
                          // sub-tile w / units)
    int whole_tiles;      // 1: a stage is one contiguous copy of whole rows (unaligned row size)
    int n_stages;
    int *status;
    int row_bytes;
    int row_stride;       // bytes between rows inside a stage
    int unit_stride;      // bytes between the K units of one row group inside a stage
    int stage_bytes;
    int use_tma;          // 1: a stage arrives as one tiled tensor copy, laid out [unit][row][unit_bytes]; 2, 3: [row][units]
    int tma_unit_div;     // the copy's third coordinate is the stage's first unit / this (use_tma == 3: 0, and its first coordinate
                          // the unit's place in the row in 64-bit elements)
    int box_bytes;        // bytes one tensor copy signals (the whole box, also where the matrix clips it)
    int ragged;           // rows are not 16-byte multiples and too long for whole tiles: how many rows on (2, 4 or 8) a row lies
                          // equally far off a 16-byte boundary, see TilePlace; else 0
    int by_stage;         // 1: the two groups take a tile's stages in turn, each with sums of its own; 0: they take tiles in turn
    int accumulate;
    int entry_gran;       // table launches: granules of every entry (all have one shape)
    int groups;           // consumer groups of a CTA
    int gran_begin[KRK_CUDA_MAX_GROUP + 1];   // first row granule of each entry
    GemvMat mat[KRK_CUDA_MAX_GROUP];
    // Table launches with tensor copies: every matrix of the table lies inside one of two stacked banks (the gate
    // and the up bank of an expert set), each described by ONE tensor map (wmap[0], wmap[1]) over all of its
    // rows; a matrix is then a row offset into its bank.
    const uint8_t *bank_base[2];
    // Fused all-gather (single-matrix launches of a row shard): y goes to slot `peer_offset` of the full
    // output row in every peer's memory (this GPU's own buffer included), then the peers are told.
    float *peer_y[KRK_CUDA_MAX_PEERS];
    int *peer_flag[KRK_CUDA_MAX_PEERS];   // peer_flag[q][my_rank] <- epoch once every CTA here has stored
    int n_peers, my_rank, epoch, wait_peers;
    long long peer_row_stride, peer_offset;
    // per matrix (ragged rows: per matrix and phase, see TilePlace): the weights as a 3-d tensor, see weight_maps
    CUtensorMap wmap[kMaxMaps];
};
static_assert(sizeof(StreamParams) <= 4096, "what every launch may pass");
static_assert(offsetof(StreamParams, status) == 64 && offsetof(StreamParams, gran_begin) == 120 && offsetof(StreamParams, mat) == 192, "the lines above");


// ---- PTX wrappers ----------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// An arrival that cannot issue before `a` and `b` are there, whatever their values.
__device__ __forceinline__ void mbar_arrive_after(uint32_t bar, uint32_t a, uint32_t b) {
    asm volatile("{\n .reg .pred p;\n setp.gt.u32 p, %1, %2;\n @p mbarrier.arrive.shared::cta.b64 _, [%0];\n"
                 " @!p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(bar), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// One tiled tensor copy global -> shared (no multicast): box origin (at, row, unit).
__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap *map, int at, int row, int unit, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(at), "r"(row), "r"(unit), "r"(bar) : "memory");
}
// c = A x B with a zero accumulator input (the sub-block scale is applied to c afterwards).
__device__ __forceinline__ void mma_s8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                           uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// The same with unsigned A bytes (raw nibble pairs q_lo + 16 q_hi, or masked nibbles).
__device__ __forceinline__ void mma_u8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                           uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// k16 with the accumulator preset to the bits of 1.5 * 2^23: for |sum| < 2^22 the s32 result read as a
// float is exactly 12582912 + sum, so the conversion to float costs one subtraction instead of an I2F.
constexpr float kMagic = 12582912.0f;
__device__ __forceinline__ void mma_s8_k16_biased(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    int r[4];
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(0x4B400000));
#pragma unroll
    for (int i = 0; i < 4; i++) c[i] = __int_as_float(r[i]) - kMagic;
}
// the k16 form adding onto an accumulator that already holds the biased sum of an earlier MMA
__device__ __forceinline__ void mma_s8_k16_chain(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_u8_k16_chain(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_u8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
// x << log2(M), issued as a multiply-add: the units below are bound by the integer ALU pipe (shifts, logic ops,
// byte permutes) while the multiply-add pipe idles, so the left shifts of the operand assembly go there. The
// compiler turns a plain `x * M` back into a shift.
template <uint32_t M>
__device__ __forceinline__ uint32_t shl_mad(uint32_t x) {
    uint32_t r;
    asm("mad.lo.u32 %0, %1, %2, 0;" : "=r"(r) : "r"(x), "n"(M));
    return r;
}
__device__ __forceinline__ uint32_t shl_mad_n(uint32_t x, int k) {   // k is a constant once the caller's loops are unrolled
    switch (k) {
    case 1: return shl_mad<2u>(x);
    case 2: return shl_mad<4u>(x);
    case 3: return shl_mad<8u>(x);
    case 4: return shl_mad<16u>(x);
    default: return x << k;
    }
}
__device__ __forceinline__ int sext_byte(uint32_t w, int i) {
    int r;
    asm("bfe.s32 %0, %1, %2, 8;" : "=r"(r) : "r"(w), "r"(8 * i));
    return r;
}
__device__ __forceinline__ float half_lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xFFFFu))); }
__device__ __forceinline__ float half_hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }

// Bounded wait on an mbarrier phase. Once any wait in the CTA has given up, every later wait
// returns after its first try (which the hardware bounds), so the CTA runs to its end (on stale data, inside its own buffers)
// instead of hanging.
// (Inline: around a call the kernels kept a frame of local memory, whose first accesses miss level 1 in every launch.)
__device__ __forceinline__ uint32_t half_milliseconds() { return (uint32_t)(clock64() >> 20); }   // about
__device__ __forceinline__ void wait_phase(uint32_t bar, uint32_t parity, volatile int *gave_up, int *status) {
    if (mbar_try_wait(bar, parity)) return;
    const uint32_t t0 = half_milliseconds();
    do {
        if (*gave_up) return;
        if (half_milliseconds() - t0 > kWaitHalfMs) {
            *gave_up = 1;
            atomicExch(status, KRK_CUDA_ETIMEOUT);
            return;
        }
    } while (!mbar_try_wait(bar, parity));   // (the hardware suspends the warp for a while in each)
}

// ---- shared-memory map ---------------------------------------------------------------------------

template <int NG, int GROUPS = consumer_groups(NG)>
struct Smem {
    unsigned long long full[kMaxStages];     // weights of a stage have landed
    unsigned long long empty[kMaxStages];    // every consumer warp is done with the stage
    unsigned long long red_full[kMaxRedSlots];  // every consumer warp has written its partial sums of a tile
    unsigned long long red_empty[kMaxRedSlots]; // the epilogue warp has consumed them
    int gave_up;
    union {
        int touched[11];            // where the parameter fetches of the first instructions end (never read)
        uint32_t lead[kMaxStages];  // ragged rows: how far the rows of a stage lie into their slots (0..15 bytes)
    };
    float gate[kMaxStack][NG][32];   // epilogue warp: the gate tile(s) of a gate/up pair, until the up tile arrives
    // per consumer warp, column group and row pair (g, g+8): {row g x even activation row, g x odd, g+8 x even, g+8 x odd}
    float4 red[GROUPS * red_slots(NG, GROUPS)][kConsumerWarps][NG][8];
    float scale[NG == 1 ? 1 : kConsumerWarps][2 * NG];   // two groups: each prepared half of the activation rows, these are the scales
};

__host__ __device__ constexpr int align_up(int v, int a) { return (v + a - 1) / a * a; }

// Limbs of an activation: three, or four where K is not a multiple of 256. Those shapes belong to the warp-per-row kernel
// otherwise, which multiplies in f32; 22 bits against the largest magnitude of a warp's slices are 2 to 9 times as far off
// (error against f64 of 2.3e-7 to 1.1e-6, f32: 1.2e-7), and the MMA's fourth column was unused. (`wide` below: shapes with K a
// multiple of 256 that would belong to that kernel too, see launch_parts.)
template <int WT>
__host__ __device__ constexpr bool fine_limbs(int n_in) { return block_size(WT) == 32 && n_in % 256 != 0; }
// Where the planes lie, so that at up to four rows the eight columns of a B fragment (column_of) are read from different banks, in
// no more room than next to each other at n_in + 32. (Worked out on the device too: as parameters they cost the Q6_K head 2 %.) Most
// formats load 4 bytes a lane, 16 a column: planes lie an odd multiple of 16 bytes apart, rows of the super-block formats 96
// (modulo 128) from three rows on. Q4_K and Q5_K load 8, 32 a column, four columns at a time: planes lie 32 on (modulo 128), and from
// three rows on limbs 0 and 1 of all rows before all limbs 2, so that rows lie 64 on. (The one-row form of Q4_0 takes a limb in two
// columns. Q5_0 loses 3 % at eight rows with limbs 16 on, and it and Q5_1 keep 32: two and more columns to a bank.) All 32 on and
// rows next to each other were two- to four-fold conflicts: 32768 x 4096, Q4_K at eight rows 33.9 -> 31.2 us, Q6_K at four 32.9 -> 30.4, Q5_K
// at four 26.4 -> 25.4; Q4_0 2080 x 5600 at four rows 12.1 -> 10.4. At five to eight rows the group of all limbs 2 (32-value
// blocks: the columns of rows 6 and 7) still meets two columns to a bank.
template <int WT>
constexpr bool kWidePlanes = WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q5_K;
template <int WT>
__host__ __device__ inline int plane_pitch(int n_in, int rows, bool wide = false) {
    return n_in + (kWidePlanes<WT> || WT == KRK_CUDA_Q5_0 || WT == KRK_CUDA_Q5_1 || (WT == KRK_CUDA_Q4_0 && rows == 1 && !wide && !fine_limbs<WT>(n_in)) ? 32 : 16);
}
// Byte offset of a limb plane of activation row r of `rows`.
template <int WT>
__host__ __device__ inline int plane_at(int n_in, int rows, int r, int limb, bool wide = false) {
    const int pitch = plane_pitch<WT>(n_in, rows, wide);
    if (kWidePlanes<WT> && rows > 2) return (limb < 2 ? 2 * r + limb : limb * rows + r) * pitch;
    return r * ((wide || fine_limbs<WT>(n_in) ? 4 : 3) * pitch + (block_size(WT) == 256 && !kWidePlanes<WT> && rows > 2 ? 48 : 0)) + limb * pitch;
}
template <int WT>
__host__ __device__ inline int plane_bytes(int n_in, int rows, bool wide = false) {
    return align_up(kWidePlanes<WT> ? (wide ? 4 : 3) * rows * plane_pitch<WT>(n_in, rows, wide) : plane_at<WT>(n_in, rows, rows, 0, wide), 128);
}
// Sums of the quantised activation over the stretch of K that shares one minimum or offset: 32 values (2^5) for
// Q4_K, Q5_K, Q4_0 and Q5_1, 16 for Q2_K.
template <int WT>
constexpr int kSumShift = WT == KRK_CUDA_Q2_K ? 4 : 5;
// Elements from a plane of sums to the next: signed-byte limbs (four planes a row; eight columns are read at a time, 8 bytes each,
// or 16 for Q2_K, so the pitch is an odd multiple of that where the ring is none the smaller for it: spread, see setup_format), or
// one plane of floats a row (Q4_0, Q5_1).
template <int WT>
__host__ __device__ inline int sum_pitch(int n_in, int spread) {
    const int runs = (n_in >> 8) | spread;
    return kWidePlanes<WT> ? 8 * runs : WT == KRK_CUDA_Q2_K ? 16 * runs : n_in >> 5;
}
template <int WT>
__host__ __device__ inline int chunk_sum_bytes(int n_in, int rows, int spread) {   // four planes of bytes or one of floats
    return (WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q5_K || WT == KRK_CUDA_Q4_0 || WT == KRK_CUDA_Q5_1 || WT == KRK_CUDA_Q2_K)
               ? align_up(rows * 4 * sum_pitch<WT>(n_in, spread), 128) : 0;
}

// ---- the walk over this CTA's stages: identical in the producer and in the consumers -------------

struct StageInfo {
    int mat;        // matrix index
    int which;      // 0, or 1 for the `up` half of a gate/up pair
    int row0;       // first output row of the tile
    int n_rows;     // valid rows in the stage (1..16 * tps); ragged rows: every p.ragged-th from row0 on
    int of, k;      // ragged rows: the tile's phase, and its first row among those of the phase (TilePlace)
    int unit0;      // first K unit of this stage
    int n_units;    // units in this stage (1..16)
    int last;       // last stage of the tile
    int slot;       // ring slot of this stage
    int phase;      // parity of the slot's current use
};

// Where the list of matrices lives: the kernel parameters (host-built launches) or a table in
// device memory written by an earlier kernel (the routed-expert launches, whose matrices depend on
// expert ids that never leave the device).
// (Parameters are read as parameters, never through a pointer that may also be a table's: such a generic load of the
// parameter space misses to level 2, and four of them in a row kept a launch of 5.7 us waiting for 0.8 us.)
struct TableView {
    const StreamParams &p;
    const StreamTable *dev;
    int n_entries;
    int gran_q, gran_r;
    __device__ __forceinline__ explicit TableView(const StreamParams &params) : p(params), dev(params.dev_table) {
        if (dev) {
            n_entries = dev->n_entries;
            const int total = n_entries * p.entry_gran;
            gran_q = total / (int)gridDim.x;
            gran_r = total % (int)gridDim.x;
        } else {
            n_entries = p.n_entries;
            gran_q = p.gran_q;
            gran_r = p.gran_r;
        }
    }
    __device__ __forceinline__ int begin(int e) const { return dev ? e * p.entry_gran : p.gran_begin[e]; }
    __device__ __forceinline__ int first(int g) const { return dev ? g / p.entry_gran : 0; }   // no entry before it holds granule g
    __device__ __forceinline__ const uint8_t *w(int m) const { return dev ? dev->mat[m].w : p.mat[m].w; }
    __device__ __forceinline__ const float *x(int m) const { return dev ? dev->mat[m].x : p.mat[m].x; }
    __device__ __forceinline__ float *y(int m) const { return dev ? dev->mat[m].y : p.mat[m].y; }
    __device__ __forceinline__ int n_out(int m) const { return (int)(dev ? dev->mat[m].n_out : p.mat[m].n_out); }
};

// Ragged rows: rows `ragged` apart lie equally far off a 16-byte boundary, so a tile takes such rows, of one phase (row modulo
// `ragged`): they are a matrix of 16-byte-multiple pitch, of which a stage arrives as one tensor copy, and every word of the tile lies
// alike. An entry's granules are tiles, phase by phase: all phases have as many, or the first ones one more, and a phase's rows are
// dealt to its tiles evenly (16 * tps at most). A phase without rows, in matrices of fewer than eight, has tiles of none: their stages are
// copied like any other (by a map of the first phase's rows, see weight_maps) and their sums go nowhere.
struct TilePlace {
    int phase, n, i;   // the tile's phase, how many tiles that has (0: not looked up yet), and which of them it is
    int each, more;    // rows of a tile of the phase: the first `more` have one more than `each`
    __host__ __device__ __forceinline__ static int shift_of(const StreamParams &p) { return (p.ragged >> 2) + 1; }   // of 2, 4 or 8
    __host__ __device__ __forceinline__ static int tiles(const StreamParams &p, int granules, int phase) {
        const int shift = shift_of(p), all_have = granules >> shift, n = all_have + (phase < granules - (all_have << shift) ? 1 : 0);
        return n < 1 ? 1 : n;
    }
    __host__ __device__ __forceinline__ TilePlace(const StreamParams &p, int at, int granules) : n(0), each(0), more(0) {   // granule `at` of an entry's
        const int most = tiles(p, granules, 0), fewest = tiles(p, granules, p.ragged - 1), n_most = most == fewest ? 0 : granules - (fewest * p.ragged);
        const bool first = at < n_most * most;
        const int of_one = first ? most : fewest, rel = first ? at : at - n_most * most, of = rel / of_one;
        phase = of + (first ? 0 : n_most);
        i = rel - of * of_one;
    }
    // Before a tile is looked at. (A division for each phase, not for each tile: a producer with several short tiles waits for it. Q2_K
    // 32768 x 1280 at three rows 17.5 -> 15.7 us.)
    __host__ __device__ __forceinline__ void look(const StreamParams &p, int granules, int n_out) {
        if (n != 0) return;
        n = tiles(p, granules, phase);
        const int all = (n_out - phase + p.ragged - 1) >> shift_of(p);
        each = all / n;
        more = all - each * n;
    }
    __host__ __device__ __forceinline__ void next() {
        if (++i < n) return;
        phase++;
        i = n = 0;
    }
    __host__ __device__ __forceinline__ int first_row() const { return i * each + (i < more ? i : more); }   // of the phase's
    __host__ __device__ __forceinline__ int count() const { return each + (i < more ? 1 : 0); }
};
template <int WT>
constexpr bool kRagForm = WT == KRK_CUDA_Q6_K || WT == KRK_CUDA_Q3_K || block_size(WT) == 32;
template <bool RAGGED, class SegmentFn, class StageFn>
__device__ __forceinline__ void walk(const StreamParams &p, const TableView &tv, int tps, SegmentFn &&on_segment, StageFn &&on_stage) {
    // balanced split of the granules over the CTAs: the first gran_r CTAs take one more
    const int c = (int)blockIdx.x;
    const int g0 = c * tv.gran_q + min(c, tv.gran_r);
    const int g1 = g0 + tv.gran_q + (c < tv.gran_r ? 1 : 0);
    const int ku_max = p.whole_tiles ? p.units : kConsumerWarps;
    int slot = 0, phase = 0;
    for (int e = tv.first(g0); e < tv.n_entries; e++) {
        const int lo = max(g0, tv.begin(e)), hi = min(g1, tv.begin(e + 1));
        if (tv.begin(e) >= g1) break;
        if (lo >= hi) continue;
        const int n_out = tv.n_out(e * p.step);
        const int r0 = (lo - tv.begin(e)) * p.gran;
        const int r1 = min(n_out, (hi - tv.begin(e)) * p.gran);
        on_segment(e * p.step);
        const int stage_rows = kTileRows * tps;
        auto tile = [&](int row0, int n_rows, int of, int k) {
            for (int which = 0; which < p.step; which++) {
                for (int u0 = 0; u0 < p.units; u0 += ku_max) {
                    StageInfo s;
                    s.mat = e * p.step + which;
                    s.which = which;
                    s.row0 = row0;
                    s.n_rows = n_rows;
                    s.of = of;
                    s.k = k;
                    s.unit0 = u0;
                    s.n_units = min(ku_max, p.units - u0);
                    s.last = u0 + ku_max >= p.units;
                    s.slot = slot;
                    s.phase = phase;
                    if (++slot == p.n_stages) {
                        slot = 0;
                        phase ^= 1;
                    }
                    on_stage(s);
                }
            }
        };
        if (RAGGED && p.ragged) {
            const int granules = tv.begin(e + 1) - tv.begin(e);
            TilePlace at(p, lo - tv.begin(e), granules);
            for (int i = lo; i < hi; i++, at.next()) {
                at.look(p, granules, n_out);
                tile(at.phase + p.ragged * at.first_row(), at.count(), at.phase, at.first_row());
            }
            continue;
        }
        for (int tr = r0; tr < r1; tr += stage_rows) tile(tr, min(stage_rows, r1 - tr), 0, 0);
    }
}

// ---- activation preparation -------------------------------------------------------------------------
// Consumer warp w only ever multiplies K units w, w + WARPS, ... so it (of two groups, the warp w of one of them: each prepares every
// other activation row) prepares exactly those slices of x. Per activation row: s = max|x| / (2^22 - 1) over the warp's slices,
// X = rint(x / s) as three balanced s8 limbs (four where K is not a multiple of 256) written as byte planes (plane_at) in the
// order the B fragments are read, and (formats with a minimum or an offset) the integer sum of X over every stretch of K that shares
// one, as four planes of s8 limbs or one of floats (sum_pitch). s is NaN when a slice holds a non-finite activation, so the output
// becomes NaN as it would in f32; it multiplies the warp's partial sums at the end of each tile.

__device__ __forceinline__ int sext8(int v) { return (v << 24) >> 24; }

// Balanced signed-byte limbs of a fixed-point value: adding 128 at every byte position turns the limbs
// l in [-128, 127] into the bytes l + 128 of an unsigned number (carries do the balancing), and flipping
// bit 7 of every byte turns l + 128 back into l as a two's complement byte.
__device__ __forceinline__ uint32_t limbs3(int X) { return ((uint32_t)X + 0x00808080u) ^ 0x00808080u; }   // |X| < 2^23
__device__ __forceinline__ uint32_t limbs4(int X) { return ((uint32_t)X + 0x80808080u) ^ 0x80808080u; }

// OCTETS: a lane's eight values' limbs are stored together: 8 bytes a lane meet no bank twice, 4 do. Three and more rows (Q6_K 4096 x
// 11008 at four rows 18.4 -> 18.0 us, Q4_K 15.2 -> 14.9); one row holds the first four longer and gains nothing (a Q4_K model's pass 1089 and 1093).
template <int WT, bool OCTETS>
__device__ __forceinline__ void quantize_slice(const float (&f)[Fmt<WT>::unit_values / 32], float inv, int k0, int8_t *p0,
                                               int8_t *p1, int8_t *p2, int8_t *sums, int n_chunks, int lane) {
    constexpr int PER = Fmt<WT>::unit_values / 32;
    constexpr bool kInOrder = !(WT == KRK_CUDA_Q8_0 || WT == KRK_CUDA_Q5_0 || WT == KRK_CUDA_Q4_0 || WT == KRK_CUDA_IQ4_NL);
    uint32_t low[3];
    int total = 0;
#pragma unroll
    for (int j4 = 0; j4 < PER; j4 += 4) {
        // The bits of x * inv + 1.5 * 2^23 are those of 1.5 * 2^23 plus X (|X| <= 2^22); adding 0x00808080 less that
        // constant makes the limb bytes l + 128, whose sign bits are flipped back once they are packed.
        uint32_t z[4];   // byte 0: limb 2 (weight 1), byte 1: limb 1 (256), byte 2: limb 0 (65536)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int bits = __float_as_int(fmaf(f[j4 + j], inv, kMagic));
            total += bits;
            z[j] = (uint32_t)(bits + (0x00808080 - 0x4B400000));
        }
        const uint32_t lo01 = __byte_perm(z[0], z[1], 0x5140), lo23 = __byte_perm(z[2], z[3], 0x5140);   // l2a l2b l1a l1b
        const uint32_t w2 = __byte_perm(lo01, lo23, 0x5410) ^ 0x80808080u, w1 = __byte_perm(lo01, lo23, 0x7632) ^ 0x80808080u;
        const uint32_t w0 = __byte_perm(__byte_perm(z[0], z[1], 0x0062), __byte_perm(z[2], z[3], 0x0062), 0x5410) ^ 0x80808080u;
        const int i = k0 + j4;
        if (!kInOrder) {
            // The blocks of these formats are an odd number of half words long: the quants of every other (even) block start 2
            // bytes off a word boundary, and their lanes take them in another order, which the limbs follow in pairs: pair
            // (e, e + 1) lands at ka, (e + 2, e + 3) at kb. (Odd blocks go the same way, e and e + 2: no lane branches.)
            //   Q8_0: [0,1,30,31, 2..29].
            //   Q4_0, IQ4_NL: a block's 16 quant bytes hold value j in their low and value 16 + j in their high nibbles, so its
            //   limbs lie as [16 of the low half][16 of the high half], each as [0,1,14,15, 2..13].
            //   Q5_0: halves alike, but the quants start 6 bytes into the block: rotated by two, [14,15, 0..13], so that lane t
            //   holds values 4t-2..4t+1 of a half and their fifth bits are four neighbours of the rotated mask.
            constexpr int kRun = WT == KRK_CUDA_Q8_0 ? 32 : 16;
            const int e = i & (kRun - 1), base = i & ~(kRun - 1);
            int ka, kb;
            if (WT == KRK_CUDA_Q5_0) {
                ka = (e + 2) & 15;
                kb = (e + 4) & 15;
            } else {
                ka = e < 2 ? e : e + 2;
                kb = e + 2 >= kRun - 2 ? e + 6 - kRun : e + 4;
            }
            if ((i >> 5) & 1) ka = e, kb = e + 2;
            *reinterpret_cast<uint16_t *>(p0 + base + ka) = (uint16_t)(w0 & 0xFFFF);
            *reinterpret_cast<uint16_t *>(p0 + base + kb) = (uint16_t)(w0 >> 16);
            *reinterpret_cast<uint16_t *>(p1 + base + ka) = (uint16_t)(w1 & 0xFFFF);
            *reinterpret_cast<uint16_t *>(p1 + base + kb) = (uint16_t)(w1 >> 16);
            *reinterpret_cast<uint16_t *>(p2 + base + ka) = (uint16_t)(w2 & 0xFFFF);
            *reinterpret_cast<uint16_t *>(p2 + base + kb) = (uint16_t)(w2 >> 16);
        } else {
            static_assert(!kInOrder || PER == 8, "two quads a lane");
            if (!OCTETS) {
                *reinterpret_cast<uint32_t *>(p0 + i) = w0;
                *reinterpret_cast<uint32_t *>(p1 + i) = w1;
                *reinterpret_cast<uint32_t *>(p2 + i) = w2;
            } else if (j4 == 0) {
                low[0] = w0, low[1] = w1, low[2] = w2;
            } else {
                *reinterpret_cast<uint2 *>(p0 + k0) = make_uint2(low[0], w0);
                *reinterpret_cast<uint2 *>(p1 + k0) = make_uint2(low[1], w1);
                *reinterpret_cast<uint2 *>(p2 + k0) = make_uint2(low[2], w2);
            }
        }
    }
    total -= (int)((unsigned)PER * 0x4B400000u);   // the sum of X
    if (WT == KRK_CUDA_Q4_0 || WT == KRK_CUDA_Q5_1) {
        // the sum of X over each 32-value block, as a float: the -8 of every quant leaves -8 * d * sum per block
        // (Q5_1: the block's offset m enters as m * sum)
        total += __shfl_xor_sync(0xFFFFFFFFu, total, 1);
        total += __shfl_xor_sync(0xFFFFFFFFu, total, 2);
        if ((lane & 3) == 0) reinterpret_cast<float *>(sums)[k0 >> 5] = (float)total;   // |sum| < 2^28
    }
    if (WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q5_K || WT == KRK_CUDA_Q2_K) {
        // a 32-value chunk is held by 4 consecutive lanes (Q2_K: a 16-value group by 2); |sum| <= 32 * 2^22
        constexpr int kLanes = WT == KRK_CUDA_Q2_K ? 2 : 4;
        total += __shfl_xor_sync(0xFFFFFFFFu, total, 1);
        if (kLanes == 4) total += __shfl_xor_sync(0xFFFFFFFFu, total, 2);
        if ((lane & (kLanes - 1)) == 0) {
            const int c = k0 >> kSumShift<WT>;
            const uint32_t z = limbs4(total);   // byte 0: limb 3 (weight 1) ... byte 3: limb 0 (2^24)
            sums[c] = (int8_t)(z >> 24);
            sums[n_chunks + c] = (int8_t)(z >> 16);
            sums[2 * n_chunks + c] = (int8_t)(z >> 8);
            sums[3 * n_chunks + c] = (int8_t)z;
        }
    }
}

// The same where K is not a multiple of 256: four limbs, in value order everywhere (rows whose blocks start at any even
// address). x * inv is exact (inv is a power of two): 22 bits and, in units of 2^-8, what they leave.
// `live`: the lane's values lie inside the row (the last unit of such a row may be short).
template <int WT>
__device__ __forceinline__ void quantize_slice_fine(const float (&f)[Fmt<WT>::unit_values / 32], float inv, int k0, int8_t *p01, int8_t *p23, int ps0, int ps2,
                                                    int8_t *sums, int n_chunks, int lane, bool live) {
    constexpr int PER = Fmt<WT>::unit_values / 32;
    int total = 0, rest = 0;
#pragma unroll
    for (int j4 = 0; j4 < PER; j4 += 4) {
        uint32_t z[4];   // byte 3: limb 0 (weight 65536) ... byte 0: limb 3 (1/256)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float big = fmaf(f[j4 + j], inv, kMagic);
            const int X = __float_as_int(big) - 0x4B400000;
            const int r = __float_as_int(fmaf(fmaf(f[j4 + j], inv, kMagic - big), 256.0f, kMagic)) - 0x4B400000;   // |r| <= 128
            total += X;
            rest += r;
            z[j] = limbs4(X * 256 + r);   // |X| <= 2^22
        }
        const uint32_t lo01 = __byte_perm(z[0], z[1], 0x5140), lo23 = __byte_perm(z[2], z[3], 0x5140);   // l3 l3 l2 l2
        const uint32_t hi01 = __byte_perm(z[0], z[1], 0x7362), hi23 = __byte_perm(z[2], z[3], 0x7362);   // l1 l1 l0 l0
        if (live) {
            const int at = k0 + j4;
            *reinterpret_cast<uint32_t *>(p01 + at) = __byte_perm(hi01, hi23, 0x7632);
            *reinterpret_cast<uint32_t *>(p01 + ps0 + at) = __byte_perm(hi01, hi23, 0x5410);
            *reinterpret_cast<uint32_t *>(p23 + at) = __byte_perm(lo01, lo23, 0x7632);
            *reinterpret_cast<uint32_t *>(p23 + ps2 + at) = __byte_perm(lo01, lo23, 0x5410);
        }
    }
    if (WT == KRK_CUDA_Q5_1) {   // the sum over each 32-value block, see quantize_slice
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
            total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
            rest += __shfl_xor_sync(0xFFFFFFFFu, rest, o);
        }
        if ((lane & 3) == 0 && live) reinterpret_cast<float *>(sums)[k0 >> 5] = fmaf((float)rest, 0.00390625f, (float)total);
    }
    if (WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q5_K || WT == KRK_CUDA_Q2_K) {   // see quantize_slice; in eighths (see add_min), |sum| <= 2^30
        total = 8 * total + ((rest + 16) >> 5);
        total += __shfl_xor_sync(0xFFFFFFFFu, total, 1);
        if (WT != KRK_CUDA_Q2_K) total += __shfl_xor_sync(0xFFFFFFFFu, total, 2);
        if ((lane & (WT == KRK_CUDA_Q2_K ? 1 : 3)) == 0) {
            const int c = k0 >> kSumShift<WT>;
            const uint32_t z = limbs4(total);
#pragma unroll
            for (int l = 0; l < 4; l++) sums[l * n_chunks + c] = (int8_t)(z >> (24 - 8 * l));
        }
    }
}

// N values of x, or zeros. Predicated, not branched around (arrays that are filled in branches were spilled, 130 bytes and more a
// thread) and not read from elsewhere instead (that is as much traffic as the real thing). And in this order, all before their
// first use: left to itself the compiler put some behind the others' arithmetic, a round trip to level 2 more.
template <int N>
__device__ __forceinline__ void load_values(const float *__restrict__ x, float (&f)[N], bool there) {
#pragma unroll
    for (int j = 0; j < N; j += 4)
        asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n mov.f32 %2, 0f00000000;\n"
                     " mov.f32 %3, 0f00000000;\n @p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
                     : "=&f"(f[j]), "=&f"(f[j + 1]), "=&f"(f[j + 2]), "=&f"(f[j + 3]) : "l"(x + j), "r"((uint32_t)there) : "memory");
}
// max(mx, |f|), a NaN if there is one
template <int N>
__device__ __forceinline__ void max_abs(float &mx, const float (&f)[N]) {
#pragma unroll
    for (int j = 0; j < N; j += 2) asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(mx) : "f"(f[j]), "f"(f[j + 1]));
}

// Forms that load the next activation row before they quantise one. The others have no registers for it: spilled, they read local
// memory that misses level 1 in every launch (five to eight rows of 2048 to 6656 values 5 to 16 % longer), or their loop over the
// tiles came out slower (ragged Q6_K 16384 x 11008 at one row 50.5 us without, 54.2 with it; the other way round Q5_1 16384 x 14336
// 78.4 and 75.3, Q6_K 16384 x 4096 15.5 and 15.0, Q8_0 1024 x 2304 at three rows 6.0 and 5.5).
template <int WT, int NG, bool RAG>
constexpr bool kLoadsAhead = NG == 1 ? WT == KRK_CUDA_Q5_1 || ((WT == KRK_CUDA_Q6_K || WT == KRK_CUDA_Q3_K) && !RAG) : NG == 2 && WT == KRK_CUDA_Q8_0;
// All slices that a warp will read of activation rows r0, r0 + step, ... < rows (row(r) is where row r lies); scale(r, s) gets
// the row's scale for this warp. FINE: four limbs, and the last unit may hold fewer values than a full one.
// Every CTA prepares all of x, so this is bound by issue slots and by the latency of x: a maximum takes half an instruction a
// value, a row's loads go out together (kHeld slices stay in registers between the maximum and the quantisation, K <= 4096;
// further ones are read twice, kBatch at a time for the maximum).
template <int WT, bool FINE, bool WIDE, bool AHEAD, bool OCTETS, int WARPS, class RowFn, class ScaleFn>
__device__ __forceinline__ void prepare_x(RowFn &&row, ScaleFn &&scale, int r0, int step, int rows, const StreamParams &p, int8_t *planes,
                                          int8_t *chunk_sum, int wid, int lane) {
    constexpr int UV = Fmt<WT>::unit_values, PER = UV / 32, kHeld = 16 / PER, kBatch = 32 / PER;
    const int n_chunks = sum_pitch<WT>(p.n_in, p.spread_sums), units = p.units;
    constexpr bool wide = FINE || WIDE;
    const int ps = plane_pitch<WT>(p.n_in, p.rows, wide);
    auto at = [&](int u) { return u * UV + lane * PER; };
    auto live = [&](int u) { return !FINE || at(u) < p.n_in; };
    auto load_slice = [&](const float *xr, int u, float (&f)[PER]) { load_values(xr + at(u), f, u < units && live(u)); };
    float held[kHeld][PER], next[AHEAD ? kHeld : 1][PER];
    auto load = [&](const float *xr, auto &f) {
#pragma unroll
        for (int j = 0; j < kHeld; j++) load_slice(xr, wid + j * WARPS, f[j]);
    };
    if (r0 >= rows || wid >= units) return;
    const float *xr = row(r0);
    load(xr, held);
#pragma unroll 1
    for (int r = r0; r < rows; r += step) {
        float mx = 0.0f;
#pragma unroll 1
        for (int u0 = wid + kHeld * WARPS; u0 < units; u0 += kBatch * WARPS) {
            float f[kBatch][PER];
#pragma unroll
            for (int j = 0; j < kBatch; j++) load_slice(xr, u0 + j * WARPS, f[j]);
#pragma unroll
            for (int j = 0; j < kBatch; j++) max_abs(mx, f[j]);
        }
#pragma unroll
        for (int j = 0; j < kHeld; j++) max_abs(mx, held[j]);
        const float *const xr1 = r + step < rows ? row(r + step) : xr;
        if constexpr (AHEAD)
            if (r + step < rows) load(xr1, next);
        // (bit patterns of magnitudes order like the values, infinities and NaNs above them)
        const uint32_t mxb = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(mx));
        // |x * inv| <= 2^22 over the whole f32 range: where the quotient would overflow, a power of two takes its place; a
        // non-finite activation makes the output NaN
        mx = __uint_as_float(mxb);
        float inv, s;
        if constexpr (FINE || WIDE) {   // the power of two that takes the maximum to 2^21 .. 2^22, 2^127 at most
            const uint32_t e = min(275u - (mxb >> 23), 254u);
            inv = __uint_as_float(e << 23);
            s = __uint_as_float(e < 254u ? (254u - e) << 23 : 0x00400000u);
        } else {
            inv = __fdiv_rn(kFixedOne, mx);
            s = __fdiv_rn(mx, kFixedOne);
            if (mx < 1.25e-32f) {
                inv = 1.7014118346046923e38f;   // 2^127
                s = 5.877471754111438e-39f;     // 2^-127
            }
        }
        if (mxb > 0x7F7FFFFFu) {
            inv = 0.0f;
            s = __int_as_float(0x7FC00000);
        }
        int8_t *p0 = planes + plane_at<WT>(p.n_in, p.rows, r, 0, wide), *p2 = planes + plane_at<WT>(p.n_in, p.rows, r, 2, wide), *sums = chunk_sum + (size_t)(r * 4) * n_chunks;
        auto quantize = [&](const float (&f)[PER], int u) {
            if constexpr (FINE || WIDE)
                quantize_slice_fine<WT>(f, inv, at(u), p0, p2, ps, plane_at<WT>(p.n_in, p.rows, r, 3, wide) - plane_at<WT>(p.n_in, p.rows, r, 2, wide), sums, n_chunks, lane, live(u));
            else quantize_slice<WT, OCTETS>(f, inv, at(u), p0, p0 + ps, p2, sums, n_chunks, lane);
        };
#pragma unroll
        for (int j = 0; j < kHeld; j++) {
            const int u = wid + j * WARPS;
            if (u < units) quantize(held[j], u);
        }
        int u = wid + kHeld * WARPS;
        if (u < units) {
            float f[PER], g[PER];
            load_slice(xr, u, f);
#pragma unroll 1
            for (; u < units; u += WARPS) {
                load_slice(xr, u + WARPS, g);
                quantize(f, u);
#pragma unroll
                for (int j = 0; j < PER; j++) f[j] = g[j];
            }
        }
        scale(r, s);
        xr = xr1;
        if constexpr (AHEAD) {
#pragma unroll
            for (int j = 0; j < kHeld; j++)
#pragma unroll
                for (int i = 0; i < PER; i++) held[j][i] = next[j][i];
        } else if (r + step < rows) {
            load(xr, held);
        }
    }
}

// ---- per-format unit kernels -------------------------------------------------------------------------
// A unit is 256 values (128 for Q8_0) of 16 weight rows: lane (g, t) = (lane/4, lane%4) holds the
// A fragments of rows g and g+8, column g of the B fragment (limb g%3 of activation row g/3 of
// the column group), and accumulator columns 2t, 2t+1.

// Column groups that go through the MMAs (32-value block formats). One or two groups carry two activation rows each in
// columns 0..5, and so does the one group of the super-block formats at one or two activation rows. The
// form for five to eight rows has four groups of outputs but multiplies only three: rows 0..5 sit in columns 0..5
// of groups 0..2 and rows 6 and 7 in the spare columns 6 and 7, limb mg of the row in group mg, so that 24 columns
// carry 8 rows x 3 limbs with none to spare. With four limbs (FINE) every group is multiplied, two rows in its eight columns.
template <int NG, bool FINE>
constexpr int kMmaGroups = NG == 4 && !FINE ? 3 : NG;

// The 32-value block formats.
template <int NG>
struct Accum {
    float f[NG][4];   // [group][(row g | g+8) x (col 2t | 2t+1)], already times the block scale d
};
// Where rows are to be as exact as f32 (FINE: four limbs) a unit's blocks are added up by themselves, at up to four activation rows, and
// then added as one: a warp adds K / 256 blocks one after the other, and the error grows with the root of that (12544 values, against
// f64: Q8_0 1.45e-7 -> 1.05e-7, IQ4_NL 1.49e-7 -> 0.99e-7, Q5_1 1.76e-7 -> 1.16e-7; the warp-per-row kernel 1.42e-7, 1.42e-7, 1.70e-7. 1.004 of
// the time). Q4_0 and Q5_0 are below that kernel's without it.
template <bool FINE, int NG>
constexpr bool kUnitSums = FINE && NG <= 2;
template <bool FINE, int NG>
__device__ __forceinline__ float (&unit_sums(Accum<NG> &acc, float (&own)[NG][4]))[NG][4] {
    if constexpr (kUnitSums<FINE, NG>) {
#pragma unroll
        for (int mg = 0; mg < NG; mg++)
#pragma unroll
            for (int j = 0; j < 4; j++) own[mg][j] = 0.0f;
        return own;
    } else {
        return acc.f;
    }
}
template <bool FINE, int NG>
__device__ __forceinline__ void add_unit_sums(Accum<NG> &acc, const float (&own)[NG][4]) {
    if constexpr (kUnitSums<FINE, NG>) {
#pragma unroll
        for (int mg = 0; mg < NG; mg++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc.f[mg][j] += own[mg][j];
    }
}
// The super-block formats at one or two activation rows: the same, with a sum of its own for the minimum term.
struct AccumPair {
    float f[1][4];
    float m[4];   // dmin * sum(min_c * sum_X_c), columns = 4 limbs x 2 activation rows
};
// The super-block formats at three and more rows, whose registers do not hold a sum per limb. A lane holds two neighbouring
// columns of every column group, and the columns are dealt so that all it holds belongs to its own activation rows: a
// unit's integer sums, their limb weights and the minimum term then fold into one number per weight row and activation row
// (a quarter of the registers). Lane t looks after rows t and t + 4. Group 0 carries limbs 0 and 1 of row t in columns 2t
// and 2t + 1, group 1 (five and more rows) the same of row t + 4, the last group limb 2 of both: 24 limb columns in
// three groups, and nothing is left to add between lanes at the end of a tile. The minimum term's chunk sums (four limbs)
// lie the same way: limbs 0, 1 then 2, 3 of row t, then of row t + 4.
template <int NG>
constexpr int kFoldGroups = NG == 4 ? 3 : NG;
template <int NG>
constexpr int kFoldRows = NG == 4 ? 2 : 1;   // activation rows a lane looks after
// WIDE: four limbs, limb 3 (weight 1/256) in the column beside limb 2's, which nothing else uses up to four rows.
template <int NG, bool WIDE = false>
struct AccumFold {
    static_assert(!WIDE || NG == 2, "limb 3 has a column at up to four rows");
    float a[kFoldRows<NG>][2];   // [row t, t + 4][weight row g, g + 8]
};
template <int NG, bool WIDE = false>
using AccumSuper = std::conditional_t<NG == 1, AccumPair, AccumFold<NG, WIDE>>;
// acc += d * (limb sums of a unit), dA and dB the scales of weight rows g and g + 8
__device__ __forceinline__ void add_unit(AccumPair &acc, float dA, float dB, const int (&I)[1][4]) {
    acc.f[0][0] = fmaf(dA, (float)I[0][0], acc.f[0][0]);
    acc.f[0][1] = fmaf(dA, (float)I[0][1], acc.f[0][1]);
    acc.f[0][2] = fmaf(dB, (float)I[0][2], acc.f[0][2]);
    acc.f[0][3] = fmaf(dB, (float)I[0][3], acc.f[0][3]);
}
template <int NG, bool WIDE>
__device__ __forceinline__ void add_unit(AccumFold<NG, WIDE> &acc, float dA, float dB, const int (&I)[NG][4]) {
#pragma unroll
    for (int h = 0; h < kFoldRows<NG>; h++) {
        constexpr int L = kFoldGroups<NG> - 1;
        acc.a[h][0] = fmaf(dA, fmaf(65536.0f, (float)I[h][0], fmaf(256.0f, (float)I[h][1], WIDE ? fmaf(0.00390625f, (float)I[L][1], (float)I[L][0]) : (float)I[L][h])), acc.a[h][0]);
        acc.a[h][1] = fmaf(dB, fmaf(65536.0f, (float)I[h][2], fmaf(256.0f, (float)I[h][3], WIDE ? fmaf(0.00390625f, (float)I[L][3], (float)I[L][2]) : (float)I[L][2 + h])), acc.a[h][1]);
    }
}
// the minimum term: dmin * (minimums times group mg of the chunk sums)
__device__ __forceinline__ void add_min(AccumPair &acc, float nA, float nB, const int (&c)[4], int) {
    acc.m[0] = fmaf(nA, (float)c[0], acc.m[0]);
    acc.m[1] = fmaf(nA, (float)c[1], acc.m[1]);
    acc.m[2] = fmaf(nB, (float)c[2], acc.m[2]);
    acc.m[3] = fmaf(nB, (float)c[3], acc.m[3]);
}
template <int NG, bool WIDE>
__device__ __forceinline__ void add_min(AccumFold<NG, WIDE> &acc, float nA, float nB, const int (&c)[4], int mg) {
    const bool low = mg & 1;   // limbs 2 and 3 (weights 2^8, 1), else 0 and 1 (2^24, 2^16)
    constexpr float kUnit = WIDE ? 0.125f : 1.0f;
    const float w0 = kUnit * (low ? -256.0f : -16777216.0f), w1 = kUnit * (low ? -1.0f : -65536.0f);
    const int h = NG == 4 ? mg >> 1 : 0;
    acc.a[h][0] = fmaf(nA, fmaf(w0, (float)c[0], w1 * (float)c[1]), acc.a[h][0]);
    acc.a[h][1] = fmaf(nB, fmaf(w0, (float)c[2], w1 * (float)c[3]), acc.a[h][1]);
}
template <int NG>
__device__ __forceinline__ void accum_zero(Accum<NG> &a) {
#pragma unroll
    for (int i = 0; i < NG; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) a.f[i][j] = 0.0f;
}
__device__ __forceinline__ void accum_zero(AccumPair &a) {
#pragma unroll
    for (int j = 0; j < 4; j++) a.f[0][j] = a.m[j] = 0.0f;
}
template <int NG, bool WIDE>
__device__ __forceinline__ void accum_zero(AccumFold<NG, WIDE> &a) {
#pragma unroll
    for (int i = 0; i < kFoldRows<NG>; i++) a.a[i][0] = a.a[i][1] = 0.0f;
}
// All that a lane has summed, as one word (see the release of a stage).
template <int N>
__device__ __forceinline__ uint32_t bits_of(const float (&v)[N]) {
    uint32_t b = 0u;
#pragma unroll
    for (int i = 0; i < N; i++) b ^= __float_as_uint(v[i]);
    return b;
}
template <int NG>
__device__ __forceinline__ uint32_t bits_of(const Accum<NG> &a) {
    uint32_t b = 0u;
#pragma unroll
    for (int i = 0; i < NG; i++) b ^= bits_of(a.f[i]);
    return b;
}
__device__ __forceinline__ uint32_t bits_of(const AccumPair &a) { return bits_of(a.f[0]) ^ bits_of(a.m); }
template <int NG, bool WIDE>
__device__ __forceinline__ uint32_t bits_of(const AccumFold<NG, WIDE> &a) {
    uint32_t b = 0u;
#pragma unroll
    for (int i = 0; i < kFoldRows<NG>; i++) b ^= bits_of(a.a[i]);
    return b;
}

// What column g of column group mg carries: a limb of an activation row, and of its chunk sums.
struct Column {
    int row, limb, sum_row, sum_limb;
};
template <int NG, bool FOLD, bool FINE>
__host__ __device__ __forceinline__ Column column_of(int mg, int g) {
    // (columns 6 and 7, which carry nothing, read what columns 4 and 5 do)
    Column c{2 * mg + (g >= 6 ? 1 : g / 3), g >= 6 ? g - 5 : g % 3, 2 * mg + g / 4, g % 4};
    if (FINE && !FOLD) {
        c.row = 2 * mg + (g >> 2);
        c.limb = g & 3;
    } else if (FOLD) {   // see AccumFold
        const bool last = mg >= kFoldGroups<NG> - 1;
        c.row = (g >> 1) + (last ? (NG == 4 ? 4 * (g & 1) : 0) : 4 * mg);
        c.limb = last ? (FINE ? 2 + (g & 1) : 2) : g & 1;
        c.sum_row = (g >> 1) + 4 * (mg >> 1);
        c.sum_limb = 2 * (mg & 1) + (g & 1);
    } else if (NG == 4 && g >= 6) {   // the spare columns: limb mg of activation row 6 or 7 (group 3 multiplies nothing)
        c.row = g;
        c.limb = mg % 3;
    }
    return c;
}
// Byte planes this lane reads its B fragments from, one per column group. A lane whose column
// carries no limb (columns 6, 7, or an activation row past `rows`) reads some valid plane: its
// accumulator columns are never looked at, so what it multiplies does not matter.
template <int WT, int NG, bool FOLD, bool FINE>
__device__ __forceinline__ void lane_planes(const int8_t *planes, const int8_t *chunk_sum, int n_in, int n_sums, int rows, int g,
                                            const int8_t *(&bp)[NG], const int8_t *(&sp)[NG], bool wide) {
#pragma unroll
    for (int mg = 0; mg < NG; mg++) {
        const Column c = column_of<NG, FOLD, FINE>(mg, g);
        bp[mg] = planes + plane_at<WT>(n_in, rows, min(c.row, rows - 1), c.limb, wide);
        sp[mg] = chunk_sum + (size_t)(min(c.sum_row, rows - 1) * 4 + c.sum_limb) * n_sums;
    }
}

// FIFTH: the Q5_K super-block: 32 bytes after the header whose bit c is the fifth quant bit of chunk c's value at the
// same position; the nibbles follow them.
template <int NG, bool FIFTH, class Acc>
__device__ __forceinline__ void unit_q4_k(const uint8_t *rowA, const uint8_t *rowB, int kbase, const int8_t *const (&bp)[NG],
                                          const int8_t *const (&sp)[NG], int t, Acc &acc) {
    constexpr int kQs = FIFTH ? 48 : 16;
    const uint4 hA = *reinterpret_cast<const uint4 *>(rowA);
    const uint4 hB = *reinterpret_cast<const uint4 *>(rowB);
    uint2 fa = make_uint2(0u, 0u), fb = make_uint2(0u, 0u);
    if (FIFTH) {
        fa = *reinterpret_cast<const uint2 *>(rowA + 16 + 8 * t);
        fb = *reinterpret_cast<const uint2 *>(rowB + 16 + 8 * t);
    }
    // 6-bit scales and mins of the 8 chunks, four per word (src/quant.cpp:427-435 done bytewise)
    const uint32_t scA[2] = {hA.y & 0x3F3F3F3Fu, (hA.w & 0x0F0F0F0Fu) | ((hA.y >> 2) & 0x30303030u)};
    const uint32_t scB[2] = {hB.y & 0x3F3F3F3Fu, (hB.w & 0x0F0F0F0Fu) | ((hB.y >> 2) & 0x30303030u)};
    const uint32_t mnA[2] = {hA.z & 0x3F3F3F3Fu, ((hA.w >> 4) & 0x0F0F0F0Fu) | ((hA.z >> 2) & 0x30303030u)};
    const uint32_t mnB[2] = {hB.z & 0x3F3F3F3Fu, ((hB.w >> 4) & 0x0F0F0F0Fu) | ((hB.z >> 2) & 0x30303030u)};
    int I[NG][4];
#pragma unroll
    for (int mg = 0; mg < kFoldGroups<NG>; mg++)
#pragma unroll
        for (int j = 0; j < 4; j++) I[mg][j] = 0;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const uint2 qa = *reinterpret_cast<const uint2 *>(rowA + kQs + 32 * p + 8 * t);
        const uint2 qb = *reinterpret_cast<const uint2 *>(rowB + kQs + 32 * p + 8 * t);
#pragma unroll
        for (int nib = 0; nib < 2; nib++) {
            const int c = 2 * p + nib;
            uint32_t a0 = (qa.x >> (4 * nib)) & 0x0F0F0F0Fu, a1 = (qb.x >> (4 * nib)) & 0x0F0F0F0Fu;
            uint32_t a2 = (qa.y >> (4 * nib)) & 0x0F0F0F0Fu, a3 = (qb.y >> (4 * nib)) & 0x0F0F0F0Fu;
            if (FIFTH) {   // bit c of the mask bytes becomes bit 4 of the quants (0..31: still positive as s8)
                a0 |= (c < 4 ? shl_mad_n(fa.x, 4 - c) : fa.x >> (c - 4)) & 0x10101010u;
                a1 |= (c < 4 ? shl_mad_n(fb.x, 4 - c) : fb.x >> (c - 4)) & 0x10101010u;
                a2 |= (c < 4 ? shl_mad_n(fa.y, 4 - c) : fa.y >> (c - 4)) & 0x10101010u;
                a3 |= (c < 4 ? shl_mad_n(fb.y, 4 - c) : fb.y >> (c - 4)) & 0x10101010u;
            }
            const int sa = (scA[c >> 2] >> (8 * (c & 3))) & 0xFF, sb = (scB[c >> 2] >> (8 * (c & 3))) & 0xFF;
#pragma unroll
            for (int mg = 0; mg < kFoldGroups<NG>; mg++) {
                const uint2 b = *reinterpret_cast<const uint2 *>(bp[mg] + kbase + 32 * c + 8 * t);
                int cc[4];
                mma_s8_k32(cc, a0, a1, a2, a3, b.x, b.y);
                I[mg][0] += sa * cc[0];
                I[mg][1] += sa * cc[1];
                I[mg][2] += sb * cc[2];
                I[mg][3] += sb * cc[3];
            }
        }
    }
    const float dA = half_lo(hA.x), dB = half_lo(hB.x);
    add_unit(acc, dA, dB, I);
    // min term, also exact: one k16 MMA of the 8 mins of the super-block (k slots 0..7) against the
    // per-chunk sums of X, held as 4 limbs x 2 activation rows in the 8 columns
    const float nA = half_hi(hA.x), nB = half_hi(hB.x);
    // (no index that depends on the lane: that would put the words in local memory)
    const uint32_t a0 = t & 1 ? mnA[1] : mnA[0], a1 = t & 1 ? mnB[1] : mnB[0];   // (k slots 8..15, lanes 2 and 3, meet zeros)
#pragma unroll
    for (int mg = 0; mg < NG; mg++) {
        const uint32_t b0 = t < 2 ? *reinterpret_cast<const uint32_t *>(sp[mg] + (kbase >> 5) + 4 * t) : 0u;
        int cc[4];
        mma_s8_k16(cc, a0, a1, b0);
        add_min(acc, nA, nB, cc, mg);
    }
}

// Q4_K with ONE activation row: both nibbles of a byte go through the tensor core unshifted.
// The 32 bytes of a group hold chunk 2p in their low nibbles and chunk 2p+1 in their high ones.
// Column 2j of the B fragment carries limb j of x over chunk 2p, column 2j+1 limb j over chunk
// 2p+1. Two MMAs per group: L = (bytes & 0x0F) x B and R = (raw bytes) x B. Then, per limb,
//   low chunk  = L[even column],     high chunk = (R[odd column] - L[odd column]) / 16,
// because raw = q_lo + 16 q_hi. One AND per four bytes replaces the AND, shift, AND of the
// two-MMA-per-chunk form; lane t keeps limb t of rows g and g+8 (t = 3 multiplies nothing).
struct AccumSingle {
    float f[2];   // rows g, g+8: limb t of d * sum over sub-blocks, times 16
    float m[4];   // the min term as in AccumPair
};
// The B fragments of a unit (x limbs, chunk sums) are the same for every row tile: a warp that always works
// on the same K units keeps them in registers (BFrag) instead of reading them from shared memory per tile.
struct BFrag {
    uint2 b[4];     // per group of two chunks
    uint32_t m;     // chunk sums for the min term
};
__device__ __forceinline__ BFrag load_bfrag(const int8_t *bq, const int8_t *sq, int t) {
    BFrag f;
#pragma unroll
    for (int p = 0; p < 4; p++) f.b[p] = *reinterpret_cast<const uint2 *>(bq + 64 * p + 8 * t);
    f.m = t < 2 ? *reinterpret_cast<const uint32_t *>(sq + 4 * t) : 0u;
    return f;
}
__device__ __forceinline__ void unit_q4_k_single(const uint8_t *rowA, const uint8_t *rowB, const BFrag &bf, int t,
                                                 AccumSingle &acc) {
    const uint4 hA = *reinterpret_cast<const uint4 *>(rowA);
    const uint4 hB = *reinterpret_cast<const uint4 *>(rowB);
    const uint32_t scA[2] = {hA.y & 0x3F3F3F3Fu, (hA.w & 0x0F0F0F0Fu) | ((hA.y >> 2) & 0x30303030u)};
    const uint32_t scB[2] = {hB.y & 0x3F3F3F3Fu, (hB.w & 0x0F0F0F0Fu) | ((hB.y >> 2) & 0x30303030u)};
    const uint32_t mnA[2] = {hA.z & 0x3F3F3F3Fu, ((hA.w >> 4) & 0x0F0F0F0Fu) | ((hA.z >> 2) & 0x30303030u)};
    const uint32_t mnB[2] = {hB.z & 0x3F3F3F3Fu, ((hB.w >> 4) & 0x0F0F0F0Fu) | ((hB.z >> 2) & 0x30303030u)};
    int loA = 0, hrA = 0, hlA = 0, loB = 0, hrB = 0, hlB = 0;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const uint2 qa = *reinterpret_cast<const uint2 *>(rowA + 16 + 32 * p + 8 * t);
        const uint2 qb = *reinterpret_cast<const uint2 *>(rowB + 16 + 32 * p + 8 * t);
        const uint2 b = bf.b[p];
        int cl[4], cr[4];
        mma_u8_k32(cl, qa.x & 0x0F0F0F0Fu, qb.x & 0x0F0F0F0Fu, qa.y & 0x0F0F0F0Fu, qb.y & 0x0F0F0F0Fu, b.x, b.y);
        mma_u8_k32(cr, qa.x, qb.x, qa.y, qb.y, b.x, b.y);
        const int c0 = 2 * p, c1 = 2 * p + 1;
        const int sA0 = (scA[c0 >> 2] >> (8 * (c0 & 3))) & 0xFF, sA1 = (scA[c1 >> 2] >> (8 * (c1 & 3))) & 0xFF;
        const int sB0 = (scB[c0 >> 2] >> (8 * (c0 & 3))) & 0xFF, sB1 = (scB[c1 >> 2] >> (8 * (c1 & 3))) & 0xFF;
        loA += sA0 * cl[0];
        hrA += sA1 * cr[1];
        hlA += sA1 * cl[1];
        loB += sB0 * cl[2];
        hrB += sB1 * cr[3];
        hlB += sB1 * cl[3];
    }
    // |16 lo + hr - hl| < 2^29: 4 groups x 63 x 32 x (16 * 15 + 255 + 15) x 128
    const float dA = half_lo(hA.x), dB = half_lo(hB.x);
    acc.f[0] = fmaf(dA, (float)(16 * loA + hrA - hlA), acc.f[0]);
    acc.f[1] = fmaf(dB, (float)(16 * loB + hrB - hlB), acc.f[1]);
    const float nA = half_hi(hA.x), nB = half_hi(hB.x);
    // (no index that depends on the lane: that would put the words in local memory)
    const uint32_t a0 = t & 1 ? mnA[1] : mnA[0], a1 = t & 1 ? mnB[1] : mnB[0];   // (k slots 8..15, lanes 2 and 3, meet zeros)
    float cm[4];
    mma_s8_k16_biased(cm, a0, a1, bf.m);   // |sum| <= 8 x 63 x 128 < 2^22
    acc.m[0] = fmaf(nA, cm[0], acc.m[0]);
    acc.m[1] = fmaf(nA, cm[1], acc.m[1]);
    acc.m[2] = fmaf(nB, cm[2], acc.m[2]);
    acc.m[3] = fmaf(nB, cm[3], acc.m[3]);
}

// 32-bit words at constant even offsets of a block or row in shared memory that starts on a word boundary (BY2 0), 2 bytes off one
// (1: blocks of 210 and 110 bytes, every other one of a row; ragged rows, those of every other phase), or either (2: both starts that a
// word may have and both shifts are found once for all words). A word off the boundary is glued from two.
template <int BY2>
struct Words {
    const uint8_t *p0, *p2;   // 2: for offsets that are multiples of 4, and for the others
    uint32_t s0, s2;
    __device__ __forceinline__ explicit Words(const uint8_t *at) : p0(at), p2(at), s0(0), s2(0) {
        if (BY2 == 2) {
            const uint32_t by = smem_u32(at) & 2u;
            p0 = at - by;
            p2 = at + by - 2;
            s0 = 8u * by;
            s2 = 16u - s0;
        }
    }
    __device__ __forceinline__ uint32_t operator()(int off) const {
        if (BY2 == 2) {
            const uint32_t *w = reinterpret_cast<const uint32_t *>((off & 2 ? p2 : p0) + off);
            return __funnelshift_r(w[0], w[1], off & 2 ? s2 : s0);
        }
        if (((off >> 1) & 1) == BY2) return *reinterpret_cast<const uint32_t *>(p0 + off);
        return __byte_perm(*reinterpret_cast<const uint32_t *>(p0 + off - 2), *reinterpret_cast<const uint32_t *>(p0 + off + 2), 0x5432);
    }
};

// The 32-value blocks of rows that start at any even address (K not a multiple of 256): the limbs lie in value order, words are
// read as they lie or glued (see Words; BY2: the tile's rows start 2 bytes off a word boundary), and only the first `nb` blocks of a unit exist (the last unit of a row may be
// short; what its slot holds past the row is never looked at).
__device__ __forceinline__ float half_at(const uint8_t *p) { return __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(p))); }

// Eight Q4_0 blocks (src/quant.cpp:331-339), one activation row. A block is a 2-byte scale d and 16 bytes whose
// low nibbles are quants 0..15 and whose high nibbles are quants 16..31; the value is d * (q - 8). Per block two
// k16 MMAs over the same 16 bytes, L = (bytes & 0x0F) and R = raw bytes, against columns [limb j over the low
// half, limb j over the high half]: low half = L[even column], high half = (R[odd] - L[odd]) / 16. Lane t keeps
// limb t of rows g and g+8 (times 16); lane t = 3, whose columns carry no limb, keeps d * (sum of X over the
// block) instead, which enters the result with weight -8. Blocks at an even index have their quants 2 bytes off
// a word boundary: lane t = 0 glues the half words at the two ends (the limbs are laid out to match).
__device__ __forceinline__ void unit_q4_0(const uint8_t *rowA, const uint8_t *rowB, const int8_t *bq, const float *fs, int t,
                                          AccumSingle &acc) {
#pragma unroll
    for (int b = 0; b < 8; b++) {
        uint32_t qa, qb;
        float dA, dB;
        if ((b & 1) == 0) {
            const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 18 * b);
            const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 18 * b);
            const uint32_t a_first = wa[0], b_first = wb[0];
            qa = t == 0 ? __byte_perm(a_first, wa[4], 0x5432) : wa[t];
            qb = t == 0 ? __byte_perm(b_first, wb[4], 0x5432) : wb[t];
            dA = half_lo(a_first);
            dB = half_lo(b_first);
        } else {
            qa = reinterpret_cast<const uint32_t *>(rowA + 18 * b + 2)[t];
            qb = reinterpret_cast<const uint32_t *>(rowB + 18 * b + 2)[t];
            dA = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowA + 18 * b)));
            dB = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowB + 18 * b)));
        }
        const uint32_t bw = *reinterpret_cast<const uint32_t *>(bq + 32 * b + 4 * t);
        int cl[4], cr[4];
        mma_u8_k16(cl, qa & 0x0F0F0F0Fu, qb & 0x0F0F0F0Fu, bw);
        mma_u8_k16(cr, qa, qb, bw);
        // |16 lo + hr - hl| < 2^21: 16 x (16 * 15 + 255 + 15) x 128, so the bits of 1.5 * 2^23 turn it into a float
        const int vA = 16 * cl[0] + cr[1] - cl[1], vB = 16 * cl[2] + cr[3] - cl[3];
        const float sum = fs[b];
        const float fa = t == 3 ? sum : __int_as_float(vA + 0x4B400000) - kMagic;
        const float fb = t == 3 ? sum : __int_as_float(vB + 0x4B400000) - kMagic;
        acc.f[0] = fmaf(dA, fa, acc.f[0]);
        acc.f[1] = fmaf(dB, fb, acc.f[1]);
    }
}

// The same eight blocks for 2..8 activation rows: the quants are centred first ((q + 0x78) ^ 0x80 is q - 8 as a
// signed byte, no carry since q <= 15), low and high nibbles go to one k16 MMA each per column group, and the
// columns carry the limbs of two activation rows as in the other general forms.
template <int NG, bool RAG, int BY2>
__device__ __forceinline__ void unit_q4_0_rows(const uint8_t *rowA, const uint8_t *rowB, int kbase, const int8_t *const (&bp)[NG],
                                               int t, Accum<NG> &acc, int nb) {
    const Words<BY2> wA(rowA + 4 * t), wB(rowB + 4 * t);
#pragma unroll
    for (int b = 0; b < 8; b++) {
        if (RAG && b >= nb) break;
        uint32_t qa, qb;
        float dA, dB;
        if (RAG) {
            qa = wA(18 * b + 2);
            qb = wB(18 * b + 2);
            dA = half_at(rowA + 18 * b);
            dB = half_at(rowB + 18 * b);
        } else if ((b & 1) == 0) {
            const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 18 * b);
            const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 18 * b);
            const uint32_t a_first = wa[0], b_first = wb[0];
            qa = t == 0 ? __byte_perm(a_first, wa[4], 0x5432) : wa[t];
            qb = t == 0 ? __byte_perm(b_first, wb[4], 0x5432) : wb[t];
            dA = half_lo(a_first);
            dB = half_lo(b_first);
        } else {
            qa = reinterpret_cast<const uint32_t *>(rowA + 18 * b + 2)[t];
            qb = reinterpret_cast<const uint32_t *>(rowB + 18 * b + 2)[t];
            dA = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowA + 18 * b)));
            dB = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowB + 18 * b)));
        }
        // The A operand is 16 * (q - 8) as a signed byte: the nibble in the high half of the byte with its top bit
        // flipped (one instruction for the high nibbles, a shift more for the low ones); the 16 leaves with d.
        // Both MMAs of a block add onto one accumulator preset to the bits of 1.5 * 2^23, whose bits read as a
        // float are that plus the sum (|sum| <= 32 * 128 * 128 = 2^19), so the int-to-float step is a subtraction.
        const uint32_t la = ((qa << 4) & 0xF0F0F0F0u) ^ 0x80808080u, lb = ((qb << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
        const uint32_t ha = (qa & 0xF0F0F0F0u) ^ 0x80808080u, hb = (qb & 0xF0F0F0F0u) ^ 0x80808080u;
        dA *= 0.0625f;
        dB *= 0.0625f;
#pragma unroll
        for (int mg = 0; mg < kMmaGroups<NG, RAG>; mg++) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 4 * t);
            const uint32_t b1 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 16 + 4 * t);
            int c[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};
            mma_s8_k16_chain(c, la, lb, b0);
            mma_s8_k16_chain(c, ha, hb, b1);
            acc.f[mg][0] = fmaf(dA, __int_as_float(c[0]) - kMagic, acc.f[mg][0]);
            acc.f[mg][1] = fmaf(dA, __int_as_float(c[1]) - kMagic, acc.f[mg][1]);
            acc.f[mg][2] = fmaf(dB, __int_as_float(c[2]) - kMagic, acc.f[mg][2]);
            acc.f[mg][3] = fmaf(dB, __int_as_float(c[3]) - kMagic, acc.f[mg][3]);
        }
    }
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// Eight IQ4_NL blocks (src/quant.cpp:88-91, 566-575): Q4_0's layout, but a nibble is an index into a grid of 16
// signed bytes. The grid lies in four words; a byte permute looks four indices up in two of them at a time (the
// low three bits of each nibble of the selector), once in the lower and once in the upper half of the grid, and
// the index's top bit picks between the two through a mask made by another permute in its sign-replicating mode.
// Nibbles 0..3 of a quant word are [low 0, high 0, low 1, high 1], so two last permutes regroup the results into
// the four low-nibble and the four high-nibble values. 13 integer instructions per eight values. The limbs lie
// as for Q4_0.
template <int NG, bool RAG, int BY2>
__device__ __forceinline__ void unit_iq4_nl(const uint8_t *rowA, const uint8_t *rowB, int kbase, const int8_t *const (&bp)[NG],
                                            int t, Accum<NG> &acc, int nb) {
    float own[NG][4];
    float (&sum)[NG][4] = unit_sums<RAG>(acc, own);
    constexpr uint32_t kG0 = 0xBFAD9881u, kG1 = 0xF6EADDCFu, kG2 = 0x26190D01u, kG3 = 0x71594535u;
    auto grid = [&](uint32_t q, uint32_t &lo4, uint32_t &hi4) {
        const uint32_t s = q & 0x77777777u, s2 = s >> 16, y = q << 4;
        const uint32_t m01 = prmt(y, q, 0xD9C8u), m23 = prmt(y, q, 0xFBEAu);   // 0xFF where the index is 8..15
        const uint32_t r01 = (prmt(kG0, kG1, s) & ~m01) | (prmt(kG2, kG3, s) & m01);
        const uint32_t r23 = (prmt(kG0, kG1, s2) & ~m23) | (prmt(kG2, kG3, s2) & m23);
        lo4 = prmt(r01, r23, 0x6420u);
        hi4 = prmt(r01, r23, 0x7531u);
    };
    const Words<BY2> wA(rowA + 4 * t), wB(rowB + 4 * t);
#pragma unroll
    for (int b = 0; b < 8; b++) {
        if (RAG && b >= nb) break;
        uint32_t qa, qb;
        float dA, dB;
        if (RAG) {
            qa = wA(18 * b + 2);
            qb = wB(18 * b + 2);
            dA = half_at(rowA + 18 * b);
            dB = half_at(rowB + 18 * b);
        } else if ((b & 1) == 0) {
            const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 18 * b);
            const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 18 * b);
            const uint32_t a_first = wa[0], b_first = wb[0];
            qa = t == 0 ? __byte_perm(a_first, wa[4], 0x5432) : wa[t];
            qb = t == 0 ? __byte_perm(b_first, wb[4], 0x5432) : wb[t];
            dA = half_lo(a_first);
            dB = half_lo(b_first);
        } else {
            qa = reinterpret_cast<const uint32_t *>(rowA + 18 * b + 2)[t];
            qb = reinterpret_cast<const uint32_t *>(rowB + 18 * b + 2)[t];
            dA = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowA + 18 * b)));
            dB = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowB + 18 * b)));
        }
        uint32_t la, ha, lb, hb;
        grid(qa, la, ha);
        grid(qb, lb, hb);
#pragma unroll
        for (int mg = 0; mg < kMmaGroups<NG, RAG>; mg++) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 4 * t);
            const uint32_t b1 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 16 + 4 * t);
            int c[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};   // |sum| <= 32 * 127 * 128 < 2^19
            mma_s8_k16_chain(c, la, lb, b0);
            mma_s8_k16_chain(c, ha, hb, b1);
            sum[mg][0] = fmaf(dA, __int_as_float(c[0]) - kMagic, sum[mg][0]);
            sum[mg][1] = fmaf(dA, __int_as_float(c[1]) - kMagic, sum[mg][1]);
            sum[mg][2] = fmaf(dB, __int_as_float(c[2]) - kMagic, sum[mg][2]);
            sum[mg][3] = fmaf(dB, __int_as_float(c[3]) - kMagic, sum[mg][3]);
        }
    }
    add_unit_sums<RAG>(acc, own);
}

// Bits 0..3 of n to bit 7 of bytes 0..3: bit i times 2^(7j + 7) lands at 8k + 7 only for i = j = k, and no two
// products share a position, so nothing carries.
__device__ __forceinline__ uint32_t spread_top(uint32_t n) { return (n * 0x10204080u) & 0x80808080u; }

// Eight Q5_0 blocks (src/quant.cpp:352-364): a 2-byte scale d, a 32-bit mask of fifth bits, 16 bytes whose low
// nibbles are quants 0..15 and whose high nibbles are quants 16..31; the value is d * (q - 16). The A operand is
// 8 * (q - 16) as a signed byte: the nibble at bits 3-6 and the inverted fifth bit at bit 7 (q - 16 is q with
// bit 4 flipped, read as a 5-bit two's complement); the 8 leaves with d. Two k16 MMAs per block and column
// group, chained on one accumulator preset to the bits of 1.5 * 2^23 (|sum| <= 32 * 128 * 128 = 2^19). Blocks at
// an even index have mask and quants 2 bytes off a word boundary: the mask is glued from two words, lane t takes
// quant bytes 4t-2..4t+1 (lane 0: 14, 15, 0, 1) and the mask is rotated to match.
template <int NG, bool RAG, int BY2>
__device__ __forceinline__ void unit_q5_0(const uint8_t *rowA, const uint8_t *rowB, int kbase, const int8_t *const (&bp)[NG],
                                          int t, Accum<NG> &acc, int nb) {
    const Words<BY2> wA(rowA), wB(rowB);
#pragma unroll
    for (int b = 0; b < 8; b++) {
        if (RAG && b >= nb) break;
        uint32_t qa, qb, ma, mb;
        float dA, dB;
        if (RAG) {
            qa = wA(22 * b + 6 + 4 * t);
            qb = wB(22 * b + 6 + 4 * t);
            ma = ~wA(22 * b + 2);
            mb = ~wB(22 * b + 2);
            dA = half_at(rowA + 22 * b);
            dB = half_at(rowB + 22 * b);
        } else if ((b & 1) == 0) {
            const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 22 * b);
            const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 22 * b);
            const uint32_t a0 = wa[0], a1 = wa[1], b0 = wb[0], b1 = wb[1];
            qa = t == 0 ? __byte_perm(a1, wa[5], 0x3254) : wa[t + 1];
            qb = t == 0 ? __byte_perm(b1, wb[5], 0x3254) : wb[t + 1];
            const uint32_t ha = ~__byte_perm(a0, a1, 0x5432), hb = ~__byte_perm(b0, b1, 0x5432);
            ma = ((ha << 2) & 0xFFFCFFFCu) | ((ha >> 14) & 0x00030003u);   // both 16-bit halves rotated left by 2
            mb = ((hb << 2) & 0xFFFCFFFCu) | ((hb >> 14) & 0x00030003u);
            dA = half_lo(a0);
            dB = half_lo(b0);
        } else {
            qa = reinterpret_cast<const uint32_t *>(rowA + 22 * b + 6)[t];
            qb = reinterpret_cast<const uint32_t *>(rowB + 22 * b + 6)[t];
            ma = ~*reinterpret_cast<const uint32_t *>(rowA + 22 * b + 2);
            mb = ~*reinterpret_cast<const uint32_t *>(rowB + 22 * b + 2);
            dA = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowA + 22 * b)));
            dB = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowB + 22 * b)));
        }
        const uint32_t la = ((qa << 3) & 0x78787878u) | spread_top((ma >> (4 * t)) & 0xFu);
        const uint32_t lb = ((qb << 3) & 0x78787878u) | spread_top((mb >> (4 * t)) & 0xFu);
        const uint32_t ha = ((qa >> 1) & 0x78787878u) | spread_top((ma >> (16 + 4 * t)) & 0xFu);
        const uint32_t hb = ((qb >> 1) & 0x78787878u) | spread_top((mb >> (16 + 4 * t)) & 0xFu);
        dA *= 0.125f;
        dB *= 0.125f;
#pragma unroll
        for (int mg = 0; mg < kMmaGroups<NG, RAG>; mg++) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 4 * t);
            const uint32_t b1 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 16 + 4 * t);
            int c[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};
            mma_s8_k16_chain(c, la, lb, b0);
            mma_s8_k16_chain(c, ha, hb, b1);
            acc.f[mg][0] = fmaf(dA, __int_as_float(c[0]) - kMagic, acc.f[mg][0]);
            acc.f[mg][1] = fmaf(dA, __int_as_float(c[1]) - kMagic, acc.f[mg][1]);
            acc.f[mg][2] = fmaf(dB, __int_as_float(c[2]) - kMagic, acc.f[mg][2]);
            acc.f[mg][3] = fmaf(dB, __int_as_float(c[3]) - kMagic, acc.f[mg][3]);
        }
    }
}

// Eight Q5_1 blocks (src/quant.cpp:366-379): scale d, offset m, the mask, the nibbles, all on word boundaries;
// the value is d * q + m with q = 0..31. The A operand is 8 * q as an unsigned byte; the offset enters as
// m * (sum of X over the block), which the activation pass leaves per block as a float: the lanes whose columns
// carry the limb of weight 1 (column 2 of the even, column 5 of the odd activation row of a group; of four limbs columns
// 2 and 6) add it.
template <int NG, bool RAG>
__device__ __forceinline__ void unit_q5_1(const uint8_t *rowA, const uint8_t *rowB, int kbase, const int8_t *const (&bp)[NG],
                                          const float *const (&fe)[NG], const float *const (&fo)[NG], int t, Accum<NG> &acc, int nb) {
    float own[NG][4];
    float (&sum)[NG][4] = unit_sums<RAG>(acc, own);
#pragma unroll
    for (int b = 0; b < 8; b++) {
        if (RAG && b >= nb) break;   // (rows start on 8-byte boundaries: words stay aligned)
        const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 24 * b);
        const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 24 * b);
        const uint32_t a0 = wa[0], b0w = wb[0], ma = wa[1], mb = wb[1], qa = wa[2 + t], qb = wb[2 + t];
        const float dA = 0.125f * half_lo(a0), dB = 0.125f * half_lo(b0w), oA = half_hi(a0), oB = half_hi(b0w);
        const uint32_t la = ((qa << 3) & 0x78787878u) | spread_top((ma >> (4 * t)) & 0xFu);
        const uint32_t lb = ((qb << 3) & 0x78787878u) | spread_top((mb >> (4 * t)) & 0xFu);
        const uint32_t ha = ((qa >> 1) & 0x78787878u) | spread_top((ma >> (16 + 4 * t)) & 0xFu);
        const uint32_t hb = ((qb >> 1) & 0x78787878u) | spread_top((mb >> (16 + 4 * t)) & 0xFu);
#pragma unroll
        for (int mg = 0; mg < kMmaGroups<NG, RAG>; mg++) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 4 * t);
            const uint32_t b1 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 16 + 4 * t);
            int c[4] = {0x4B400000, 0x4B400000, 0x4B400000, 0x4B400000};   // |sum| <= 32 * 248 * 128 < 2^20
            mma_u8_k16_chain(c, la, lb, b0);
            mma_u8_k16_chain(c, ha, hb, b1);
            // (five to eight rows: the weight-1 limbs of rows 6 and 7 are columns 6 and 7 of group 2, in lane t = 3)
            const bool spare = NG == 4 && mg == 2 && t == 3;
            const int at = (kbase >> 5) + b;
            const float se = t == 1 ? fe[mg][at] : RAG ? (t == 3 ? fo[mg][at] : 0.0f) : spare ? fe[NG - 1][at] : 0.0f;
            const float so = RAG ? 0.0f : t == 2 ? fo[mg][at] : spare ? fo[NG - 1][at] : 0.0f;
            sum[mg][0] = fmaf(dA, __int_as_float(c[0]) - kMagic, fmaf(oA, se, sum[mg][0]));
            sum[mg][1] = fmaf(dA, __int_as_float(c[1]) - kMagic, fmaf(oA, so, sum[mg][1]));
            sum[mg][2] = fmaf(dB, __int_as_float(c[2]) - kMagic, fmaf(oB, se, sum[mg][2]));
            sum[mg][3] = fmaf(dB, __int_as_float(c[3]) - kMagic, fmaf(oB, so, sum[mg][3]));
        }
    }
    add_unit_sums<RAG>(acc, own);
}

// Four Q8_0 blocks. A block is a 2-byte scale then 32 quants, so blocks at an even index have
// their quants 2 bytes off a word boundary: their lanes read the aligned words and lane t = 0
// glues the two half words at the ends into one (the activation limbs are permuted to match).
template <int NG, bool RAG, int BY2>
__device__ __forceinline__ void unit_q8_0(const uint8_t *rowA, const uint8_t *rowB, int kbase, const int8_t *const (&bp)[NG],
                                          int t, Accum<NG> &acc, int nb) {
    float own[NG][4];
    float (&sum)[NG][4] = unit_sums<RAG>(acc, own);
    const Words<BY2> wA(rowA + 4 * t), wB(rowB + 4 * t);
#pragma unroll
    for (int b = 0; b < 4; b++) {
        if (RAG && b >= nb) break;
        uint32_t a0, a1, a2, a3;
        float dA, dB;
        if (RAG) {
            a0 = wA(34 * b + 2);
            a1 = wB(34 * b + 2);
            a2 = wA(34 * b + 18);
            a3 = wB(34 * b + 18);
            dA = half_at(rowA + 34 * b);
            dB = half_at(rowB + 34 * b);
        } else if ((b & 1) == 0) {
            const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 34 * b);
            const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 34 * b);
            const uint32_t a_first = wa[0], b_first = wb[0];
            a0 = t == 0 ? __byte_perm(a_first, wa[8], 0x5432) : wa[t];
            a1 = t == 0 ? __byte_perm(b_first, wb[8], 0x5432) : wb[t];
            a2 = wa[t + 4];
            a3 = wb[t + 4];
            dA = half_lo(a_first);
            dB = half_lo(b_first);
        } else {
            const uint32_t *wa = reinterpret_cast<const uint32_t *>(rowA + 34 * b + 2);
            const uint32_t *wb = reinterpret_cast<const uint32_t *>(rowB + 34 * b + 2);
            a0 = wa[t];
            a1 = wb[t];
            a2 = wa[t + 4];
            a3 = wb[t + 4];
            dA = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowA + 34 * b)));
            dB = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(rowB + 34 * b)));
        }
#pragma unroll
        for (int mg = 0; mg < kMmaGroups<NG, RAG>; mg++) {
            const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 4 * t);
            const uint32_t b1 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 32 * b + 16 + 4 * t);
            int cc[4];   // (presetting the accumulator to 1.5 * 2^23 to save the int-to-float step is 0.3-3 % slower here)
            mma_s8_k32(cc, a0, a1, a2, a3, b0, b1);
            sum[mg][0] = fmaf(dA, (float)cc[0], sum[mg][0]);
            sum[mg][1] = fmaf(dA, (float)cc[1], sum[mg][1]);
            sum[mg][2] = fmaf(dB, (float)cc[2], sum[mg][2]);
            sum[mg][3] = fmaf(dB, (float)cc[3], sum[mg][3]);
        }
    }
    add_unit_sums<RAG>(acc, own);
}

// The A operand is 4 * (q - 32) as a signed byte: the low four quant bits at bits 2-5, the high two at bits 6-7
// with the top one flipped (q - 32 is q with bit 5 flipped, read as a 6-bit two's complement; at the top of the
// byte it needs no sign extension). The flip is done once per word of high bits, before the fields are split.
// Four integer instructions per four quants against six for assembling q and then centring it; the factor 4
// leaves with the block scale.

template <int NG, int BY2, class Acc>
__device__ __forceinline__ void unit_q6_k(const uint8_t *blkA, const uint8_t *blkB, int kbase, const int8_t *const (&bp)[NG],
                                          int t, Acc &acc) {
    const Words<BY2> wA(blkA), wB(blkB);
    int I[NG][4];
#pragma unroll
    for (int mg = 0; mg < kFoldGroups<NG>; mg++)
#pragma unroll
        for (int j = 0; j < 4; j++) I[mg][j] = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t qlA[4], qlB[4], qhA[2], qhB[2], scA[2], scB[2];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            qlA[i] = wA(64 * h + 16 * i + 4 * t);
            qlB[i] = wB(64 * h + 16 * i + 4 * t);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            qhA[i] = wA(128 + 32 * h + 16 * i + 4 * t) ^ 0xAAAAAAAAu;
            qhB[i] = wB(128 + 32 * h + 16 * i + 4 * t) ^ 0xAAAAAAAAu;
            scA[i] = wA(192 + 8 * h + 4 * i);
            scB[i] = wB(192 + 8 * h + 4 * i);
        }
        // group G = 2*quad + s covers values 16G..16G+15 of the half (src/quant.cpp:491-512):
        // low 4 bits from ql[32*(quad&1) + 16s ...] (high nibble when quad >= 2), bits 4-5 from
        // qh[16s ...] >> 2*quad.
#pragma unroll
        for (int G = 0; G < 8; G++) {
            const int quad = G >> 1, s = G & 1;
            const uint32_t la = qlA[2 * (quad & 1) + s], lb = qlB[2 * (quad & 1) + s];
            const uint32_t lowA = (quad & 2) ? (la >> 2) : shl_mad<4u>(la);
            const uint32_t lowB = (quad & 2) ? (lb >> 2) : shl_mad<4u>(lb);
            const uint32_t hiA = quad == 0 ? shl_mad<64u>(qhA[s]) : quad == 1 ? shl_mad<16u>(qhA[s]) : quad == 2 ? shl_mad<4u>(qhA[s]) : qhA[s];
            const uint32_t hiB = quad == 0 ? shl_mad<64u>(qhB[s]) : quad == 1 ? shl_mad<16u>(qhB[s]) : quad == 2 ? shl_mad<4u>(qhB[s]) : qhB[s];
            const uint32_t a0 = (lowA & 0x3C3C3C3Cu) | (hiA & 0xC0C0C0C0u);
            const uint32_t a1 = (lowB & 0x3C3C3C3Cu) | (hiB & 0xC0C0C0C0u);
            const int sa = sext_byte(scA[G >> 2], G & 3), sb = sext_byte(scB[G >> 2], G & 3);
#pragma unroll
            for (int mg = 0; mg < kFoldGroups<NG>; mg++) {
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 128 * h + 16 * G + 4 * t);
                int cc[4];
                mma_s8_k16(cc, a0, a1, b0);
                I[mg][0] += sa * cc[0];
                I[mg][1] += sa * cc[1];
                I[mg][2] += sb * cc[2];
                I[mg][3] += sb * cc[3];
            }
        }
    }
    const float dA = 0.25f * __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(blkA + 208)));
    const float dB = 0.25f * __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(blkB + 208)));
    add_unit(acc, dA, dB, I);
}

// A Q2_K super-block (src/quant.cpp:398-424): 16 bytes of (scale | min << 4), 64 bytes of 2-bit quants, d, dmin;
// value = d * scale * q - dmin * min per group of 16. Blocks are 84 bytes, so every word load is aligned. Group
// G = 8n + 2j + s takes bits 2j, 2j+1 of quant bytes 32n + 16s ..+15: one shift and one AND per four quants, one
// k16 MMA per group. The minimums go through one more MMA per super-block, the 16 of them against the group
// sums of X (acc.m, as for Q4_K).
template <int NG, class Acc>
__device__ __forceinline__ void unit_q2_k(const uint8_t *blkA, const uint8_t *blkB, int kbase, const int8_t *const (&bp)[NG],
                                          const int8_t *const (&sp)[NG], int t, Acc &acc) {
    const uint32_t *wa = reinterpret_cast<const uint32_t *>(blkA), *wb = reinterpret_cast<const uint32_t *>(blkB);
    uint32_t scA[4], scB[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        scA[k] = wa[k];
        scB[k] = wb[k];
    }
    int I[NG][4];
#pragma unroll
    for (int mg = 0; mg < kFoldGroups<NG>; mg++)
#pragma unroll
        for (int j = 0; j < 4; j++) I[mg][j] = 0;
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const uint32_t qA[2] = {wa[4 + 8 * n + t], wa[8 + 8 * n + t]}, qB[2] = {wb[4 + 8 * n + t], wb[8 + 8 * n + t]};
#pragma unroll
        for (int js = 0; js < 8; js++) {
            const int j = js >> 1, s = js & 1, G = 8 * n + js;
            const uint32_t a0 = (qA[s] >> (2 * j)) & 0x03030303u, a1 = (qB[s] >> (2 * j)) & 0x03030303u;
            const int sa = (scA[G >> 2] >> (8 * (G & 3))) & 0xF, sb = (scB[G >> 2] >> (8 * (G & 3))) & 0xF;
#pragma unroll
            for (int mg = 0; mg < kFoldGroups<NG>; mg++) {
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 16 * G + 4 * t);
                int cc[4];
                mma_s8_k16(cc, a0, a1, b0);
                I[mg][0] += sa * cc[0];
                I[mg][1] += sa * cc[1];
                I[mg][2] += sb * cc[2];
                I[mg][3] += sb * cc[3];
            }
        }
    }
    const uint32_t hA = wa[20], hB = wb[20];
    const float dA = half_lo(hA), dB = half_lo(hB), nA = half_hi(hA), nB = half_hi(hB);
    const uint32_t m0 = (wa[t] >> 4) & 0x0F0F0F0Fu, m1 = (wb[t] >> 4) & 0x0F0F0F0Fu;   // k slot j = group j: lane t brings 4t..4t+3
    add_unit(acc, dA, dB, I);
#pragma unroll
    for (int mg = 0; mg < NG; mg++) {
        const uint32_t b0 = *reinterpret_cast<const uint32_t *>(sp[mg] + (kbase >> 4) + 4 * t);
        int cc[4];
        mma_s8_k16(cc, m0, m1, b0);
        add_min(acc, nA, nB, cc, mg);
    }
}

// A Q3_K super-block (src/quant.cpp:514-553): 32 mask bytes, 64 bytes of 2-bit quants, sixteen 6-bit scales in 12
// bytes, d; value = d * (scale - 32) * (q2 - (mask bit ? 0 : 4)). The A operand is 32 * (q3 - 4) with q3 = q2 + 4 *
// mask bit: q2 at bits 5-6 and the inverted mask bit at bit 7 (a 3-bit two's complement at the top of the byte),
// two shifts, an AND and an AND-OR per four quants; the 32 leaves with d. Blocks are 110 bytes: every other one is
// 2 bytes off a word boundary.
template <int NG, int BY2, class Acc>
__device__ __forceinline__ void unit_q3_k(const uint8_t *blkA, const uint8_t *blkB, int kbase, const int8_t *const (&bp)[NG],
                                          int t, Acc &acc) {
    const Words<BY2> wA(blkA), wB(blkB);
    uint32_t SA[4], SB[4];
    {
        const uint32_t a0 = wA(96), a1 = wA(100), a2 = wA(104);
        const uint32_t b0 = wB(96), b1 = wB(100), b2 = wB(104);
        // scale i: low four bits in the nibbles of bytes 0..7, high two in byte 8 + i % 4 at bits 2 * (i / 4)
        SA[0] = (a0 & 0x0F0F0F0Fu) | ((a2 << 4) & 0x30303030u);
        SA[1] = (a1 & 0x0F0F0F0Fu) | ((a2 << 2) & 0x30303030u);
        SA[2] = ((a0 >> 4) & 0x0F0F0F0Fu) | (a2 & 0x30303030u);
        SA[3] = ((a1 >> 4) & 0x0F0F0F0Fu) | ((a2 >> 2) & 0x30303030u);
        SB[0] = (b0 & 0x0F0F0F0Fu) | ((b2 << 4) & 0x30303030u);
        SB[1] = (b1 & 0x0F0F0F0Fu) | ((b2 << 2) & 0x30303030u);
        SB[2] = ((b0 >> 4) & 0x0F0F0F0Fu) | (b2 & 0x30303030u);
        SB[3] = ((b1 >> 4) & 0x0F0F0F0Fu) | ((b2 >> 2) & 0x30303030u);
#pragma unroll
        for (int k = 0; k < 4; k++) {   // scale - 32 as signed bytes: add 0x60 (no carry: scale <= 63), flip the sign bit
            SA[k] = (SA[k] + 0x60606060u) ^ 0x80808080u;
            SB[k] = (SB[k] + 0x60606060u) ^ 0x80808080u;
        }
    }
    const uint32_t hmA[2] = {~wA(4 * t), ~wA(16 + 4 * t)};
    const uint32_t hmB[2] = {~wB(4 * t), ~wB(16 + 4 * t)};
    int I[NG][4];
#pragma unroll
    for (int mg = 0; mg < kFoldGroups<NG>; mg++)
#pragma unroll
        for (int j = 0; j < 4; j++) I[mg][j] = 0;
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const uint32_t qA[2] = {wA(32 + 32 * n + 4 * t), wA(48 + 32 * n + 4 * t)};
        const uint32_t qB[2] = {wB(32 + 32 * n + 4 * t), wB(48 + 32 * n + 4 * t)};
#pragma unroll
        for (int js = 0; js < 8; js++) {
            const int j = js >> 1, s = js & 1, G = 8 * n + js, hb = 4 * n + j;
            const uint32_t qa = j < 3 ? (qA[s] << (5 - 2 * j)) : (qA[s] >> 1), qb = j < 3 ? (qB[s] << (5 - 2 * j)) : (qB[s] >> 1);
            const uint32_t a0 = (qa & 0x60606060u) | ((hmA[s] << (7 - hb)) & 0x80808080u);
            const uint32_t a1 = (qb & 0x60606060u) | ((hmB[s] << (7 - hb)) & 0x80808080u);
            const int sa = sext_byte(SA[G >> 2], G & 3), sb = sext_byte(SB[G >> 2], G & 3);
#pragma unroll
            for (int mg = 0; mg < kFoldGroups<NG>; mg++) {
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp[mg] + kbase + 16 * G + 4 * t);
                int cc[4];
                mma_s8_k16(cc, a0, a1, b0);
                I[mg][0] += sa * cc[0];
                I[mg][1] += sa * cc[1];
                I[mg][2] += sb * cc[2];
                I[mg][3] += sb * cc[3];
            }
        }
    }
    const float dA = 0.03125f * __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(blkA + 108)));
    const float dB = 0.03125f * __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(blkB + 108)));
    add_unit(acc, dA, dB, I);
}

// ---- the kernel ------------------------------------------------------------------------------------------
// Three roles, connected only by mbarriers, so no warp ever waits at a CTA-wide barrier while
// weights are streaming:
//   warp 0        producer: bulk-async copies of weight rows into the stage ring. It is the first warp of
//                 the CTA to run, sets the barriers up itself and issues its first copies without waiting
//                 for the other warps to start;
//   warps 1..8    consumers: warp w takes K unit w of every stage (16 rows x 256 values), keeps the
//                 tile's partial sums in registers and hands them over at the end of the tile;
//   warp 9        epilogue: adds the partial sums of each tile in warp order (deterministic),
//                 applies the gate/up fold or the residual add, and writes y.

// SINGLE: 0 the general form; 1 Q4_K with one activation row (unit_q4_k_single); 2 the same with the B
// fragments of the warp's (at most two) K units held in registers, for rows of at most 16 units.
// Either way an SM runs sixteen consumer warps of up to 96 registers: two half-SM CTAs for one or two activation rows,
// one CTA of two consumer groups for more (see consumer_groups).

// RAG: the form for ragged rows of Q6_K and Q3_K, whose units find each word's alignment from its address, and of the 32-value block
// formats (K not a multiple of 256), whose tiles lie on a word boundary or off it as one; compiled apart so that the usual form does not
// carry another copy of the unit. (Q2_K's words are aligned at every row start: its usual form serves ragged rows too.)
// Forms whose two groups may take a tile's stages in turn (StreamParams::by_stage): ragged Q6_K. (Q3_K 4096 x 8960 at four rows
// 19.1 -> 20.0 us with it.)
template <int WT>
__host__ __device__ constexpr bool may_by_stage(bool ragged, int groups) { return WT == KRK_CUDA_Q6_K && ragged && groups == 2; }
// The form of two groups for one and two activation rows: they always take a tile's stages in turn, and a warp prepares the units
// that it multiplies, so no two warps share anything but a tile's sums.
__host__ __device__ constexpr bool in_turn(int ng, int groups) { return ng == 1 && groups == 2; }
// One result in f32 throughout, by one lane: what an infinity among the activations makes of a row (an infinity of either
// sign, or a NaN against a zero weight) is not in the limbs, which give a NaN.
template <int WT>
__device__ __noinline__ float dot_f32(const uint8_t *w, const float *x, int n_in) {
    float sum = 0.0f;
    for (int c = 0; c < n_in >> 5; c++) sum += chunk_dot<WT>(w, c, x);
    return sum;
}

template <int WT, int NG, bool STACK, int SINGLE, bool RAG = false, int GROUPS = consumer_groups(NG), bool WIDE = false>
__global__ void __launch_bounds__(cta_threads(GROUPS), GROUPS == 1 ? 2 : 1)
gemv_stream_kernel(const __grid_constant__ StreamParams p) {
    // STACK: several 16-row tiles per stage (p.tps of them); compiled apart so that the usual one-tile
    // form carries none of its index arithmetic.
    static_assert(!SINGLE || ((WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q4_0) && NG == 1), "the single-row forms are Q4_K and Q4_0");
    const int tps = STACK ? p.tps : 1;
    constexpr int kGroups = GROUPS, kThreads = cta_threads(kGroups), kEpilogueWarp = kGroups * kConsumerWarps + 1;
    constexpr bool kSuper = block_size(WT) == 256, kFold = kSuper && NG > 1;   // AccumSuper, AccumFold
    constexpr bool kFine = RAG && !kSuper;   // four limbs; in the super-block formats: WIDE
    static_assert(!WIDE || kFold, "four limbs of a super-block format: the folded form");
    constexpr bool kInTurn = in_turn(NG, kGroups), kMayByStage = kInTurn || may_by_stage<WT>(RAG, kGroups);
    constexpr int kUnitStep = kInTurn ? 2 * kConsumerWarps : kConsumerWarps;   // from a warp's K unit to its next
    constexpr bool kRagged = RAG || WT == KRK_CUDA_Q2_K;   // p.ragged may be set
    using F = Fmt<WT>;
    using SmemT = Smem<NG, GROUPS>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    SmemT *sm = reinterpret_cast<SmemT *>(smem_raw);
    int8_t *planes = reinterpret_cast<int8_t *>(smem_raw + align_up((int)sizeof(SmemT), 128));
    // one copy of the prepared activation per stacked sub-tile: the warps of a sub-tile move on to the next
    // matrix (and its activation) on their own, so they must not share planes with another sub-tile
    constexpr bool wide = kFine || WIDE;
    int8_t *chunk_sum = planes + tps * plane_bytes<WT>(p.n_in, p.rows, wide);
    uint8_t *stages = reinterpret_cast<uint8_t *>(chunk_sum) + tps * chunk_sum_bytes<WT>(p.n_in, p.rows, p.spread_sums);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_warps = min(kConsumerWarps, p.units * tps);   // consumer warps that ever hold a unit
    const int sub_warps = STACK ? p.units : n_warps;         // warps that share one 16-row tile
    // Programmatic dependent launch: the next kernel in the stream may become resident beside this one
    // (a CTA takes half an SM) as soon as every CTA here has passed this point; it prefetches weights
    // and waits for this grid to complete before touching activations or outputs.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    volatile int *gave_up = &sm->gave_up;
    // Parameters arrive cold in every launch, and a miss holds its warp for some 700 clocks, one line after the other:
    // warps 1..8 fetch a 64-byte line each, side by side (the scalars and the first entries). Q4_K 4096 x 4096 4.61 -> 4.55 us
    // in a chain of launches. Only the single-row forms: the others have the longer start anyway and gain nothing.
    static_assert(kGroups * kConsumerWarps >= 8 && sizeof(StreamParams) >= 8 * 64, "a warp for each of eight lines");
    if (SINGLE && warp >= 1 && warp <= 8 && lane == 0)
        sm->touched[warp] = reinterpret_cast<const int *>(&p)[16 * (warp - 1)];

    if (warp == 0) {
        // ===== producer warp: weights only, so it can run ahead of everything else =====
        // (a lane per barrier)
        static_assert(kMaxStages == 8 && kGroups * red_slots(NG, kGroups) <= kMaxRedSlots && kMaxRedSlots == 4, "24 lanes");
        if (lane < 8) mbar_init(smem_u32(&sm->full[lane]), 1);
        else if (lane < 16) mbar_init(smem_u32(&sm->empty[lane - 8]), kGroups * kConsumerWarps);
        else if (lane < 20) mbar_init(smem_u32(&sm->red_empty[lane - 16]), 1);
        else if (lane < 24) mbar_init(smem_u32(&sm->red_full[lane - 20]), n_warps);
        else if (lane == 24) sm->gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __threadfence_block();
        __syncwarp();
        // the other warps wait for the barriers here before they first look at one; this warp does not wait
        asm volatile("bar.arrive 1, %0;" ::"r"(kThreads) : "memory");
        // A device-side table is the output of the kernel before this one: wait for that grid.
        if (p.dev_table) asm volatile("griddepcontrol.wait;" ::: "memory");
        const TableView tv(p);
        walk<kRagged>(p, tv, tps, [](int) {}, [&](const StageInfo &s) {
            const int slot = s.slot;
            const uint32_t full = smem_u32(&sm->full[slot]), empty = smem_u32(&sm->empty[slot]);
            wait_phase(empty, s.phase ^ 1, gave_up, p.status);
            uint8_t *dst = stages + (size_t)slot * p.stage_bytes;
            const uint8_t *src = tv.w(s.mat) + (size_t)s.row0 * p.row_bytes;
            if (kRagged && !RAG && lane == 0) sm->lead[slot] = 0u;
            if (kRagged && p.ragged) {
                // from the 16-byte boundary below each row's part on; a stage starts a multiple of 8 units (a multiple of 16 bytes in
                // every format) into its rows, so a row lies equally far off in every stage
                const uint32_t a = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15);
                if (lane == 0) sm->lead[slot] = a;   // (and the arrival below, which the consumers wait for, comes after it)
                if (p.use_tma) {
                    if (lane == 0) {
                        mbar_arrive_expect_tx(full, (uint32_t)p.box_bytes);
                        tma_box(smem_u32(dst), &p.wmap[s.mat * p.ragged + s.of], s.unit0 * F::unit_bytes / 8, s.k, 0, full);
                    }
                } else {
                    const uint32_t bytes = (a + min((uint32_t)s.n_units * F::unit_bytes, (uint32_t)(p.row_bytes - s.unit0 * F::unit_bytes)) + 15u) & ~15u;
                    if (lane == 0) mbar_arrive_expect_tx(full, bytes * s.n_rows);
                    __syncwarp();
                    for (int r = lane; r < s.n_rows; r += 32)
                        bulk_g2s(smem_u32(dst + r * p.row_stride), src + (size_t)r * p.ragged * p.row_bytes + (size_t)s.unit0 * F::unit_bytes - a, bytes, full);
                }
            } else if (p.use_tma) {
                // the box is clipped where the matrix ends (rows past n_out, units past the row) and
                // still signals its full size
                if (lane == 0) {
                    mbar_arrive_expect_tx(full, (uint32_t)p.box_bytes);
                    if (p.dev_table) {
                        // (a 64-bit division per stage, by the one lane that issues a copy per stage)
                        const int bank = s.mat % p.step;
                        const int row_off = (int)((size_t)(tv.w(s.mat) - p.bank_base[bank]) / (size_t)p.row_bytes);
                        if constexpr (F::tma == 3) tma_box(smem_u32(dst), &p.wmap[bank], s.unit0 * F::unit_bytes / 8, row_off + s.row0, 0, full);
                        else tma_box(smem_u32(dst), &p.wmap[bank], 0, row_off + s.row0, s.unit0 / p.tma_unit_div, full);
                    } else {
                        if constexpr (F::tma == 3) tma_box(smem_u32(dst), &p.wmap[s.mat], s.unit0 * F::unit_bytes / 8, s.row0, 0, full);
                        else tma_box(smem_u32(dst), &p.wmap[s.mat], 0, s.row0, s.unit0 / p.tma_unit_div, full);
                    }
                }
            } else if (!p.whole_tiles) {
                const uint32_t bytes = (uint32_t)s.n_units * F::unit_bytes;
                if (lane == 0) mbar_arrive_expect_tx(full, bytes * s.n_rows);
                __syncwarp();
                for (int r = lane; r < s.n_rows; r += 32)
                    bulk_g2s(smem_u32(dst + r * p.row_stride),
                             src + (size_t)r * p.row_bytes + (size_t)s.unit0 * F::unit_bytes, bytes, full);
            } else if (lane == 0) {
                // rows are not 16-byte multiples: one copy of the whole tile, rounded down to 16 bytes,
                // and the (< 16 byte, 4-byte granular) tail with plain loads before the arrive
                const uint32_t total = (uint32_t)s.n_rows * p.row_bytes;
                const uint32_t bulk = total & ~15u;
                for (uint32_t o = bulk; o < total; o += 4)
                    *reinterpret_cast<uint32_t *>(dst + o) = *reinterpret_cast<const uint32_t *>(src + o);
                mbar_arrive_expect_tx(full, bulk);
                if (bulk) bulk_g2s(smem_u32(dst), src, bulk, full);
            }
            __syncwarp();
        });
        return;
    }
    if (p.dev_table) asm volatile("griddepcontrol.wait;" ::: "memory");
    const TableView tv(p);
    bool synced = false;   // the barriers are known to be there
    auto sync_start = [&] {
        asm volatile("bar.sync 1, %0;" ::"r"(kThreads) : "memory");
        synced = true;
    };

    if (warp == kEpilogueWarp) {
        // ===== epilogue warp =====
        sync_start();
        // Output (row, activation row) of a tile is the sum, over the consumer warps in warp order, of the
        // share each warp left in `red` (already added up over the four lanes of a row group).
        constexpr int kSlots = red_slots(NG, kGroups);
        float gate_reg[NG];   // silu of the gate tile (stacked tiles keep theirs in shared memory)
        int tile_it = 0, n_out = 0;
        float *y0 = nullptr;
        walk<kRagged>(p, tv, tps, [&](int m) {
            y0 = tv.y(m);
            n_out = tv.n_out(m);
        }, [&](const StageInfo &s) {
            if (!s.last) return;
            // (two groups take the tiles in turn, each through slots of its own)
            const bool both = kMayByStage && (kInTurn || p.by_stage);   // (a tile's sums come from both, through a slot of each)
            const int nth = both ? tile_it : tile_it / kGroups, slot = (both ? 0 : (tile_it % kGroups) * kSlots) + nth % kSlots;
            wait_phase(smem_u32(&sm->red_full[slot]), (nth / kSlots) & 1, gave_up, p.status);
            if (both) wait_phase(smem_u32(&sm->red_full[slot + kSlots]), (nth / kSlots) & 1, gave_up, p.status);
            tile_it++;
            auto sums = [&](const int sub, const int i) {   // of 16 weight rows and activation rows 2i and 2i + 1
                const int idx = lane + 32 * i, row = idx & (kTileRows - 1), r = idx >> 4;   // r = 2*i + (lane >> 4)
                const float *src = reinterpret_cast<const float *>(&sm->red[slot][sub * sub_warps][i][row & 7]) +
                                   2 * (row >> 3) + (r & 1);
                float part[kConsumerWarps];
#pragma unroll
                for (int w = 0; w < kConsumerWarps; w++) part[w] = w < sub_warps ? src[(size_t)w * (NG * 8 * 4)] : 0.0f;
                float v = 0.0f;
#pragma unroll
                for (int w = 0; w < kConsumerWarps; w++) v += part[w];
                if (both) {
                    const float *src1 = src + (size_t)kSlots * (kConsumerWarps * NG * 8 * 4);
#pragma unroll
                    for (int w = 0; w < kConsumerWarps; w++) part[w] = src1[(size_t)w * (NG * 8 * 4)];
#pragma unroll
                    for (int w = 0; w < kConsumerWarps; w++) v += part[w];
                }
                const int srow = kTileRows * sub + row;   // row inside the stage
                const int yrow = s.row0 + (kRagged && p.ragged ? srow * p.ragged : srow);
                if ((kFine || WIDE) && v != v && r < p.rows && srow < s.n_rows) {
                    const int xr = p.table_rows ? p.table_rows[s.mat / p.step * p.rows + r] : r;
                    v = dot_f32<WT>(tv.w(s.mat) + (size_t)yrow * p.row_bytes, tv.x(s.mat) + (size_t)xr * p.n_in, p.n_in);
                }
                if (r < p.rows) {
                    if (p.step == 2 && s.which == 0) {
                        v = __fdiv_rn(v, __fadd_rn(1.0f, exp_as_host(-v)));   // kept for the `up` tile
                        if (STACK) sm->gate[sub][i][lane] = v;
                        else gate_reg[i] = v;
                    } else if (srow < s.n_rows) {
                        if (p.n_peers > 0) {
                            // plain stores into every GPU's copy of the full row (NVLink peer stores)
                            const long long at = (long long)r * p.peer_row_stride + p.peer_offset + yrow;
                            for (int q = 0; q < p.n_peers; q++) p.peer_y[q][at] = v;
                        } else {
                            float *y = y0 + (size_t)r * n_out + yrow;
                            if (p.step == 2) v = __fmul_rn(STACK ? sm->gate[sub][i][lane] : gate_reg[i], v);
                            *y = p.accumulate ? __fadd_rn(*y, v) : v;
                        }
                    }
                }
            };
            if constexpr (STACK && NG > 1 && !(WT == KRK_CUDA_Q5_K && NG == 4)) {
                // This code runs once or a few times in a launch, from a cold instruction cache: where it would be long, it is a loop
                // (Q2_K 4096 x 512 at five rows 10.0 -> 7.3 us, 4096 x 256 9.7 -> 6.9; with one column group 1.00, with one tile to a
                // stage 0.98 to 1.03). Not Q5_K's, which is no longer than it was before rows in phases: at five and more rows of 1024
                // values the consumers lose by it (4736 x 1024 at eight 8.5 -> 8.9; of 512 values 0.95 to 0.99 of the time).
#pragma unroll 1
                for (int sub = 0; sub < tps; sub++) {
#pragma unroll (NG == 4 ? 1 : NG)
                    for (int i = 0; i < NG; i++) sums(sub, i);
                }
            } else {
#pragma unroll
                for (int sub = 0; sub < (STACK ? kMaxStack : 1); sub++) {
                    if (sub >= tps) break;
#pragma unroll
                    for (int i = 0; i < NG; i++) sums(sub, i);
                }
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&sm->red_empty[slot]));
                if (both) mbar_arrive(smem_u32(&sm->red_empty[slot + kSlots]));
            }
        });
        if (p.n_peers > 0) {
            // This CTA's stores are out. The CTA that reports last publishes the epoch to every peer and
            // then waits (bounded) until every peer has published the same epoch here, so that the end
            // of this kernel is the end of the all-gather on this GPU. The count of CTAs that have
            // reported lives behind this GPU's own flags (word n_peers + 1), one per exchange object.
            __threadfence_system();
            __syncwarp();
            int *own = p.peer_flag[p.my_rank];
            unsigned *done_counter = reinterpret_cast<unsigned *>(own + p.n_peers + 1);
            unsigned done = 0;
            if (lane == 0) done = atomicAdd(done_counter, 1u);
            done = __shfl_sync(0xffffffffu, done, 0);
            if (done == gridDim.x - 1) {
                int epoch = p.epoch;
                if (lane == 0) {
                    *done_counter = 0;
                    if (epoch == 0) {   // device-counted steps: the count lives behind this GPU's flags
                        epoch = own[p.n_peers] + 1;
                        own[p.n_peers] = epoch;
                    }
                    __threadfence_system();
                    for (int q = 0; q < p.n_peers; q++) *reinterpret_cast<volatile int *>(p.peer_flag[q] + p.my_rank) = epoch;
                    __threadfence_system();
                }
                epoch = __shfl_sync(0xffffffffu, epoch, 0);
                if (p.wait_peers && lane < p.n_peers) {
                    const long long t0 = clock64();
                    while (*reinterpret_cast<const volatile int *>(own + lane) < epoch) {
                        __nanosleep(100);
                        if (clock64() - t0 > kWaitCycles) {
                            atomicExch(p.status, KRK_CUDA_ETIMEOUT);
                            break;
                        }
                    }
                }
                __threadfence_system();
            }
        }
        return;
    }

    // ===== consumer warps =====
    const int grp = kGroups == 1 ? 0 : (warp - 1) / kConsumerWarps;   // consumer group: takes every other tile, or every other stage (by_stage)
    const int wid = warp - 1 - grp * kConsumerWarps, g = lane >> 2, t = lane & 3;
    const float *prepared = nullptr;
    int prepared_row = 0;
    const int8_t *bp[NG], *sp[NG];
    const float *fe[NG], *fo[NG];   // Q5_1: per-block sums of the even / odd activation row of each column group
    float xs[2 * NG];   // this warp's scale of each activation row (kFold: of its own rows, xs[0] and xs[1])
    std::conditional_t<kSuper, AccumSuper<NG, WIDE>, Accum<NG>> acc;
    AccumSingle acs;
    accum_zero(acc);
    acs.f[0] = acs.f[1] = acs.m[0] = acs.m[1] = acs.m[2] = acs.m[3] = 0.0f;
    int tile_it = 0;
    // With stacked tiles warp w holds unit w % units of sub-tile w / units of every stage; otherwise units
    // w, w + 8, ... of the stage (a stage holds at most 8 units unless it is one whole tile).
    const int my_sub = STACK ? wid / p.units : 0;
    const int my_unit = STACK ? wid - my_sub * p.units : wid;
    const bool stacked_idle = STACK && my_sub >= tps;
    const uint32_t lane_off = (uint32_t)(kTileRows * my_sub + g) * p.row_stride;
    if (!stacked_idle) {
        planes += my_sub * plane_bytes<WT>(p.n_in, p.rows, wide);
        chunk_sum += my_sub * chunk_sum_bytes<WT>(p.n_in, p.rows, p.spread_sums);
    }
    // single-row form: column g = limb g/2 of the low (g even) or high (g odd) chunk of a group
    const int8_t *bq = planes + (g < 6 ? (g >> 1) * plane_pitch<WT>(p.n_in, p.rows) + (WT == KRK_CUDA_Q4_0 ? 16 : 32) * (g & 1) : 0);
    const int8_t *sq = chunk_sum + (g & 3) * sum_pitch<WT>(p.n_in, p.spread_sums);
    BFrag held[2];

    // The same walk as walk() above, written flat: per stage a consumer warp only needs the ring
    // slot and its K units, not which matrix or rows the tile belongs to.
    const int n_chunks = p.whole_tiles ? 1 : (p.units + kConsumerWarps - 1) / kConsumerWarps;
    const uint32_t full0 = smem_u32(&sm->full[0]), empty0 = smem_u32(&sm->empty[0]);
    int slot = 0;
    uint32_t phase = 0;
    // (What only the step from one entry to the next needs is worked out there again: registers are short in the tile loop, and
    // spilled ones miss level 1 at their first use in a launch.)
    for (int e = -1;;) {
        int cta;
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta));
        const TableView tv(p);
        const int g0 = cta * tv.gran_q + min(cta, tv.gran_r);
        const int g1 = g0 + tv.gran_q + (cta < tv.gran_r ? 1 : 0);
        e = e < 0 ? tv.first(g0) : e + 1;
        if (e >= tv.n_entries || tv.begin(e) >= g1) break;
        const int lo = max(g0, tv.begin(e)), hi = min(g1, tv.begin(e + 1));
        if (lo >= hi) continue;
        const int m = e * p.step;
        const int r0 = (lo - tv.begin(e)) * p.gran;
        const int r1 = min(tv.n_out(m), (hi - tv.begin(e)) * p.gran);
        const float *x = tv.x(m);
        // lane r: which row of x is activation row r
        const bool picked = !SINGLE && p.table_rows;
        const int my_row = picked && lane < p.rows ? p.table_rows[e * p.rows + lane] : lane;
        if (x != prepared || (picked && __any_sync(0xFFFFFFFFu, my_row != prepared_row))) {
            const int first_unit = stacked_idle ? p.units : my_unit + (kInTurn ? kConsumerWarps * grp : 0);
            // x may be the output of the kernel before this one (and y its input): wait for that grid to
            // complete. Weights are never written by a kernel in flight, so the producer warp does not wait.
            if (prepared == nullptr) {
                // (x to level 2 meanwhile, where it is coherent whoever still writes it: a lane per 128-byte line of the warp's slices)
                constexpr int kLines = F::unit_values / 32;
                if (!p.dev_table)   // (a table's launch has waited)
                    for (int r = kInTurn ? 0 : grp; r < (SINGLE ? 1 : p.rows); r += kInTurn ? 1 : kGroups)
                        for (int l = lane; first_unit + l / kLines * kUnitStep < p.units; l += 32) {
                            const int k = (first_unit + l / kLines * kUnitStep) * F::unit_values + l % kLines * 32;
                            if (!kFine || k < p.n_in) asm volatile("prefetch.global.L2 [%0];" ::"l"(x + (size_t)r * p.n_in + k));
                        }
                asm volatile("griddepcontrol.wait;" ::: "memory");
            }
            // (stacked tiles: every sub-tile prepares its own copy)
            auto row = [&](int r) { return x + (SINGLE ? (size_t)0 : (size_t)__shfl_sync(0xFFFFFFFFu, my_row, r) * p.n_in); };
            if (kGroups == 1 || kInTurn) {   // every warp prepares what it reads itself
#pragma unroll
                for (int r = 0; r < 2 * NG; r++) xs[r] = 0.0f;
                prepare_x<WT, kFine, WIDE, kLoadsAhead<WT, NG, RAG>, (NG > 1), kUnitStep>(row, [&](int r, float v) {
#pragma unroll
                    for (int q = 0; q < 2 * NG; q++) xs[q] = q == r ? v : xs[q];
                }, 0, 1, SINGLE ? 1 : p.rows, p, planes, chunk_sum, first_unit, lane);
                __syncwarp();
                if (!synced) sync_start();
            } else {
                // each group prepares every other row; nobody may still read the activation before this one
                if (prepared != nullptr) asm volatile("bar.sync 2, %0;" ::"n"(kGroups * kConsumerThreads) : "memory");
                prepare_x<WT, kFine, WIDE, kLoadsAhead<WT, NG, RAG>, (NG > 1), kConsumerWarps>(row, [&](int r, float v) {
                    if (lane == 0) sm->scale[NG == 1 ? 0 : wid][r] = v;
                }, grp, kGroups, p.rows, p, planes, chunk_sum, first_unit, lane);
                if (!synced) sync_start();
                else asm volatile("bar.sync 2, %0;" ::"n"(kGroups * kConsumerThreads) : "memory");
#pragma unroll
                for (int r = 0; r < (kFold ? kFoldRows<NG> : 2 * NG); r++) {
                    const int row = kFold ? t + 4 * r : r;
                    xs[r] = row < p.rows ? sm->scale[NG == 1 ? 0 : wid][row] : 0.0f;
                }
            }
            // (zero already, but not held over the preparation, where registers are short: ragged Q6_K 4096 x 2304 at four rows 9 % less)
            if (NG == 4 || (RAG && kSuper && kGroups == 2)) accum_zero(acc);
            prepared = x;
            prepared_row = my_row;
            if (!SINGLE) lane_planes<WT, NG, kFold, kFine || WIDE>(planes, chunk_sum, p.n_in, sum_pitch<WT>(p.n_in, p.spread_sums), p.rows, g, bp, sp, wide);
            if (WT == KRK_CUDA_Q5_1) {
#pragma unroll
                for (int mg = 0; mg < NG; mg++) {   // per-block sums of the group's even and odd activation rows
                    fe[mg] = reinterpret_cast<const float *>(chunk_sum) + (size_t)min(2 * mg, p.rows - 1) * (p.n_in >> 5);
                    fo[mg] = reinterpret_cast<const float *>(chunk_sum) + (size_t)min(2 * mg + 1, p.rows - 1) * (p.n_in >> 5);
                }
            }
            if (SINGLE == 2 && !stacked_idle) {
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int u = my_unit + j * kConsumerWarps;
                    if (u < p.units) held[j] = load_bfrag(bq + u * F::unit_values, sq + ((u * F::unit_values) >> 5), t);
                }
            }
        }
        const int stage_rows = kTileRows * tps;
        const int n_tiles = (RAG || (kRagged && p.ragged) ? hi - lo : (r1 - r0 + stage_rows - 1) / stage_rows) * p.step;
        for (int tile = 0; tile < n_tiles; tile++) {
            // the other group's stage: it is seen to land (a ring slot's parity only tells two laps apart for a warp that looks at
            // every lap) and given back
            auto pass = [&] {
                wait_phase(full0 + 8 * slot, phase, gave_up, p.status);
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * slot);
                if (++slot == p.n_stages) {
                    slot = 0;
                    phase ^= 1;
                }
            };
            const bool by_stage = kMayByStage && (kInTurn || p.by_stage);
            if (kGroups == 2 && !by_stage && tile_it % 2 != grp) {
                tile_it++;
                for (int ck = 0; ck < n_chunks; ck++) pass();
                continue;
            }
            // one stage of the tile: `bf` are the warp's held B fragments for it (SINGLE == 2), else unused
            auto stage = [&](const int ck, const BFrag &bf) {
                wait_phase(full0 + 8 * slot, phase, gave_up, p.status);
                const int stage_units = p.whole_tiles ? p.units : min(kConsumerWarps, p.units - ck * kConsumerWarps);
                if (!stacked_idle) {
                    const uint32_t lead = kRagged ? sm->lead[slot] : 0u;   // (0 where rows are not ragged)
                    const bool by2 = kFine && (lead & 2u);   // rows start 2 bytes off a word boundary
                    const uint8_t *tile0 = stages + (size_t)slot * p.stage_bytes + lane_off + lead;
                    for (int su = my_unit; su < stage_units; su += kConsumerWarps) {
                        const uint8_t *rowA = tile0 + (size_t)su * p.unit_stride;
                        const uint8_t *rowB = tile0 + (size_t)su * p.unit_stride + (size_t)8 * p.row_stride;
                        const int unit = ck * kConsumerWarps + su;
                        const int kbase = unit * F::unit_values;
                        const int nb = (p.n_in - kbase) >> 5;   // 32-value blocks of the unit (short rows: fewer than a full unit's)
                        if constexpr (WT == KRK_CUDA_Q4_0 && !SINGLE) {
                            if (by2) unit_q4_0_rows<NG, RAG, 1>(rowA, rowB, kbase, bp, t, acc, nb);
                            else unit_q4_0_rows<NG, RAG, 0>(rowA, rowB, kbase, bp, t, acc, nb);
                        } else if constexpr (WT == KRK_CUDA_Q4_0) {
                            unit_q4_0(rowA, rowB, bq + kbase, reinterpret_cast<const float *>(chunk_sum) + (kbase >> 5), t, acs);
                        } else if constexpr (SINGLE == 2) {
                            unit_q4_k_single(rowA, rowB, bf, t, acs);
                        } else if constexpr (SINGLE == 1) {
                            unit_q4_k_single(rowA, rowB, load_bfrag(bq + kbase, sq + (kbase >> 5), t), t, acs);
                        } else if constexpr (WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q5_K) {
                            unit_q4_k<NG, WT == KRK_CUDA_Q5_K>(rowA, rowB, kbase, bp, sp, t, acc);
                        } else if constexpr (WT == KRK_CUDA_Q8_0) {
                            if (by2) unit_q8_0<NG, RAG, 1>(rowA, rowB, kbase, bp, t, acc, nb);
                            else unit_q8_0<NG, RAG, 0>(rowA, rowB, kbase, bp, t, acc, nb);
                        } else if constexpr (WT == KRK_CUDA_Q5_0) {
                            if (by2) unit_q5_0<NG, RAG, 1>(rowA, rowB, kbase, bp, t, acc, nb);
                            else unit_q5_0<NG, RAG, 0>(rowA, rowB, kbase, bp, t, acc, nb);
                        } else if constexpr (WT == KRK_CUDA_IQ4_NL) {
                            if (by2) unit_iq4_nl<NG, RAG, 1>(rowA, rowB, kbase, bp, t, acc, nb);
                            else unit_iq4_nl<NG, RAG, 0>(rowA, rowB, kbase, bp, t, acc, nb);
                        } else if constexpr (WT == KRK_CUDA_Q2_K) {
                            unit_q2_k<NG>(rowA, rowB, kbase, bp, sp, t, acc);
                        } else if constexpr (WT == KRK_CUDA_Q3_K) {
                            if (RAG) unit_q3_k<NG, 2>(rowA, rowB, kbase, bp, t, acc);
                            else if (unit & 1) unit_q3_k<NG, 1>(rowA, rowB, kbase, bp, t, acc);
                            else unit_q3_k<NG, 0>(rowA, rowB, kbase, bp, t, acc);
                        } else if constexpr (WT == KRK_CUDA_Q5_1) {
                            unit_q5_1<NG, RAG>(rowA, rowB, kbase, bp, fe, fo, t, acc, nb);
                        } else {
                            if (RAG) unit_q6_k<NG, 2>(rowA, rowB, kbase, bp, t, acc);
                            else if (unit & 1) unit_q6_k<NG, 1>(rowA, rowB, kbase, bp, t, acc);
                            else unit_q6_k<NG, 0>(rowA, rowB, kbase, bp, t, acc);
                        }
                    }
                }
                // The stage is given back when its words HAVE arrived: an arrival does not wait for shared-memory loads in
                // flight (see the decode warps of krk_gemm_tc.cu), and the copy of the next stage into this slot would meet
                // them. All that was loaded is in the sums by now, so the arrival waits for those. Lane 0's do for the warp:
                // what they were loaded by and multiplied by are instructions of the whole warp, which complete as one.
                __syncwarp();
                if (lane == 0) {
                    if constexpr (SINGLE != 0) mbar_arrive_after(empty0 + 8 * slot, __float_as_uint(acs.f[0]), __float_as_uint(acs.f[1]));
                    else mbar_arrive_after(empty0 + 8 * slot, bits_of(acc), 0u);
                }
                if (++slot == p.n_stages) {
                    slot = 0;
                    phase ^= 1;
                }
            };
            if (SINGLE == 2) {   // at most two stages per tile, each with its own registers
                stage(0, held[0]);
                if (n_chunks > 1) stage(1, held[1]);
            } else {
                for (int ck = 0; ck < n_chunks; ck++) {
                    if (by_stage && (ck & 1) != grp) pass();
                    else stage(ck, held[0]);
                }
            }
            {
             // ---- end of the tile: the lanes of a row group add their weighted shares ----
             constexpr int kSlots = red_slots(NG, kGroups);
             const int nth = by_stage ? tile_it : tile_it / kGroups, rslot = grp * kSlots + nth % kSlots;
             const uint32_t rphase = (nth / kSlots) & 1;
             tile_it++;
             if (wid >= n_warps) continue;
             if constexpr (kFold) {
                 float o[kFoldRows<NG>][2];
#pragma unroll
                 for (int h = 0; h < kFoldRows<NG>; h++)
#pragma unroll
                     for (int b = 0; b < 2; b++) {
                         o[h][b] = acc.a[h][b] * xs[h];
                     }
                 accum_zero(acc);
                 wait_phase(smem_u32(&sm->red_empty[rslot]), rphase ^ 1, gave_up, p.status);
#pragma unroll
                 for (int h = 0; h < kFoldRows<NG>; h++) {
                     const int r = t + 4 * h;
                     float *dst = reinterpret_cast<float *>(&sm->red[rslot][wid][r >> 1][g]) + (r & 1);
                     dst[0] = o[h][0];   // weight row g
                     dst[2] = o[h][1];   // g + 8
                 }
             } else {
                 // minimum columns: limb c%4 (weights 2^24, 2^16, 2^8, 1) of activation row c/4
                 const float me0 = t == 0 ? 16777216.0f : (t == 1 ? 256.0f : 0.0f), me1 = t == 0 ? 65536.0f : (t == 1 ? 1.0f : 0.0f);
                 float4 o[NG];
                 if constexpr (SINGLE != 0) {
                     // lane t holds limb t (weights 65536, 256, 1) of rows g and g+8, times 16
                     // (Q4_0: lane t = 3 holds d * sum of X per block, the -8 of every quant)
                     const float wl = t == 0 ? 4096.0f : (t == 1 ? 16.0f : (t == 2 ? 0.0625f : (WT == KRK_CUDA_Q4_0 ? -8.0f : 0.0f)));
                     o[0].x = (wl * acs.f[0] - fmaf(me0, acs.m[0], me1 * acs.m[1])) * xs[0];
                     o[0].z = (wl * acs.f[1] - fmaf(me0, acs.m[2], me1 * acs.m[3])) * xs[0];
                     o[0].y = o[0].w = 0.0f;
                     acs.f[0] = acs.f[1] = acs.m[0] = acs.m[1] = acs.m[2] = acs.m[3] = 0.0f;
                 } else {
                     // Column c of a group carries limb c%3 (weights 65536, 256, 1) of activation row c/3; this lane
                     // holds columns 2t and 2t+1, so its accumulators enter the even activation row with (we0, we1)
                     // and the odd one with (wo0, wo1). The minimum term is already a per-lane partial sum. Four limbs: limb c%4
                     // (weights 65536, 256, 1, 1/256) of row c/4.
                     const float w0 = t & 1 ? 1.0f : 65536.0f, w1 = t & 1 ? 0.00390625f : 256.0f;
                     const float we0 = kFine ? (t < 2 ? w0 : 0.0f) : t == 0 ? 65536.0f : (t == 1 ? 1.0f : 0.0f), we1 = kFine ? (t < 2 ? w1 : 0.0f) : t == 0 ? 256.0f : 0.0f;
                     const float wo0 = kFine ? (t < 2 ? 0.0f : w0) : t == 2 ? 256.0f : 0.0f, wo1 = kFine ? (t < 2 ? 0.0f : w1) : t == 1 ? 65536.0f : (t == 2 ? 1.0f : 0.0f);
#pragma unroll
                     for (int mg = 0; mg < NG; mg++) {
                         if (NG == 4 && mg == 3 && !kFine) {
                             // activation rows 6 and 7 rode in columns 6 and 7 (lane t = 3) of groups 0..2, limb mg in group mg
                             const float w0 = t == 3 ? 65536.0f : 0.0f, w1 = t == 3 ? 256.0f : 0.0f, w2 = t == 3 ? 1.0f : 0.0f;
                             o[mg].x = fmaf(w0, acc.f[0][0], fmaf(w1, acc.f[1 % NG][0], w2 * acc.f[2 % NG][0]));
                             o[mg].y = fmaf(w0, acc.f[0][1], fmaf(w1, acc.f[1 % NG][1], w2 * acc.f[2 % NG][1]));
                             o[mg].z = fmaf(w0, acc.f[0][2], fmaf(w1, acc.f[1 % NG][2], w2 * acc.f[2 % NG][2]));
                             o[mg].w = fmaf(w0, acc.f[0][3], fmaf(w1, acc.f[1 % NG][3], w2 * acc.f[2 % NG][3]));
                         } else {
                             o[mg].x = fmaf(we0, acc.f[mg][0], we1 * acc.f[mg][1]);   // row g,   even activation row
                             o[mg].y = fmaf(wo0, acc.f[mg][0], wo1 * acc.f[mg][1]);   // row g,   odd
                             o[mg].z = fmaf(we0, acc.f[mg][2], we1 * acc.f[mg][3]);   // row g+8, even
                             o[mg].w = fmaf(wo0, acc.f[mg][2], wo1 * acc.f[mg][3]);   // row g+8, odd
                         }
                         if constexpr (WT == KRK_CUDA_Q4_K || WT == KRK_CUDA_Q5_K || WT == KRK_CUDA_Q2_K) {
                             const float mo0 = t == 2 ? 16777216.0f : (t == 3 ? 256.0f : 0.0f), mo1 = t == 2 ? 65536.0f : (t == 3 ? 1.0f : 0.0f);
                             o[mg].x -= fmaf(me0, acc.m[0], me1 * acc.m[1]);
                             o[mg].y -= fmaf(mo0, acc.m[0], mo1 * acc.m[1]);
                             o[mg].z -= fmaf(me0, acc.m[2], me1 * acc.m[3]);
                             o[mg].w -= fmaf(mo0, acc.m[2], mo1 * acc.m[3]);
                         }
                         o[mg].x *= xs[2 * mg];
                         o[mg].y *= xs[2 * mg + 1];
                         o[mg].z *= xs[2 * mg];
                         o[mg].w *= xs[2 * mg + 1];
                     }
                     accum_zero(acc);
                 }
#pragma unroll
                 for (int mg = 0; mg < NG; mg++) {
#pragma unroll
                     for (int d = 1; d <= 2; d <<= 1) {   // (t0 + t1) + (t2 + t3): a fixed order
                         o[mg].x += __shfl_xor_sync(0xFFFFFFFFu, o[mg].x, d);
                         o[mg].z += __shfl_xor_sync(0xFFFFFFFFu, o[mg].z, d);
                         if (!SINGLE) {
                             o[mg].y += __shfl_xor_sync(0xFFFFFFFFu, o[mg].y, d);
                             o[mg].w += __shfl_xor_sync(0xFFFFFFFFu, o[mg].w, d);
                         }
                     }
                 }
                 wait_phase(smem_u32(&sm->red_empty[rslot]), rphase ^ 1, gave_up, p.status);
                 if (t == 0) {
#pragma unroll
                     for (int mg = 0; mg < NG; mg++) sm->red[rslot][wid][mg][g] = o[mg];
                 }
             }
             __syncwarp();
             if (lane == 0) mbar_arrive(smem_u32(&sm->red_full[rslot]));
            }
        }
    }
    if (!synced) sync_start();   // (a CTA without work)
}

template <int WT, int NG, bool STACK, int SINGLE, bool RAG = false, int GROUPS = consumer_groups(NG), bool WIDE = false>
int launch_one(const StreamParams &p, int grid, size_t smem, cudaStream_t st) {
    static bool configured[64] = {};   // per instantiation and device: the opt-in is sticky
    auto kernel = gemv_stream_kernel<WT, NG, STACK, SINGLE, RAG, GROUPS, WIDE>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemWhole);
        // all of the SM's configurable memory as shared memory, so that two CTAs fit
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) {
            note_cuda_error(e);
            return KRK_CUDA_ELAUNCH;
        }
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(cta_threads(GROUPS));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
    note_launch(1, KRK_CUDA_FAMILY_GEMV_STREAM);
    if (e != cudaSuccess) {
        note_cuda_error(e);
        (void)cudaGetLastError();
        return KRK_CUDA_ELAUNCH;
    }
    return KRK_CUDA_OK;
}

// StreamParams::by_stage. Two groups that take tiles in turn want a ring that holds a tile of each: a stage of the second tile only
// lands when one of the first is done with. Where it does not, they take a tile's stages in turn (Q6_K at four rows, stages to a
// tile and in the ring: 16384 x 6656, 4 and 4, 39.8 -> 37.9 us; x 8960, 5 and 3, 51.6 -> 50.1; x 11008, 6 and 3, 62.3 -> 58.0;
// three rows of x 14592, 8 and 3, 83.2 -> 75.6). Not of three stages, which leave one group twice the other's (14.9 -> 15.3), and
// not in a ring of two, where each group holds one stage and none is on its way (four rows of 4096 x 12544 29.1 -> 31.2, six of
// 16384 x 8960 69.3 -> 71.8), unless no CTA has a second tile, so that one group would have nothing to do (five rows of
// 1024 x 10496 20.1 -> 18.7, eight of x 6656 16.6 -> 15.6). Only in the forms for ragged rows: the others would lose 2 to 4 % to the
// code and gain nothing (Q4_K 4096 x 11008 17.5 -> 18.7 us).
template <int WT>
bool stages_in_turn(const StreamParams &p, bool one_tile) {
    const int tile_stages = (p.units + kConsumerWarps - 1) / kConsumerWarps;
    return may_by_stage<WT>(p.ragged != 0, p.groups) && tile_stages > 3 && p.n_stages < 2 * tile_stages && (p.n_stages >= 3 || one_tile);
}

// Bytes from row to row of a box that brings `bytes` of each (a multiple of 8): the eight rows of a fragment load meet on different
// banks where it is an odd multiple of 16, and what a box brings beyond a row's part is never looked at. One copy a stage in
// place of one a row: from a lane per row a copy takes 82 clocks to issue whatever its size, 13 bytes a clock and SM at Q8_0's 1088
// (128256 x 4096 101.5 -> 84.2 us, 1.0 of the copy bandwidth; 22016 x 4096 at one, four and eight rows 21.2, 26.7, 40.2 -> 18.5, 23.1, 29.5;
// Q3_K 22016 x 4096 18.4 -> 17.1, Q2_K 16.2 -> 14.8).
__host__ __device__ constexpr int box_pitch(int bytes) { return align_up(bytes, 16) + (align_up(bytes, 16) / 16 % 2 == 0 ? 16 : 0); }

// Whether one or two activation rows may go to two groups of consumer warps that take a tile's stages in turn (in_turn), one CTA
// to an SM. They do where a half SM has no room for the ring (one group left an SM with eight warps: Q6_K 4096 x 11008 13.9 -> 12.8 us, Q8_0 at
// two rows 15.6 -> 13.2), and where no CTA has a second tile and a tile has many stages (Q4_K 1024 x 8192 6.2 -> 4.7, 2080 x 11008 8.7 -> 6.3;
// at 4608 values, two stages and a part of a third, 0.85 to 1.16 of the time, so from beyond 5120 on; up to 8192 not where tiles for
// nearly all SMs would give up the next launch's early start, 2368 x 5632 1.00 to 1.06). A model's pass shows the same at one row (2048 /
// 8192 values 0.80 to 0.93 of the time, 1792 / 6912 0.82 to 0.95, 2048 / 5632 0.85 to 1.03), and at two through the backend (against one
// group from four fifths of the SMs on: 2048 / 8192 Q8_0 0.90 of the time, IQ4_NL 0.91, Q4_K 0.94; 2048 / 5632 0.95 to 0.99, 2304 / 8704 0.92 to
// 1.01; called matrix by matrix 0.96 to 1.08, most 1.00). Up to 4096 values results keep the order of their sums, in which eight warps add their units one after the other; beyond 5120 it
// goes by the rows of a launch's matrices (of a slice of a head, by those of the whole, see setup_launch).
template <int WT>
bool stages_halve(const StreamParams &p) {
    return p.tps == 1 && !p.whole_tiles && p.units > kConsumerWarps && (p.n_in > 4096 || fine_limbs<WT>(p.n_in));
}

// Fills the fields that depend only on the format, the width and the activation row count.
// Returns false when the streaming kernel does not address the shape.
template <int WT>
bool setup_format(StreamParams &p, int64_t n_in, int rows, int silu_pair, size_t *smem_out, bool want_tma = false, bool one_group = false,
                  bool whole_sm = false, bool wide = false) {
    using F = Fmt<WT>;
    // K not a multiple of 256: whole 32-value blocks, rows copied the ragged way, the last unit short. (Below 256 values
    // there is little to stream, and the warp-per-row kernel serves.)
    const bool odd_k = n_in % 256 != 0;
    if ((odd_k && (block_size(WT) != 32 || n_in % 32 != 0 || n_in < 256)) || n_in > (1 << 20) || rows < 1 || rows > KRK_CUDA_MAX_ROWS) return false;
    p.n_in = (int)n_in;
    p.units = (int)((n_in + F::unit_values - 1) / F::unit_values);
    p.row_bytes = (int)row_bytes(WT, n_in);
    p.rows = rows;
    const bool pair = rows <= 2 && !(wide && block_size(WT) == 256);   // the form for two rows, not that for three and four
    p.groups = pair || one_group ? 1 : 2;
    p.accumulate = 0;
    p.step = silu_pair ? 2 : 1;
    p.whole_tiles = 0;
    p.ragged = 0;
    p.gran = 1;
    p.dev_table = nullptr;
    p.table_rows = nullptr;
    p.entry_gran = 0;
    p.n_peers = 0;
    p.my_rank = p.epoch = 0;
    p.peer_row_stride = p.peer_offset = 0;
    if (WT == KRK_CUDA_Q6_K && (n_in % 2048) != 0) {
        // 210-byte blocks: rows are 16-byte multiples only for K % 2048 == 0. Otherwise whole 16-row
        // tiles are copied contiguously (needs 4-byte-multiple rows and the tile in one stage), or, for longer
        // or odd rows (K = 11008: 9030 bytes), rows that lie alike together, see TilePlace.
        if ((p.row_bytes & 3) == 0 && p.units <= 2 * kConsumerWarps) {
            p.whole_tiles = 1;
            p.gran = 8;
        } else {
            p.ragged = 1;
        }
    }
    // Q2_K rows are 16-byte multiples for K % 1024 == 0, Q3_K rows for K % 2048 == 0
    if ((WT == KRK_CUDA_Q2_K || WT == KRK_CUDA_Q3_K) && (p.row_bytes & 15) != 0) p.ragged = 1;
    if (odd_k || (wide && block_size(WT) == 32)) p.ragged = 1;   // (wide: for the form of four limbs, whose rows may be 16-byte multiples too)
    if (p.ragged) p.ragged = p.row_bytes & 2 ? 8 : p.row_bytes & 4 ? 4 : 2;
    const int ku_max = p.whole_tiles ? p.units : (p.units < kConsumerWarps ? p.units : kConsumerWarps);
    p.tps = kConsumerWarps / p.units;   // 0 when a tile has more units than there are consumer warps
    p.tps = p.tps < 1 ? 1 : (p.tps > kMaxStack ? kMaxStack : p.tps);
    // (what decides whether a shape is taken, see below, and is the pitch of row copies of 16-byte multiples)
    const int raw = ku_max * F::unit_bytes + (p.ragged ? 48 : 0), rows_stride = raw + ((F::stride_mod - raw % 128) + 128) % 128;
    p.use_tma = 0;
    p.box_bytes = 0;
    p.unit_stride = F::unit_bytes;
    p.tma_unit_div = 1;
    if (want_tma && F::tma == 1 && !p.whole_tiles && !p.ragged) {
        // a stage is one tensor copy: [units of the stage][rows of the stage][unit_bytes]. The 144-byte
        // pitch of a Q4_K unit puts the eight rows of a fragment load 16 bytes apart in the banks.
        p.use_tma = 1;
        p.row_stride = F::unit_bytes;
        p.unit_stride = kTileRows * p.tps * F::unit_bytes;
        p.box_bytes = ku_max * p.unit_stride;
        p.stage_bytes = align_up(p.box_bytes, 128);
        p.gran = kTileRows * p.tps;   // a copy brings whole tiles: CTAs split the rows at tile boundaries, so no row is fetched twice
    } else if (want_tma && F::tma == 2 && !p.whole_tiles && ku_max == kConsumerWarps && p.units % kConsumerWarps == 0) {
        // a stage is one tensor copy of eight units of each row: [row][8 units], pitch 8 * unit_bytes (1680 for
        // Q6_K: the rows of a fragment load again lie 16 bytes apart in the banks)
        p.use_tma = 2;
        p.tma_unit_div = kConsumerWarps;
        p.row_stride = ku_max * F::unit_bytes;
        p.box_bytes = kTileRows * p.tps * p.row_stride;
        p.stage_bytes = align_up(p.box_bytes, 128);
        p.gran = kTileRows * p.tps;
    } else if (p.ragged || (want_tma && F::tma == 3)) {
        p.use_tma = want_tma ? 3 : 0;
        p.row_stride = box_pitch(ku_max * F::unit_bytes + (p.ragged ? 14 : 0));
        p.box_bytes = kTileRows * p.tps * p.row_stride;
        p.stage_bytes = align_up(p.box_bytes, 128);
        p.gran = kTileRows * p.tps;
    } else if (p.whole_tiles) {
        p.row_stride = p.row_bytes;
        p.stage_bytes = align_up(kTileRows * p.tps * p.row_bytes, 128);
    } else {
        p.row_stride = rows_stride;
        p.stage_bytes = align_up(kTileRows * p.tps * p.row_stride, 128);
    }
    const int smem_struct = pair ? (int)sizeof(Smem<1>) : one_group ? (int)sizeof(Smem<2, 1>) : rows <= 4 ? (int)sizeof(Smem<2>) : (int)sizeof(Smem<4>);
    // Depth of the ring: as many stages as fit beside the prepared activation in half an SM, at most kMaxHalfStages. Wide
    // activations (large K) leave too little of a half; they, and the forms of two consumer groups, take the whole SM.
    bool halves = p.groups == 1;
    int most = halves ? kMaxHalfStages : kMaxStages;
    auto fixed_bytes = [&](int spread) {
        return align_up(smem_struct, 128) + p.tps * (plane_bytes<WT>(p.n_in, rows, wide) + chunk_sum_bytes<WT>(p.n_in, rows, spread));
    };
    auto depth = [&](int fixed, bool half) {
        const int fit = ((half ? kSmemLimit : kSmemWhole) - fixed) / p.stage_bytes;
        return fit < most ? fit : most;
    };
    auto fits_half = [&](int fixed) { return halves && depth(fixed, true) >= 3; };
    // Chunk sums without bank conflicts take 128 bytes and more; a stage, or the half SM, is worth more than they are (Q2_K at five
    // rows of 8192: 41.5 us with seven stages, 41.7 with six).
    const int close = fixed_bytes(0), apart = fixed_bytes(1);
    if (pair && (whole_sm || !fits_half(close)) && stages_halve<WT>(p)) {
        p.groups = 2;
        halves = false;
        most = kMaxStages;
    }
    p.spread_sums = fits_half(apart) == fits_half(close) && depth(apart, fits_half(apart)) == depth(close, fits_half(close));
    const int fixed = p.spread_sums ? apart : close;
    p.n_stages = depth(fixed, fits_half(fixed));
    // (a shape is taken if it would be with limb planes of n_in + 32 bytes and stages of row copies: beyond, the warp-per-row kernel multiplies in f32)
    const int spread = wide ? 0 : align_up(rows * (fine_limbs<WT>(p.n_in) ? 4 : 3) * (p.n_in + 32), 128) - plane_bytes<WT>(p.n_in, rows);
    const int stage = !wide && (p.ragged || F::tma == 3) ? align_up(kTileRows * p.tps * rows_stride, 128) : p.stage_bytes;
    if (p.n_stages < 2 || kSmemWhole - close - p.tps * spread < 2 * stage) return false;
    p.by_stage = stages_in_turn<WT>(p, false);
    *smem_out = (size_t)fixed + (size_t)p.n_stages * p.stage_bytes;
    return true;
}

template <int WT>
int launch_rows(const StreamParams &p, int grid, size_t smem, cudaStream_t st) {
    constexpr bool kQ4K = WT == KRK_CUDA_Q4_K;
    if constexpr (kRagForm<WT>) {
        if (p.ragged) {
            if (p.tps > 1) {
                if (p.rows <= 2) return launch_one<WT, 1, true, 0, true>(p, grid, smem, st);
                if (p.rows <= 4) return launch_one<WT, 2, true, 0, true>(p, grid, smem, st);
                return launch_one<WT, 4, true, 0, true>(p, grid, smem, st);
            }
            if (p.rows <= 2 && p.groups == 2) return launch_one<WT, 1, false, 0, true, 2>(p, grid, smem, st);
            if (p.rows <= 2) return launch_one<WT, 1, false, 0, true>(p, grid, smem, st);
            if (p.rows <= 4) return launch_one<WT, 2, false, 0, true>(p, grid, smem, st);
            return launch_one<WT, 4, false, 0, true>(p, grid, smem, st);
        }
    }
    if constexpr (WT == KRK_CUDA_Q4_0) {
        if (p.rows <= 2 && p.groups == 2)
            return p.rows == 1 ? launch_one<WT, 1, false, 1, false, 2>(p, grid, smem, st) : launch_one<WT, 1, false, 0, false, 2>(p, grid, smem, st);
        if (p.rows == 1) return p.tps > 1 ? launch_one<WT, 1, true, 1>(p, grid, smem, st) : launch_one<WT, 1, false, 1>(p, grid, smem, st);
        if (p.rows <= 2) return p.tps > 1 ? launch_one<WT, 1, true, 0>(p, grid, smem, st) : launch_one<WT, 1, false, 0>(p, grid, smem, st);
        if (p.rows <= 4) return p.tps > 1 ? launch_one<WT, 2, true, 0>(p, grid, smem, st) : launch_one<WT, 2, false, 0>(p, grid, smem, st);
        return p.tps > 1 ? launch_one<WT, 4, true, 0>(p, grid, smem, st) : launch_one<WT, 4, false, 0>(p, grid, smem, st);
    } else {
        if (p.tps > 1) {
            if (kQ4K && p.rows == 1) return launch_one<WT, 1, true, kQ4K ? 2 : 0>(p, grid, smem, st);
            if (p.rows <= 2) return launch_one<WT, 1, true, 0>(p, grid, smem, st);
            if (p.rows <= 4) return launch_one<WT, 2, true, 0>(p, grid, smem, st);
            return launch_one<WT, 4, true, 0>(p, grid, smem, st);
        }
        if (p.rows <= 2 && p.groups == 2)
            return kQ4K && p.rows == 1 ? launch_one<WT, 1, false, kQ4K ? 1 : 0, false, 2>(p, grid, smem, st) : launch_one<WT, 1, false, 0, false, 2>(p, grid, smem, st);
        if (kQ4K && p.rows == 1 && !p.whole_tiles && p.units <= 2 * kConsumerWarps) return launch_one<WT, 1, false, kQ4K ? 2 : 0>(p, grid, smem, st);
        if (kQ4K && p.rows == 1) return launch_one<WT, 1, false, kQ4K ? 1 : 0>(p, grid, smem, st);
        if (p.rows <= 2) return launch_one<WT, 1, false, 0>(p, grid, smem, st);
        if constexpr (WT == KRK_CUDA_Q8_0)
            if (p.rows <= 4 && p.groups == 1) return launch_one<WT, 2, false, 0, false, 1>(p, grid, smem, st);
        if (p.rows <= 4) return launch_one<WT, 2, false, 0>(p, grid, smem, st);
        return launch_one<WT, 4, false, 0>(p, grid, smem, st);
    }
}

// Up to four rows of a super-block format with four limbs. 0: no such form.
template <int WT>
int launch_rows_wide(const StreamParams &p, int grid, size_t smem, cudaStream_t st) {
    if (p.tps > 1 || p.rows > 4) return 0;
    if constexpr (kRagForm<WT>) {
        if (p.ragged) {
            const int rc = launch_one<WT, 2, false, 0, true, 2, true>(p, grid, smem, st);
            return rc == KRK_CUDA_OK ? 1 : rc;
        }
    }
    const int rc = launch_one<WT, 2, false, 0, false, 2, true>(p, grid, smem, st);
    return rc == KRK_CUDA_OK ? 1 : rc;
}

// CTAs of one launch per SM. 2 (default): both halves of an SM work on this launch (16 consumer warps per SM:
// 0.80-0.83 of the copy bandwidth on large Q4_K / Q8_0 matrices against 0.5-0.7 with one). 1
// (KRK_CUDA_GEMV_CTAS_PER_SM=1): the other half is left to the next launch in the stream, which becomes
// resident early, sets itself up and fills its ring while this one streams; measured on the layer-sized
// matrices of a decode step the slower streaming of eight warps costs more than the overlap saves.
// The forms of two consumer groups get one whatever their shared memory.
template <int WT>
int ctas_per_sm(size_t smem, int groups) {
    static const int want = [] {
        const char *e = std::getenv("KRK_CUDA_GEMV_CTAS_PER_SM");
        const int v = e ? std::atoi(e) : 0;
        return v == 1 ? 1 : 2;
    }();
    return groups == 1 && smem <= (size_t)kSmemLimit ? want : 1;
}

// Tensor maps are encoded on the host (a driver call of a microsecond or two) and kept per (matrix, box):
// weights stay where they were uploaded, so a decode loop encodes each matrix once.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
struct MapKey {
    const void *w;
    int64_t n_out;
    int row_bytes, unit_bytes, box_rows, box_units, ragged;
    bool operator==(const MapKey &o) const {
        return w == o.w && n_out == o.n_out && row_bytes == o.row_bytes && unit_bytes == o.unit_bytes &&
               box_rows == o.box_rows && box_units == o.box_units && ragged == o.ragged;
    }
};
struct MapKeyHash {
    size_t operator()(const MapKey &k) const {
        size_t h = reinterpret_cast<size_t>(k.w) * 0x9E3779B97F4A7C15ull;
        h ^= (size_t)k.n_out * 0xC2B2AE3D27D4EB4Full + (size_t)k.row_bytes * 31 + (size_t)k.box_rows * 7 + (size_t)k.box_units + (size_t)k.ragged * 131;
        return h;
    }
};
inline CUtensorMapL2promotion l2_promotion() {
    static const int v = [] {
        const char *e = std::getenv("KRK_CUDA_GEMV_L2PROMO");
        return e ? std::atoi(e) : 3;
    }();
    return v == 0 ? CU_TENSOR_MAP_L2_PROMOTION_NONE : v == 1 ? CU_TENSOR_MAP_L2_PROMOTION_L2_64B
           : v == 2 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B : CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
}
// The tensor maps of a matrix, one, or one per phase of its rows (`ragged`, see TilePlace): mode 1: {unit bytes, rows, units of a row} in
// bytes; mode 2: {box_units units as 64-bit elements, rows, groups of box_units units of a row}; mode 3: {the row as 64-bit elements, rows,
// 1}; ragged: {that from the 16-byte boundary below the phase's first row on, its rows, 1}.
inline bool weight_maps(CUtensorMap *out, const uint8_t *w, int64_t n_out, int row_bytes, int unit_bytes, int box_rows, int box_units,
                int mode, int ragged) {
    static EncodeTiledFn encode = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    if (!encode) return false;
    const int n = ragged ? ragged : 1;
    static std::mutex mu;
    static std::unordered_map<MapKey, std::vector<CUtensorMap>, MapKeyHash> cache;
    const MapKey key{w, n_out, row_bytes, unit_bytes, box_rows, mode == 1 ? box_units : -box_units, ragged};
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
        for (int c = 0; c < n; c++) out[c] = it->second[c];
        return true;
    }
    for (int c = 0; c < n; c++) {
        const int64_t first = c < n_out ? c : 0;   // (a phase without rows: its empty tiles are copied all the same, from these)
        const int lead = ragged ? (int)((size_t)first * row_bytes & 15) : 0;
        const int inner_bytes = ragged ? align_up(lead + row_bytes, 8) : mode == 3 ? row_bytes : mode == 2 ? box_units * unit_bytes : unit_bytes;
        const int box_inner = mode == 3 ? box_pitch(box_units * unit_bytes + (ragged ? 14 : 0)) : inner_bytes, size = mode == 1 ? 1 : 8;
        if (mode != 1 && (box_inner / 8 > 256 || (!ragged && (inner_bytes % 16 != 0 || row_bytes % inner_bytes != 0)))) return false;
        const cuuint64_t dims[3] = {(cuuint64_t)(inner_bytes / size), (cuuint64_t)(ragged ? (n_out - first + ragged - 1) / ragged : n_out),
                                    (cuuint64_t)(ragged ? 1 : row_bytes / inner_bytes)};
        const cuuint64_t strides[2] = {(cuuint64_t)row_bytes * n, (cuuint64_t)(ragged ? (size_t)row_bytes * n : (size_t)inner_bytes)};
        const cuuint32_t box[3] = {(cuuint32_t)(box_inner / size), (cuuint32_t)box_rows, (cuuint32_t)(mode == 1 ? box_units : 1)};
        const cuuint32_t elem[3] = {1, 1, 1};
        const uint8_t *base = w + (size_t)first * row_bytes - lead;
        if (encode(&out[c], mode != 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT64 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t *>(base), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, l2_promotion(),
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    // bounded, at 8 MB of maps: a host that keeps re-uploading weights starts over
    static size_t held = 0;
    if (held + n > 65536) {
        cache.clear();
        held = 0;
    }
    cache.emplace(key, std::vector<CUtensorMap>(out, out + n));
    held += n;
    return true;
}

// Fills p.wmap for the first n matrices of p.mat; on failure the launch falls back to row copies.
template <int WT>
bool encode_maps(StreamParams &p, int n) {
    using F = Fmt<WT>;
    const int ku_max = p.units < kConsumerWarps ? p.units : kConsumerWarps, each = p.ragged ? p.ragged : 1;
    if (n * each > kMaxMaps) return false;
    for (int m = 0; m < n; m++) {
        if (p.mat[m].n_out <= 0) continue;
        if ((reinterpret_cast<uintptr_t>(p.mat[m].w) & 15) != 0) return false;
        if (!weight_maps(&p.wmap[m * each], p.mat[m].w, p.mat[m].n_out, p.row_bytes, F::unit_bytes, kTileRows * p.tps, ku_max, p.use_tma, p.ragged)) return false;
    }
    return true;
}

// Granules of a matrix. (Ragged rows: every phase has as many, some of the last phases' maybe without a row.)
inline int64_t granules(const StreamParams &p, int64_t n_out) {
    if (p.ragged) return p.ragged * (((n_out + p.ragged - 1) / p.ragged + p.gran - 1) / p.gran);
    return (n_out + p.gran - 1) / p.gran;
}

// Launches of a format whose stages could be one box each (use_tma == 3) that copy row by row all the same. Row copies let any number
// of rows go to a CTA, a box brings whole tiles.
// One and two activation rows, up to two tiles an SM. Fewer tiles than half of the SMs: all SMs at work on parts of tiles beat a
// tile each on some (box against rows, us: Q2_K 1024 x 4096 4.7 against 4.2, Q8_0 1024 x 8192 7.5 against 6.8). Of one stage in Q2_K and
// Q3_K (2048 values) up to a tile an SM (1280 to 2304 x 2048 1.02 to 1.03). Two activation rows: boxes fill the ring sooner,
// which the loads of x then wait behind, and only just over a tile an SM is that worth it (Q8_0 4096 x 4096 7.4 against 6.7, 4700 x 4096
// 8.2 against 7.0, 2048 x 4096 4.8 against 4.7; 3200 x 4096 5.9 against 6.1).
// Further on, CTAs that all have as many tiles gain nothing by whole ones. Two rows of Q8_0 in one stage or two (8192 and 14000 x 1024
// 1.03 and 1.10, x 2048 1.07 and 1.04; 5632 x 1024 0.95, 65536 x 1024 0.94, 22016 x 2048 0.94, and 0.80 to 1.00 at 2304 values), one row of it in four
// (4200 to 4736 x 4096 1.02 to 1.07; x 3072 and x 5120 0.96 to 1.01).
// Q5_1's rows of 1536 bytes stream as well by themselves: up to two tiles an SM (4700 x 5632 10.6 against 9.8, 4096 x 1024 at two
// rows 5.3 against 4.9; beyond, 6000 x 5632, 12.1 against 12.7) and where CTAs have as many tiles (14208 x 2048 at one and two rows 1.05
// and 1.09, x 1024 0.91 and 0.95, 32768 x 5632 0.98; two rows of 8192 x 2048 and x 4096 1.03 and 1.05, one of x 2048 0.98; 4736 x 4096 at three to five rows 1.04 to 1.07, 6144 x 4096 0.95 to 0.99, 14000 x
// 5120 at eight 0.97).
template <int WT>
bool rows_apart(const StreamParams &p, int64_t tiles, size_t smem) {
    const int sms = sm_count();
    const bool few = p.rows <= 2;
    const int64_t ctas = few && smem <= (size_t)kSmemLimit ? 2 * sms : sms, last = tiles % ctas;
    auto even = [&](int tenths) { return tiles >= ctas && (last == 0 || 10 * last >= tenths * ctas); };
    if (WT == KRK_CUDA_Q5_1) {
        if (few) return tiles <= 2 * sms || (even(p.rows == 2 || p.n_in >= 4096 ? 7 : 9) && p.n_in >= 1280 && p.n_in <= 5632 && tiles <= (p.n_in <= 3072 ? 7 : 3) * ctas);
        return p.rows <= 5 && even(9) && p.n_in >= 2048 && p.n_in <= 5632;
    }
    if (!few || p.units < kConsumerWarps) return false;
    if (tiles <= sms / 2 || ((WT == KRK_CUDA_Q2_K || WT == KRK_CUDA_Q3_K) && p.units == kConsumerWarps && tiles <= sms)) return true;
    if (tiles <= 2 * sms)
        return p.rows == 2 ? p.units > kConsumerWarps && smem <= (size_t)kSmemLimit && (tiles <= sms || tiles > 3 * sms / 2)
                           : WT == KRK_CUDA_Q8_0 && p.units == 4 * kConsumerWarps && tiles > 7 * sms / 4;
    if (WT != KRK_CUDA_Q8_0 || p.rows != 2 || tiles > 7 * ctas) return false;
    return p.units == kConsumerWarps ? even(7) || tiles > 3 * ctas : p.units == 2 * kConsumerWarps && even(7) && tiles < 3 * ctas;
}

// setup_format with the tensor-copy layout where the format and the matrices allow it (the maps are encoded here),
// else with per-row copies. False when the streaming kernel does not address the shape. `whole_rows`: the rows of the matrix that
// the one here is a slice of, which then decide in place of its own: the forms add up in orders of their own.
template <int WT>
bool setup_launch(StreamParams &p, const GemvMat *mats, int n_mat, int64_t n_in, int rows, int silu_pair, size_t *smem, bool wide = false,
                  int64_t whole_rows = 0) {
    static const bool no_tma = std::getenv("KRK_CUDA_GEMV_NO_TMA") != nullptr;
    int64_t tiles = 0;
    for (int m = 0; m < n_mat; m += silu_pair ? 2 : 1) tiles += ((whole_rows ? whole_rows : mats[m].n_out) + kTileRows - 1) / kTileRows;
    // A tile for an SM at most, of many stages: two groups, see stages_halve.
    const bool whole_sm = rows <= 2 && n_in > 5120 && tiles <= (n_in >= 8192 ? sm_count() : sm_count() * 7 / 8);
    bool tma = Fmt<WT>::tma != 0 && !no_tma;
    if (tma) {
        if (!setup_format<WT>(p, n_in, rows, silu_pair, smem, true, false, whole_sm, wide)) return false;
        if (p.use_tma == 3 && !p.ragged && (rows > 2 || p.groups == 1) && rows_apart<WT>(p, tiles, *smem)) tma = false;
        if (tma && p.use_tma) {
            for (int m = 0; m < n_mat; m++) p.mat[m] = mats[m];
            if (!encode_maps<WT>(p, n_mat)) tma = false;   // a map cannot be encoded: set up again for row copies
        }
    }
    if (WT == KRK_CUDA_Q8_0 && !wide) {
        // Many tiles at three rows, or at three and four of one stage each (1024 values and fewer): one group and two CTAs per SM (three rows of
        // 22016 x 4096 22.2 us against 22.9 with two groups, 8192 x 768 5.6 against 6.0; four of 32768 x 1024 12.6 against 14.4). Else two groups:
        // 6144 x 4096 10.6 against 9.8, at four rows 11.6 against 10.0, 11008 x 4096 15.3 against 14.0, 22016 x 4096 23.4 against 23.0 (since a
        // stage is one copy they no longer wait for the ring, of which a tile is four stages there). Tiles of one stage come faster as
        // row copies from five to fourteen an SM (14000 x 1024 at three rows 7.9 against 7.3, 32768 x 1024 at four 13.2 against 12.3; 8192 x 1024 5.9
        // against 6.1, 49152 x 768 14.5 against 15.5, 128256 x 1024 33.2 against 36.8).
        const int64_t least = rows == 3 ? (n_in <= 1024 ? 3 : 6) : n_in < 1024 ? 3 : 5;
        if (n_in % 256 == 0 && (rows == 3 || (rows == 4 && n_in <= 1024)) && tiles > least * sm_count()) {
            if (setup_format<WT>(p, n_in, rows, silu_pair, smem, tma && (n_in > 1024 || tiles <= 5 * sm_count() || tiles > 14 * sm_count()), true) && p.tps == 1 && p.n_stages >= 3 && *smem <= (size_t)kSmemLimit) return true;
            if (tma && !setup_format<WT>(p, n_in, rows, silu_pair, smem, true)) return false;
        }
    }
    return tma || setup_format<WT>(p, n_in, rows, silu_pair, smem, false, false, whole_sm, wide);
}

template <int WT>
int launch_fmt(const GemvMat *mats, int n_mat, int64_t n_in, int rows, int accumulate, int silu_pair, bool wide, cudaStream_t st) {
    StreamParams p;
    size_t smem = 0;
    if (!setup_launch<WT>(p, mats, n_mat, n_in, rows, silu_pair, &smem, wide)) return 0;
    p.accumulate = accumulate;
    p.n_entries = 0;
    int total = 0, tiles = 0;
    for (int m = 0; m < n_mat; m += p.step) {
        if (mats[m].n_out > (1 << 30)) return 0;
        for (int j = 0; j < p.step; j++) p.mat[p.n_entries * p.step + j] = mats[m + j];
        p.gran_begin[p.n_entries] = total;
        total += (int)granules(p, mats[m].n_out);
        tiles += p.ragged ? (int)granules(p, mats[m].n_out) : (int)((mats[m].n_out + kTileRows * p.tps - 1) / (kTileRows * p.tps));
        p.n_entries++;
    }
    p.gran_begin[p.n_entries] = total;
    if (total == 0) return 1;
    p.status = device_status_word();
    if (!p.status) return KRK_CUDA_EDEVICE;
    // A launch whose tiles fit one to an SM takes one CTA per SM: a second would only cut tiles in two (both halves still
    // cost a whole tile of MMAs), and the other half of the SM lets the next launch start early (Q8_0 2048x2048 3.92 ->
    // 3.42 us, Q6_K 2048x6656 10.5 -> 8.1 us).
    const int per_sm = tiles <= sm_count() ? 1 : ctas_per_sm<WT>(smem, p.groups);
    if (tiles <= sm_count()) p.by_stage = stages_in_turn<WT>(p, true);
    const int sms = sm_count() * per_sm;
    // Tiles for fewer SMs than there are. The CTAs of the next launch, which find room beside these, go to the idle SMs two at a time and
    // take twice as long there: a chain of launches of one shape is quicker if the rows are dealt to all SMs, up to 16 each (a
    // box brings some that belong to the next CTA; 1280 to 2304 x 4096 0.7 to 0.9 of the time). In a model's pass the CTAs of several launches
    // to come find room beside fewer, and whole tiles are quicker: rows dealt cost the formats with tensor copies of packed units 1 to 10 %
    // there (one row, 1792 / 4864 values, Q5_0 1.11 of the time, Q4_0 1.06, Q5_K 1.05; two rows, 1024 / 3584, Q4_K 1.08, Q5_K 1.07), so
    // their tiles stay whole, but at two rows, of one stage, for over seven tenths of the SMs (q, k and v of one size one after the other,
    // 1792 and 2048 values 0.95 to 0.97 of the time, where k and v are smaller 0.99 to 1.02). Where a box takes the place of row copies, which went to all SMs by themselves, rows are dealt above half of the
    // SMs (Q8_0 2304 x 5120 5.3 us, whole tiles 6.5, row copies 6.0; a pass, 2048 / 4096, 0.92, 0.88 and 1), ragged ones above nine
    // twentieths (one row, tiles on 48, 64, 80 and 104 SMs and on all: Q3_K x 5120 5.0, 5.7, 6.3, 6.7 and 5.1 us, row copies 6.0; a pass,
    // 1024 / 2816, 64 tiles on as many 1.03 and on all 1.12 of the time that row copies took, Q2_K 1.06 and 1.11). Not the forms that
    // take a whole SM: there the idle SMs let the next launch start (four rows of 2048 x 5632 7.4 and 7.7; ragged ones 1.02 to 1.17 of the time).
    if (p.groups == 1 && smem <= (size_t)kSmemLimit && p.tps == 1 && p.n_entries == 1 && tiles <= sm_count()) {
        if (p.ragged) {
            if (total > sm_count() * 9 / 20) p.gran_begin[1] = total = sm_count();
        } else if ((p.use_tma == 3 && tiles > sm_count() / 2) || (p.use_tma && rows == 2 && p.units <= kConsumerWarps && tiles > sm_count() * 7 / 10)) {
            p.gran = 1;
            p.gran_begin[1] = total = (int)mats[0].n_out;
        }
    }
    const int grid = total < sms ? total : sms;
    p.gran_q = total / grid;
    p.gran_r = total % grid;
    if constexpr (block_size(WT) == 256)
        if (wide) return launch_rows_wide<WT>(p, grid, smem, st);
    const int rc = launch_rows<WT>(p, grid, smem, st);
    return rc == KRK_CUDA_OK ? 1 : rc;
}

template <int WT>
int launch_table_fmt(const StreamTable *table, const int32_t *x_rows, int64_t n_out, int64_t n_in, int rows, int silu_pair, const StreamBanks *banks, cudaStream_t st) {
    StreamParams p;
    size_t smem = 0;
    // With the banks known, a stage arrives as one tensor copy out of the bank's map.
    static const bool no_tma = std::getenv("KRK_CUDA_GEMV_NO_TMA") != nullptr;
    bool tma = false;
    if (banks && (Fmt<WT>::tma == 1 || Fmt<WT>::tma == 3) && !no_tma && setup_format<WT>(p, n_in, rows, silu_pair, &smem, true) &&
        (p.use_tma == 1 || p.use_tma == 3) && !p.ragged) {
        tma = true;
        const int ku_max = p.units < kConsumerWarps ? p.units : kConsumerWarps;
        for (int b = 0; b < p.step && tma; b++) {
            p.bank_base[b] = banks->base[b];
            tma = banks->base[b] && (reinterpret_cast<uintptr_t>(banks->base[b]) & 15) == 0 && banks->rows > 0 &&
                  weight_maps(&p.wmap[b], banks->base[b], banks->rows, p.row_bytes, Fmt<WT>::unit_bytes, kTileRows * p.tps, ku_max, p.use_tma, 0);
        }
    }
    if (!tma && !setup_format<WT>(p, n_in, rows, silu_pair, &smem)) return 0;
    p.n_entries = 0;
    p.gran_q = p.gran_r = 0;
    p.dev_table = table;
    p.table_rows = x_rows;
    p.entry_gran = (int)granules(p, n_out);
    p.status = device_status_word();
    if (!p.status) return KRK_CUDA_EDEVICE;
    const int rc = launch_rows<WT>(p, sm_count() * ctas_per_sm<WT>(smem, p.groups), smem, st);
    return rc == KRK_CUDA_OK ? 1 : rc;
}

template <int WT>
int launch_peers_fmt(const GemvMat &mat, int64_t n_in, int rows, const PeerScatter &ps, cudaStream_t st) {
    StreamParams p;
    size_t smem = 0;
    if (mat.n_out > (1 << 30) || mat.n_out <= 0) return 0;
    if (!setup_launch<WT>(p, &mat, 1, n_in, rows, 0, &smem, false, ps.row_stride)) return 0;
    // (as launch_fmt has it for the whole row)
    if ((p.ragged ? granules(p, ps.row_stride) : (ps.row_stride + kTileRows * p.tps - 1) / (kTileRows * p.tps)) <= sm_count()) p.by_stage = stages_in_turn<WT>(p, true);
    p.mat[0] = mat;
    p.n_entries = 1;
    p.gran_begin[0] = 0;
    const int total = (int)granules(p, mat.n_out);
    p.gran_begin[1] = total;
    p.status = device_status_word();
    if (!p.status) return KRK_CUDA_EDEVICE;
    p.n_peers = ps.n_peers;
    for (int q = 0; q < ps.n_peers; q++) {
        p.peer_y[q] = ps.y[q];
        p.peer_flag[q] = ps.flag[q];
    }
    p.my_rank = ps.my_rank;
    p.epoch = ps.epoch;
    p.wait_peers = ps.wait_peers;
    p.peer_row_stride = ps.row_stride;
    p.peer_offset = ps.offset;
    const int sms = sm_count() * ctas_per_sm<WT>(smem, p.groups);
    const int grid = total < sms ? total : sms;
    p.gran_q = total / grid;
    p.gran_r = total % grid;
    const int rc = launch_rows<WT>(p, grid, smem, st);
    return rc == KRK_CUDA_OK ? 1 : rc;
}

// setup_format's answer alone
template <int WT>
bool takes_fmt(int64_t n_in, int rows) {
    StreamParams p;
    size_t smem = 0;
    return setup_format<WT>(p, n_in, rows, 0, &smem);
}

#define KRK_STREAM_FORMAT(LINKAGE, WT)                                                                                                  \
    LINKAGE template int launch_fmt<WT>(const GemvMat *, int, int64_t, int, int, int, bool, cudaStream_t);                                    \
    LINKAGE template int launch_table_fmt<WT>(const StreamTable *, const int32_t *, int64_t, int64_t, int, int, const StreamBanks *, cudaStream_t); \
    LINKAGE template int launch_peers_fmt<WT>(const GemvMat &, int64_t, int, const PeerScatter &, cudaStream_t);                        \
    LINKAGE template bool takes_fmt<WT>(int64_t, int);

} // namespace stream
} // namespace krk_cuda
