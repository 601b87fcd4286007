// Prefill GEMM for sm_100a: Y[rows][n_out] = X[rows][n_in] . W^T with W block-quantized in HBM,
// decoded to f16 and contracted on the 5th-generation tensor cores (tcgen05.mma, f32 accumulators
// in tensor memory).
//
// Mapping. The weight tile is the MMA's A operand (128 weight rows = the 128 TMEM lanes), the
// token tile its B operand (up to 256 tokens = TMEM columns), so a weight tile is decoded once
// per 256 tokens and the accumulator D[weight row][token] is Y transposed: the epilogue reads one
// TMEM lane per thread and 32 neighbouring weight rows of one token form one coalesced 128-byte
// store.
//
// The decoded weights never touch shared memory: a decode thread owns a weight row = a TMEM lane,
// so it writes its f16 values straight into tensor memory (tcgen05.st) and the MMA takes A from
// TMEM. Shared memory then carries only the X tiles (TMA, 128-byte swizzle) and the raw quantized
// bytes, which leaves its bandwidth to the one operand the MMA still reads from it.
//
// One persistent CTA per SM, warp-specialised, everything connected by mbarriers:
//   warps 0..15  decode, two groups of eight that fill alternate A stages: two threads per weight row, 32 values
//                each per 64-value K step. The raw blocks of
//                128 rows x 256 values (Q8_0: 128 values) arrive in shared memory by TMA: a 2-D tensor map
//                over the raw byte matrix where a row's 256-value segments start on 16-byte boundaries, eight
//                maps (rows 8 apart) for Q6_K, Q3_K and Q2_K, whose rows do not; a thread takes its row's bytes
//                into registers and decodes them four values at a time. 16 x 32-bit TMEM columns per thread and step;
//   warps 16..19 epilogue: tcgen05.ld of the accumulator (warp w%4 owns TMEM lanes 32*(w%4)..), 32 tokens
//                at a time into a [token][weight row] staging buffer in shared memory, TMA stores of Y;
//   warp 20      TMA producer of X tiles (cp.async.bulk.tensor.2d, each CTA loads its own copy);
//   warp 21      TMA producer of the raw block columns;
//   warps 22, 23 TMEM allocation and issue of tcgen05.mma / tcgen05.commit.
// Tensor memory: columns 0..255 the accumulator (two of 128 columns when a tile has at most 128 tokens, so that
// one is read out while the next tile is multiplied), 256..511 four A stages of 64 columns (two K steps each).
//
// Ring depths are chosen per launch from the tile: what bounds a narrow tile is the latency of the copies, not
// HBM (a four-deep X ring and three raw stages cost 330 ns per K step at every M <= 128 and in every format,
// against 104 ns of HBM time for Q4_K), so the shared memory that a small X tile leaves goes into more stages.
//
// Tiles come in whole waves, and the CTAs of a cluster share each of the tiles left over (all of them, for a short prompt
// or a narrow matrix), a piece of K each; the accumulators meet over distributed shared memory and are added in K
// order, the same on every run.
//
// Same contract as gemm_wmma_kernel of the reference (src/hip/kernels/gemm.hpp:621-970): f16
// staged operands, f32 accumulation; here the output stays f32.
//
// Every mbarrier wait is bounded; a wait that gives up raises the device status word, and the CTA
// runs to its end without waiting again and frees its tensor memory.
#include <cuda.h>

#include <cstddef>
#include <mutex>

#include "krk_common.cuh"
#include "krk_gemm_plan.h"

namespace krk_cuda {

namespace {

constexpr int kBK = 64;                // K values per step: one 128-byte swizzle row of f16 X, 32 TMEM columns of A
constexpr int kMaxB = 16, kMinB = 4;   // X tiles in shared memory
constexpr int kAStages = 4;            // decoded weight tiles in tensor memory, two K steps (64 columns) each
constexpr int kMaxRaw = 8, kMinRaw = 2;   // raw block columns (256 values x 128 rows) in shared memory
// Formats whose 256-value row segment is a multiple of 16 bytes arrive as one box per stage: Q4_K (144), Q4_0 and
// IQ4_NL (8 x 18 = 144), Q5_K (176), Q5_0 (8 x 22 = 176), Q5_1 (8 x 24 = 192). Q8_0 arrives 128 values at a time:
// four 34-byte blocks = 136 bytes, which start 0 or 8 bytes after a 16-byte boundary, so a 144-byte box that starts
// on the boundary covers them.

// The 210-, 110- and 84-byte blocks of Q6_K, Q3_K and Q2_K start on even addresses only, but eight rows on, the
// address is the same modulo 16 (row lengths are even): the rows r = c (mod 8) of the matrix, seen from the 16-byte
// boundary at or before row c, are a tensor with a 16-byte-multiple pitch. One map per c; a stage is eight boxes of
// 16 rows (the 16-byte granules that hold a block), and the 128 staged rows are in the order (c, k) <-> row c + 8k.
// Slot pitches: 224 holds a Q6_K block at any lead; 144 (Q3_K) and 112 (Q2_K) keep the eight rows of a 16-byte load
// phase on different banks.
__host__ __device__ constexpr bool row_phased(int wt) { return wt == KRK_CUDA_Q6_K || wt == KRK_CUDA_Q3_K || wt == KRK_CUDA_Q2_K; }
constexpr int kPhases = 8;
__host__ __device__ constexpr int raw_seg(int wt) {
    return (wt == KRK_CUDA_Q5_K || wt == KRK_CUDA_Q5_0) ? 176 : wt == KRK_CUDA_Q5_1 ? 192 : wt == KRK_CUDA_Q6_K ? 224
           : wt == KRK_CUDA_Q2_K ? 112 : 144;
}

// What a launch computes. kDense: Y = X . W^T. The other two serve the routed experts, whose tiles come from a
// device-side list of (expert, token group) entries: kGateUp takes 64 gate rows and the 64 up rows of the same
// outputs as one weight tile and leaves f16 silu(gate) * up, kDown leaves f32 rows.
enum GemmKind { kDense = 0, kGateUp = 1, kDown = 2 };

// Which staged row and which weight row the decode thread of TMEM lane t works on. A weight tile is one run of 128
// rows, or (kGateUp) 64 of each matrix. Phased formats: a warp's 32 lanes take 32 neighbouring rows (so the read-out
// writes 32 different banks) in an order whose neighbouring lanes read staged rows on different banks.
template <int WT, int KIND>
__host__ __device__ constexpr int tile_row(int t) {   // row inside the tile; kGateUp: inside the matrix's half, up rows + 64
    if (!row_phased(WT)) return t;
    const int w = t >> 5, half = KIND == kGateUp ? w >> 1 : 0, wh = KIND == kGateUp ? w & 1 : w;
    return 64 * half + ((t & 31) >> 2) + 8 * (4 * wh + (t & 3));
}
template <int WT, int KIND>
__host__ __device__ constexpr int tile_slot(int t) {
    if (!row_phased(WT)) return t;
    const int w = t >> 5, half = KIND == kGateUp ? w >> 1 : 0, wh = KIND == kGateUp ? w & 1 : w;
    return 64 * half + (KIND == kGateUp ? 8 : 16) * ((t & 31) >> 2) + 4 * wh + (t & 3);
}
template <int KIND>
struct WMaps {
    CUtensorMap m[KIND == kGateUp ? 2 * kPhases : kPhases];   // m[0] (kGateUp: m[0] gate, m[1] up) alone for the formats staged as one box
};
constexpr int kDecodeGroups = 2, kGroupThreads = 256;   // two decode threads per weight row in each group
constexpr int kDecodeThreads = kDecodeGroups * kGroupThreads, kEpilogueThreads = 128;
constexpr int kDecodeWarps = kDecodeThreads / 32, kEpilogueWarps = kEpilogueThreads / 32;
constexpr int kXWarp = kDecodeWarps + kEpilogueWarps, kRawWarp = kXWarp + 1, kMmaWarp = kXWarp + 2;   // two MMA warps
constexpr int kThreads = 32 * (kMmaWarp + 2);
constexpr int kTmemCols = 512, kTmemA = 256;
constexpr int kGroupBox = 32;          // tokens per X box of the expert kinds
constexpr long long kWaitCycles = 4000000000LL;
constexpr int kSmemMax = 227 * 1024;

struct GemmParams {
    float *y;
    __half *h;           // kGateUp: output [x rows][n_out] f16
    int64_t n_out, n_in, rows;
    int tile_m;          // tokens per tile: multiple of 16, <= 256
    int n_tiles_n, n_tiles_m;
    int group;           // tiles in a row that share a weight tile (dense: n_tiles_m) or a token group (expert kinds: n_tiles_n)
    uint32_t per_group;  // ceil(2^32 / group) where the high half of a product with it divides every tile's number exactly, else 0
    int k_blocks, kb_each, kb_more;   // super-blocks of K; a piece has kb_each of them, the first kb_more pieces one more
    int sum_tokens;      // tokens of a shared tile that one CTA of the cluster adds up
    int row_bytes;
    uint32_t zero;       // always 0, which the compiler does not know (see the decode warps)
    int xk;              // K steps per X stage: 4, 2 or 1
    int dual;            // 1: both MMA warps issue, super-blocks in turn, into an accumulator each
    int n_b, n_raw;      // ring depths (stages)
    int raw_off, y_off, bar_off;   // where the raw ring, the read-out buffers and the barriers start (the X ring starts at 0)
    int split;           // CTAs per cluster (1: no cluster)
    int n_full;          // tiles that one CTA computes alone; the clusters share the rest, at most one each
    int y_tma;           // 1: tiles leave through shared memory and TMA stores (y 16-byte aligned, n_out % 4 == 0)
    int *status;
    const GemmGroup *groups;   // kGateUp, kDown: token groups, and how many
    const int *n_groups;
};

struct GemmBars {
    unsigned long long b_full[kMaxB], b_empty[kMaxB];
    unsigned long long a_full[kAStages], a_empty[kAStages];
    unsigned long long raw_full[kMaxRaw], raw_empty[kMaxRaw];
    unsigned long long d_full[2], d_empty[2];
    uint32_t tmem_base;
    int gave_up;
};

// ---- PTX wrappers -------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes, uint32_t elected) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n"
                 ::"r"(bar), "r"(bytes), "r"(elected) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, volatile int *gave_up, int *status) {
    const long long t0 = clock64();
    for (;;) {
        for (int i = 0; i < 32; i++) {
            if (mbar_try_wait(bar, parity)) return;
            __nanosleep(20);
        }
        if (*gave_up) return;
        if (clock64() - t0 > kWaitCycles) {
            *gave_up = 1;
            atomicExch(status, KRK_CUDA_ETIMEOUT);
            return;
        }
    }
}
__device__ __forceinline__ void wait_phase(uint32_t bar, uint32_t parity, volatile int *gave_up, int *status) {
    if (mbar_try_wait(bar, parity)) return;
    if (*gave_up) return;
    wait_slow(bar, parity, gave_up, status);
}
// Issued by the elected lane of a converged warp (see umma_f16_ts_step: operands in uniform registers).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar, uint32_t elected) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
                 " @q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}\n"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar), "r"(elected) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, int x, int y, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
                 ::"l"(map), "r"(x), "r"(y), "r"(src) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// One K step: four MMAs over 16 K values each, A from tensor memory (lane = row, 32-bit column = two consecutive K
// values, so 8 columns per MMA), B from shared memory (32 bytes of every row per MMA). `first`: the first MMA starts a
// new sum. Executed by a whole converged warp whose operands are all warp-uniform, issued by the lane `elected` picks:
// with the operands in uniform registers a step issues in 80 cycles; from a one-lane branch the operands go through
// per-lane registers first and a step takes 470-510 cycles whatever N is (608 at N = 256 against the pipe's 512).
// `b_lo` is the low half of the descriptor (16 K values are 2 units of its address field; the field cannot carry out of
// it), `hi` the constant other half.
__device__ __forceinline__ void umma_f16_ts_step(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t first, uint32_t elected) {
    asm volatile("{\n .reg .pred p, q, t;\n .reg .b64 b0, b1, b2, b3;\n .reg .b32 a1, a2, a3, l1, l2, l3;\n"
                 " setp.eq.b32 p, %4, 0;\n setp.ne.b32 q, %6, 0;\n setp.eq.b32 t, 0, 0;\n"
                 " add.s32 l1, %2, 2;\n add.s32 l2, %2, 4;\n add.s32 l3, %2, 6;\n"
                 " mov.b64 b0, {%2, %7};\n mov.b64 b1, {l1, %7};\n mov.b64 b2, {l2, %7};\n mov.b64 b3, {l3, %7};\n"
                 " add.s32 a1, %1, 8;\n add.s32 a2, %1, 16;\n add.s32 a3, %1, 24;\n"
                 " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b0, %3, {%5, %5, %5, %5}, p;\n"
                 " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, {%5, %5, %5, %5}, t;\n"
                 " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, {%5, %5, %5, %5}, t;\n"
                 " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, {%5, %5, %5, %5}, t;\n}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(first), "r"(0u), "r"(elected), "r"(hi) : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
    return e;
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
                   "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t elected) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n"
                 ::"r"(bar), "r"(elected) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile of 128-byte rows in the 128-byte swizzle:
// start address >> 4 in bits 0-13, leading byte offset (unused for this layout) 1 in bits 16-29,
// stride byte offset 1024 >> 4 (eight rows) in bits 32-45, descriptor version 1 in bits 46-47,
// layout type 2 (SWIZZLE_128B) in bits 61-63.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t kSmemDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);

// Instruction descriptor, kind::f16: D f32 (bits 4-5 = 1), A and B f16 (0), both K-major (0),
// N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Cluster plumbing of the split-K form: barriers over all threads of the cluster's CTAs, and loads from another CTA's
// shared memory.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
    int v;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    return v;
}
__device__ __forceinline__ int cluster_id() {
    int v;
    asm("mov.u32 %0, %%clusterid.x;" : "=r"(v));
    return v;
}
__device__ __forceinline__ float4 ld_peer(uint32_t addr, int rank) {
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}

// ---- decode of half a weight row's K step (32 values) to f16 ---------------------------------------
// A 256-value block column is four K steps. Decode group `grp` takes K steps 2 grp and 2 grp + 1 of it; a thread
// (half h of its row) first LOADS the raw bytes it needs for both, then CONVERTS one step at a time: out[j] holds
// values 2j, 2j+1 (low, high half) of its 32 (`half` is a template argument: it fixes shift distances). f16 arithmetic runs on exact small integers; the scale products are
// formed in f32 as the host decoder forms them and rounded to f16 once. (A Q8_0 stage is two K steps: each group takes
// one. Groups that took turns over whole stages would meet a ring slot only every other lap where the ring has an odd
// number of slots, and a parity wait cannot tell a lap from the one two before it.)

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<__half2 *>(&u); }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// Byte i of t as an exact float plus 2^23: the byte under the exponent of 2^23.
__device__ __forceinline__ float byte_plus_2_23(uint32_t t, int i) { return __uint_as_float(prmt(t, 0x4B000000u, 0x7650u + i)); }
// Four quant bytes to two half2: (bytes 0, 1) and (bytes 2, 3), each under a 0x64 high byte, i.e. 1024 + q.
__device__ __forceinline__ __half2 halves_lo(uint32_t t) { return bits_h2(__byte_perm(t, 0x64646464u, 0x4140)); }
__device__ __forceinline__ __half2 halves_hi(uint32_t t) { return bits_h2(__byte_perm(t, 0x64646464u, 0x4342)); }
// out[0..1] = (q - bias) * d, or (q - bias) * d + m, of the four quant bytes in t
__device__ __forceinline__ void scale4(uint32_t t, __half2 bias, __half2 d, uint32_t *out) {
    out[0] = h2_bits(__hmul2(__hsub2(halves_lo(t), bias), d));
    out[1] = h2_bits(__hmul2(__hsub2(halves_hi(t), bias), d));
}
__device__ __forceinline__ void scale4(uint32_t t, __half2 bias, __half2 d, __half2 m, uint32_t *out) {
    out[0] = h2_bits(__hfma2(__hsub2(halves_lo(t), bias), d, m));
    out[1] = h2_bits(__hfma2(__hsub2(halves_hi(t), bias), d, m));
}
// Low (HALF 0) or high nibbles in place, and 1024 + q or 1024 + 16 q of them to q - bias by one operation that is exact either way:
// no shift for the high ones (the decode is bound by the pipe that shifts; Q4_K 8192 x 4096 at 32 tokens 11.75 -> 11.45 us, Q4_0
// 11.67 -> 11.34).
template <int HALF>
__device__ __forceinline__ uint32_t nibbles_of(uint32_t t) { return t & (HALF ? 0xF0F0F0F0u : 0x0F0F0F0Fu); }
template <int HALF>
__device__ __forceinline__ __half2 nibble_pair(__half2 h, float bias) {
    return HALF ? __hfma2(h, __float2half2_rn(0.0625f), __float2half2_rn(-64.0f - bias)) : __hsub2(h, __float2half2_rn(1024.0f + bias));
}
__device__ __forceinline__ __half2 half2_of_bits(uint32_t h) { return __half2half2(__ushort_as_half((unsigned short)h)); }
__device__ __forceinline__ float float_of_half_bits(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }
template <int N>
__device__ __forceinline__ void load_quads(const uint8_t *src, uint32_t *w) {   // N 16-byte loads
    const uint4 *b = reinterpret_cast<const uint4 *>(src);
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint4 v = b[i];
        w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
    }
}
// Half of a block column whose halves are 8 bytes past a multiple of 16 long (72 or 88 bytes): `QUADS` 16-byte loads
// and one of 8 bytes, before them in the second half.
template <int QUADS>
__device__ __forceinline__ void load_half_column(const uint8_t *column, int grp, uint32_t (&w)[4 * QUADS + 2]) {
    if (grp == 0) {
        load_quads<QUADS>(column, w);
        const uint2 v = *reinterpret_cast<const uint2 *>(column + 16 * QUADS);
        w[4 * QUADS] = v.x, w[4 * QUADS + 1] = v.y;
    } else {
        const uint2 v = *reinterpret_cast<const uint2 *>(column + 16 * QUADS + 8);
        w[0] = v.x, w[1] = v.y;
        load_quads<QUADS>(column + 16 * QUADS + 16, w + 2);
    }
}

// loaded(): a word that depends on every load of load_block.
template <int WT>
struct Raw;

// The eight words that start `o` bytes (even) into a slot.
__device__ __forceinline__ void window(const uint8_t *slot, int o, uint32_t (&y)[8]) {
    uint32_t x[12];
    load_quads<3>(slot + (o & ~15), x);
    const bool by2 = (o & 8) != 0, by1 = (o & 4) != 0;
#pragma unroll
    for (int i = 0; i < 10; i++) x[i] = by2 ? x[i + 2] : x[i];
#pragma unroll
    for (int i = 0; i < 9; i++) x[i] = by1 ? x[i + 1] : x[i];
    const int sh = 8 * (o & 2);
#pragma unroll
    for (int i = 0; i < 8; i++) y[i] = __funnelshift_r(x[i], x[i + 1], sh);
}

// Q6_K: the staged slot of a row holds its 210-byte block (src/quant.cpp:491-512) `lead` bytes (even, 0..14)
// after the slot's 16-byte-aligned start. Group grp takes 128-value half grp: its thread half h the 32 ql bytes at
// 64 grp + 32 h, the 32 qh bytes at 128 + 32 grp, two scale pairs and d. Step j's chunk is quad 2j + h: the low (j = 0)
// or high nibbles of those ql bytes and bit pair 2j + h of the qh bytes, four quants per operation.
template <>
struct Raw<KRK_CUDA_Q6_K> {
    static constexpr int kSteps = 4;
    uint32_t ql[8], qh[8], sc[2], dbits;
    int lead = 0;
    __device__ __forceinline__ void load_block(const uint8_t *slot, int half, int, int grp) {
        window(slot, lead + 64 * grp + 32 * half, ql);
        window(slot, lead + 128 + 32 * grp, qh);
#pragma unroll
        for (int j = 0; j < 2; j++) sc[j] = *reinterpret_cast<const unsigned short *>(slot + lead + 192 + 8 * grp + 4 * j + 2 * half);
        dbits = *reinterpret_cast<const unsigned short *>(slot + lead + 208);
    }
    // f16(d * scale) is formed in f32 as the host decoder forms d * scale.
    __device__ __forceinline__ uint32_t loaded() const { return ql[0] ^ ql[7] ^ qh[0] ^ qh[7] ^ sc[0] ^ sc[1] ^ dbits; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const float d = float_of_half_bits(dbits);
        const __half2 dl0 = __float2half2_rn(__fmul_rn(d, (float)(int8_t)(sc[j] & 0xFF)));
        const __half2 dl1 = __float2half2_rn(__fmul_rn(d, (float)(int8_t)(sc[j] >> 8)));
        const __half2 bias = __float2half2_rn(1056.0f);   // 1024 + q; the quant is q - 32
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int up = 4 - (4 * j + 2 * half);   // bit pair 2j + half of every qh byte to bits 4 and 5
            const uint32_t hi = (up >= 0 ? qh[i] << up : qh[i] >> -up) & 0x30303030u;
            const uint32_t t = ((ql[i] >> (4 * j)) & 0x0F0F0F0Fu) | hi;
            scale4(t, bias, i < 4 ? dl0 : dl1, out + 2 * i);
        }
    }
};

// The 6-bit scales and mins of chunks 4 grp .. 4 grp + 3 of a Q4_K / Q5_K header, a byte each (src/quant.cpp:427-435).
__device__ __forceinline__ void k_scales(const uint4 &hdr, int grp, uint32_t &sc, uint32_t &mn) {
    if (grp == 0) {
        sc = hdr.y & 0x3F3F3F3Fu;
        mn = hdr.z & 0x3F3F3F3Fu;
    } else {
        sc = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
        mn = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
    }
}

// Q4_K: K step p of the 144-byte block covers chunks 2p, 2p+1: the low and the high nibbles of the
// same 32 bytes (src/quant.cpp:437-460). Thread half h converts chunk 2p+h.
template <>
struct Raw<KRK_CUDA_Q4_K> {
    static constexpr int kSteps = 4;
    uint32_t q[16], sc, mn, dd;
    __device__ __forceinline__ void load_block(const uint8_t *block, int, int, int grp) {
        const uint4 hdr = *reinterpret_cast<const uint4 *>(block);
        load_quads<4>(block + 16 + 64 * grp, q);
        k_scales(hdr, grp, sc, mn);
        dd = hdr.x;
    }
    __device__ __forceinline__ uint32_t loaded() const { return q[0] ^ q[4] ^ q[8] ^ q[12] ^ dd; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const int k = 2 * j + half;
        const float s = byte_plus_2_23(sc, k) - 8388608.0f, m = byte_plus_2_23(mn, k) - 8388608.0f;
        const __half2 dl = __float2half2_rn(__fmul_rn(float_of_half_bits(dd & 0xFFFF), s));
        const __half2 ml = __float2half2_rn(-__fmul_rn(float_of_half_bits(dd >> 16), m));
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t t = nibbles_of<half>(q[8 * j + i]);
            out[2 * i] = h2_bits(__hfma2(nibble_pair<half>(halves_lo(t), 0.0f), dl, ml));
            out[2 * i + 1] = h2_bits(__hfma2(nibble_pair<half>(halves_hi(t), 0.0f), dl, ml));
        }
    }
};

// Q5_K: the 176-byte super-block (src/quant.cpp:462-489) is Q4_K's header and nibbles plus 32 mask bytes whose
// bit c is the fifth quant bit of chunk c.
template <>
struct Raw<KRK_CUDA_Q5_K> {
    static constexpr int kSteps = 4;
    uint32_t q[16], qh[8], sc, mn, dd;
    __device__ __forceinline__ void load_block(const uint8_t *block, int, int, int grp) {
        const uint4 hdr = *reinterpret_cast<const uint4 *>(block);
        load_quads<2>(block + 16, qh);
#pragma unroll
        for (int i = 0; i < 8; i++) qh[i] >>= 4 * grp;
        load_quads<4>(block + 48 + 64 * grp, q);
        k_scales(hdr, grp, sc, mn);
        dd = hdr.x;
    }
    __device__ __forceinline__ uint32_t loaded() const { return q[0] ^ q[4] ^ q[8] ^ q[12] ^ qh[0] ^ qh[4] ^ dd; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const int k = 2 * j + half, up = 4 - k;   // (the masks were moved down by the group's 4 bits when loaded)
        const float s = byte_plus_2_23(sc, k) - 8388608.0f, m = byte_plus_2_23(mn, k) - 8388608.0f;
        const __half2 dl = __float2half2_rn(__fmul_rn(float_of_half_bits(dd & 0xFFFF), s));
        const __half2 ml = __float2half2_rn(-__fmul_rn(float_of_half_bits(dd >> 16), m));
        const __half2 k1024 = __float2half2_rn(1024.0f);
#pragma unroll
        for (int i = 0; i < 8; i++)
            scale4(((q[8 * j + i] >> (4 * half)) & 0x0F0F0F0Fu) | ((qh[i] << up) & 0x10101010u), k1024, dl, ml, out + 2 * i);
    }
};

// Q4_0: eight 18-byte blocks per 256 values = the same 144-byte column as Q4_K. K step p covers blocks 2p
// (thread half 0) and 2p + 1 (half 1): block 2p starts on a word of the column, block 2p + 1 half a word
// later, so its 16 quant bytes are whole words (src/quant.cpp:331-339). (Both candidates with constant indices, then a
// select: `half` in the index would put w[] in local memory.)
template <>
struct Raw<KRK_CUDA_Q4_0> {
    static constexpr int kSteps = 4;
    uint32_t w[18];
    __device__ __forceinline__ void load_block(const uint8_t *block, int, int, int grp) { load_half_column<4>(block, grp, w); }
    __device__ __forceinline__ uint32_t loaded() const { return w[0] ^ w[2] ^ w[4] ^ w[8] ^ w[12] ^ w[14] ^ w[16]; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const __half2 d2 = half2_of_bits(half ? (w[9 * j + 4] >> 16) : (w[9 * j] & 0xFFFFu));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // byte b of the block: value b in its low nibble, value 16 + b in its high one; the quant is the nibble - 8
            const uint32_t q = half ? w[9 * j + 5 + i] : __funnelshift_r(w[9 * j + i], w[9 * j + i + 1], 16);
            const uint32_t lo = nibbles_of<0>(q), hi = nibbles_of<1>(q);
            out[2 * i] = h2_bits(__hmul2(nibble_pair<0>(halves_lo(lo), 8.0f), d2));
            out[2 * i + 1] = h2_bits(__hmul2(nibble_pair<0>(halves_hi(lo), 8.0f), d2));
            out[8 + 2 * i] = h2_bits(__hmul2(nibble_pair<1>(halves_lo(hi), 8.0f), d2));
            out[8 + 2 * i + 1] = h2_bits(__hmul2(nibble_pair<1>(halves_hi(hi), 8.0f), d2));
        }
    }
};

// IQ4_NL: Q4_0's block with indices into a grid of 16 signed bytes (src/quant.cpp:88-91, 566-575). The grid lies in
// four words, biased by 128; a byte permute looks four indices up in half of it at a time and another permute in its
// sign-replicating mode makes the mask that picks between the halves by the index's top bit. d is an f16 and the
// grid value an exact one, so the product is rounded once.
template <>
struct Raw<KRK_CUDA_IQ4_NL> {
    static constexpr int kSteps = 4;
    uint32_t w[18];
    __device__ __forceinline__ void load_block(const uint8_t *block, int, int, int grp) { load_half_column<4>(block, grp, w); }
    __device__ __forceinline__ uint32_t loaded() const { return w[0] ^ w[2] ^ w[4] ^ w[8] ^ w[12] ^ w[14] ^ w[16]; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        constexpr uint32_t kG0 = 0x3F2D1801u, kG1 = 0x766A5D4Fu, kG2 = 0xA6998D81u, kG3 = 0xF1D9C5B5u;   // grid + 128
        const __half2 d2 = half2_of_bits(half ? (w[9 * j + 4] >> 16) : (w[9 * j] & 0xFFFFu));
        const __half2 bias = __float2half2_rn(1152.0f);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t q = half ? w[9 * j + 5 + i] : __funnelshift_r(w[9 * j + i], w[9 * j + i + 1], 16);
            const uint32_t s = q & 0x77777777u, s2 = s >> 16, y = q << 4;
            const uint32_t m01 = prmt(y, q, 0xD9C8u), m23 = prmt(y, q, 0xFBEAu);   // 0xFF where the index is 8..15
            const uint32_t r01 = (prmt(kG0, kG1, s) & ~m01) | (prmt(kG2, kG3, s) & m01);     // [low 0, high 0, low 1, high 1]
            const uint32_t r23 = (prmt(kG0, kG1, s2) & ~m23) | (prmt(kG2, kG3, s2) & m23);
            out[2 * i] = h2_bits(__hmul2(__hsub2(bits_h2(__byte_perm(r01, 0x64646464u, 0x4240)), bias), d2));
            out[2 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(__byte_perm(r23, 0x64646464u, 0x4240)), bias), d2));
            out[8 + 2 * i] = h2_bits(__hmul2(__hsub2(bits_h2(__byte_perm(r01, 0x64646464u, 0x4341)), bias), d2));
            out[8 + 2 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(__byte_perm(r23, 0x64646464u, 0x4341)), bias), d2));
        }
    }
};

// Four bits (a nibble's worth of fifth quant bits) spread to bit 4 of four bytes: bit m of b goes to bit 8m + 4.
__device__ __forceinline__ uint32_t spread_fifth(uint32_t b) { return (((b & 0xFu) * 0x00204081u) & 0x01010101u) << 4; }

// Q5_0: eight 22-byte blocks per 256 values (src/quant.cpp:351-364): f16 d, 32 fifth bits, 16 bytes whose low nibbles
// are quants 0..15 and whose high nibbles are quants 16..31; value = d * (q - 16). K step p covers blocks 2p (thread
// half 0: the block starts on a word of the column) and 2p + 1 (half 1: half a word later, so its bit word and its
// quant bytes are whole words).
template <>
struct Raw<KRK_CUDA_Q5_0> {
    static constexpr int kSteps = 4;
    uint32_t w[22];
    __device__ __forceinline__ void load_block(const uint8_t *block, int, int, int grp) { load_half_column<5>(block, grp, w); }
    __device__ __forceinline__ uint32_t loaded() const { return w[0] ^ w[2] ^ w[4] ^ w[8] ^ w[12] ^ w[16] ^ w[18] ^ w[20]; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const int W = 11 * j;
        const __half2 d2 = half2_of_bits(half ? (w[W + 5] >> 16) : (w[W] & 0xFFFFu));
        const uint32_t qh = half ? w[W + 6] : __funnelshift_r(w[W], w[W + 1], 16);
        const __half2 bias = __float2half2_rn(1040.0f);   // 1024 + q; the quant is q - 16
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t q = half ? w[W + 7 + i] : __funnelshift_r(w[W + 1 + i], w[W + 2 + i], 16);
            scale4((q & 0x0F0F0F0Fu) | spread_fifth(qh >> (4 * i)), bias, d2, out + 2 * i);
            scale4(((q >> 4) & 0x0F0F0F0Fu) | spread_fifth(qh >> (16 + 4 * i)), bias, d2, out + 8 + 2 * i);
        }
    }
};

// Q5_1: eight 24-byte blocks per 256 values (src/quant.cpp:366-379): f16 d, f16 m, 32 fifth bits, 16 quant bytes;
// value = d * q + m, q unsigned. Every field of every block is word aligned.
template <>
struct Raw<KRK_CUDA_Q5_1> {
    static constexpr int kSteps = 4;
    uint32_t w[24];
    __device__ __forceinline__ void load_block(const uint8_t *block, int, int, int grp) { load_quads<6>(block + 96 * grp, w); }
    __device__ __forceinline__ uint32_t loaded() const { return w[0] ^ w[4] ^ w[8] ^ w[12] ^ w[16] ^ w[20]; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        uint32_t b[6];
#pragma unroll
        for (int i = 0; i < 6; i++) b[i] = half ? w[12 * j + 6 + i] : w[12 * j + i];
        const __half2 d2 = half2_of_bits(b[0] & 0xFFFFu), m2 = half2_of_bits(b[0] >> 16);
        const uint32_t qh = b[1];
        const __half2 k1024 = __float2half2_rn(1024.0f);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t q = b[2 + i];
            scale4((q & 0x0F0F0F0Fu) | spread_fifth(qh >> (4 * i)), k1024, d2, m2, out + 2 * i);
            scale4(((q >> 4) & 0x0F0F0F0Fu) | spread_fifth(qh >> (16 + 4 * i)), k1024, d2, m2, out + 8 + 2 * i);
        }
    }
};

// Q8_0: a stage is 128 values = four 34-byte blocks (f16 d, 32 int8; src/quant.cpp:381-387) inside a 144-byte
// box that starts 0 (even stage) or 8 (odd stage) bytes before them. K step p = grp covers blocks 2p (thread half 0)
// and 2p + 1 (half 1); a thread takes only its own block, as nine words: block 2p starts on a word,
// block 2p + 1 half a word later, so its quants are whole words.
template <>
struct Raw<KRK_CUDA_Q8_0> {
    static constexpr int kSteps = 2;
    uint32_t w[9];
    __device__ __forceinline__ void load_block(const uint8_t *box, int half, int ks, int grp) {
        // (four loads of 8 bytes, from multiples of 8, and one of 4: nine of 4 met the same banks four-fold; 8192 x 4096 at 128
        // tokens 16.9 -> 16.5 us)
        const uint8_t *b = box + 8 * ((ks >> 1) & 1) + 32 * half + 68 * grp;
        auto load_pairs = [&](const uint8_t *src, uint32_t *to) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint2 v = reinterpret_cast<const uint2 *>(src)[i];
                to[2 * i] = v.x, to[2 * i + 1] = v.y;
            }
        };
        if (grp == 0) {
            load_pairs(b, w);
            w[8] = *reinterpret_cast<const uint32_t *>(b + 32);
        } else {
            w[0] = *reinterpret_cast<const uint32_t *>(b);
            load_pairs(b + 4, w + 1);
        }
    }
    __device__ __forceinline__ uint32_t loaded() const { return w[0] ^ w[1] ^ w[2] ^ w[3] ^ w[4] ^ w[5] ^ w[6] ^ w[7] ^ w[8]; }
    template <int half>
    __device__ __forceinline__ void convert(int, uint32_t (&out)[16]) const {
        const __half2 d2 = half2_of_bits(half ? (w[0] >> 16) : (w[0] & 0xFFFFu));
        const __half2 bias = __float2half2_rn(1152.0f);   // q ^ 0x80 under a 0x64 high byte is the half 1024 + 128 + q
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t q = half ? w[1 + i] : __funnelshift_r(w[i], w[i + 1], 16);
            scale4(q ^ 0x80808080u, bias, d2, out + 2 * i);
        }
    }
};

// Q2_K (84-byte super-blocks, src/quant.cpp:398-424) and Q3_K (110, src/quant.cpp:514-553). Step j of group grp covers
// 2-bit fields 2j + h (thread half h) of the 32 quant bytes of 128-value half grp, two scales of 16 values each.
// Their scale products need more than 11 bits, so a value is formed in f32 exactly as the host decoder forms it
// and rounded to f16 once (single-precision arithmetic also issues at twice the rate of the packed f16 kind).
template <>
struct Raw<KRK_CUDA_Q2_K> {
    static constexpr int kSteps = 4;
    uint32_t q[8], sc[2], dm;
    int lead = 0;
    __device__ __forceinline__ void load_block(const uint8_t *slot, int, int, int grp) {
        window(slot, lead + 16 + 32 * grp, q);
        const uint32_t *w = reinterpret_cast<const uint32_t *>(slot + lead);   // 84-byte blocks: word aligned
        sc[0] = w[2 * grp];
        sc[1] = w[2 * grp + 1];
        dm = w[20];
    }
    __device__ __forceinline__ uint32_t loaded() const { return q[0] ^ q[7] ^ sc[0] ^ sc[1] ^ dm; }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const float d = float_of_half_bits(dm & 0xFFFF), dmin = float_of_half_bits(dm >> 16);
        const uint32_t lo = sc[j] & 0x0F0F0F0Fu, hi = (sc[j] >> 4) & 0x0F0F0F0Fu;   // scales, minimums: bytes 2h, 2h + 1 are this chunk's
        const float dl0 = __fmul_rn(d, byte_plus_2_23(lo, 2 * half) - 8388608.0f), dl1 = __fmul_rn(d, byte_plus_2_23(lo, 2 * half + 1) - 8388608.0f);
        const float ml0 = -__fmul_rn(dmin, byte_plus_2_23(hi, 2 * half) - 8388608.0f), ml1 = -__fmul_rn(dmin, byte_plus_2_23(hi, 2 * half + 1) - 8388608.0f);
        const int shift = 4 * j + 2 * half;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t t = (q[i] >> shift) & 0x03030303u;
            const float dl = i < 4 ? dl0 : dl1, ml = i < 4 ? ml0 : ml1;
            const float v0 = fmaf(dl, byte_plus_2_23(t, 0) - 8388608.0f, ml), v1 = fmaf(dl, byte_plus_2_23(t, 1) - 8388608.0f, ml);
            const float v2 = fmaf(dl, byte_plus_2_23(t, 2) - 8388608.0f, ml), v3 = fmaf(dl, byte_plus_2_23(t, 3) - 8388608.0f, ml);
            out[2 * i] = h2_bits(__floats2half2_rn(v0, v1));
            out[2 * i + 1] = h2_bits(__floats2half2_rn(v2, v3));
        }
    }
};
template <>
struct Raw<KRK_CUDA_Q3_K> {
    static constexpr int kSteps = 4;
    uint32_t q[8], hm[8], sc[2];
    float d;
    int lead = 0;
    __device__ __forceinline__ void load_block(const uint8_t *slot, int, int, int grp) {
        window(slot, lead, hm);
#pragma unroll
        for (int i = 0; i < 8; i++) hm[i] >>= 4 * grp;   // mask bit 4 grp + f to bit f
        window(slot, lead + 32 + 32 * grp, q);
        const unsigned short *u = reinterpret_cast<const unsigned short *>(slot + lead + 96);
        const uint32_t a0 = u[0] | ((uint32_t)u[1] << 16), a1 = u[2] | ((uint32_t)u[3] << 16), a2 = u[4] | ((uint32_t)u[5] << 16);
        d = float_of_half_bits(u[6]);
        // scale i: low four bits in the nibbles of bytes 0..7, high two in byte 8 + i % 4 at bits 2 * (i / 4)
        sc[0] = ((a0 >> (4 * grp)) & 0x0F0F0F0Fu) | (((a2 >> (4 * grp)) << 4) & 0x30303030u);
        sc[1] = ((a1 >> (4 * grp)) & 0x0F0F0F0Fu) | (((a2 >> (4 * grp)) << 2) & 0x30303030u);
    }
    __device__ __forceinline__ uint32_t loaded() const { return hm[0] ^ hm[7] ^ q[0] ^ q[7] ^ sc[0] ^ sc[1] ^ __float_as_uint(d); }
    template <int half>
    __device__ __forceinline__ void convert(int j, uint32_t (&out)[16]) const {
        const float dl0 = __fmul_rn(d, byte_plus_2_23(sc[j], 2 * half) - 8388640.0f);   // d * (scale - 32)
        const float dl1 = __fmul_rn(d, byte_plus_2_23(sc[j], 2 * half + 1) - 8388640.0f);
        const int f = 2 * j + half;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int up = 2 - f;
            const uint32_t t = ((q[i] >> (2 * f)) & 0x03030303u) | ((up >= 0 ? hm[i] << up : hm[i] >> -up) & 0x04040404u);
            const float dl = i < 4 ? dl0 : dl1;
            const float v0 = dl * (byte_plus_2_23(t, 0) - 8388612.0f), v1 = dl * (byte_plus_2_23(t, 1) - 8388612.0f);   // q - 4 without the mask bit
            const float v2 = dl * (byte_plus_2_23(t, 2) - 8388612.0f), v3 = dl * (byte_plus_2_23(t, 3) - 8388612.0f);
            out[2 * i] = h2_bits(__floats2half2_rn(v0, v1));
            out[2 * i + 1] = h2_bits(__floats2half2_rn(v2, v3));
        }
    }
};

// ---- the kernel ------------------------------------------------------------------------------------

// One tile of work. Tiles are dealt to the CTAs (clusters) in whole waves; an expert launch's tiles come from its
// device-side list, weight tiles of one token group in a row so that the CTAs at work share the group's X in L2.
struct Tile {
    int w_row;      // first weight row (of the matrix, or of the expert bank)
    int n0;         // first output column
    int x_row;      // first X row
    int m;          // valid tokens
    int kb0, kb1;   // super-blocks of K
    bool piece;     // of a tile that the cluster shares (a CTA's last)
};
// at / p.group. (A division here is 100 clocks and more of every warp's way to its first work, and of a shared tile's end.)
__device__ __forceinline__ int tile_group(const GemmParams &p, int at) {
    return p.group == 1 ? at : p.per_group ? (int)__umulhi((uint32_t)at, p.per_group) : at / p.group;
}
template <int KIND>
struct TileIter {
    int i, n, stride, shared;   // shared: the cluster's shared tile, -1: none (any more)
    __device__ __forceinline__ void init(const GemmParams &p) {
        i = (int)blockIdx.x;
        stride = (int)gridDim.x;
        n = KIND == kDense ? p.n_full : *p.n_groups * p.n_tiles_n;
        shared = -1;
        if (KIND == kDense && p.split > 1) {
            const int at = p.n_full + cluster_id();
            if (at < p.n_tiles_n * p.n_tiles_m) shared = at;
        }
    }
    __device__ __forceinline__ bool next(const GemmParams &p, Tile &t) {
        int at = i;
        t.kb0 = 0, t.kb1 = p.k_blocks, t.piece = false;
        if (i >= n) {
            if (KIND != kDense || shared < 0) return false;
            const int rank = cluster_rank();
            at = shared, shared = -1;
            t.kb0 = rank * p.kb_each + min(rank, p.kb_more), t.kb1 = t.kb0 + p.kb_each + (rank < p.kb_more ? 1 : 0), t.piece = true;
        }
        if (KIND == kDense) {
            const int nt = tile_group(p, at), mt = at - nt * p.n_tiles_m;
            t.w_row = t.n0 = nt * kTileN;
            t.x_row = mt * p.tile_m;
            t.m = p.tile_m;
        } else {
            const int g = tile_group(p, at), nt = at - g * p.n_tiles_n;
            const GemmGroup gr = p.groups[g];
            t.n0 = nt * (KIND == kGateUp ? kTileN / 2 : kTileN);
            t.w_row = gr.expert * (int)p.n_out + t.n0;   // an expert holds n_out rows of (each) bank
            t.x_row = gr.x_row;
            t.m = gr.m;
        }
        i += stride;
        return true;
    }
};
// Tokens the MMA of a tile covers: all of tile_m, or (expert kinds) the group's own rounded up to 16.
template <int KIND>
__device__ __forceinline__ int tile_tokens(const GemmParams &p, const Tile &t) {
    return KIND == kDense ? p.tile_m : (t.m + 15) & ~15;
}

template <int WT, int KIND>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ CUtensorMap x_map,
               const __grid_constant__ WMaps<KIND> w_maps, const __grid_constant__ CUtensorMap y_map) {
    constexpr int kSeg = raw_seg(WT), kStageBytes = kTileN * kSeg;
    constexpr bool kOwnStages = Raw<WT>::kSteps == 4;   // a decode group fills A stages of its own (else both fill every one)
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // (the offset to the next 1024-byte boundary is the same in every CTA of a cluster: same kernel, same layout)
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *raw_ring = smem + p.raw_off;
    float *ystage = reinterpret_cast<float *>(smem + p.y_off);   // [2][kYChunk][kTileN]: accumulator read-out on its way to Y
    GemmBars *sm = reinterpret_cast<GemmBars *>(smem + p.bar_off);
    const int b_bytes = p.tile_m * 128;                          // X of a K step: [tokens][64 f16], 128-byte swizzle
    const int b_stage = b_bytes * p.xk;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);   // warp-uniform to the compiler too
    volatile int *gave_up = &sm->gave_up;

    // Barriers, two per lane: by one thread they took longer than all else before the first copy. The maps are fetched
    // meanwhile.
    if (warp == 0) {
        constexpr int kBars = 2 * (kMaxB + kAStages + kMaxRaw + 2);
        static_assert(offsetof(GemmBars, tmem_base) == 8 * kBars, "barriers come first, in this order");
        for (int b = lane; b < kBars; b += 32) {
            const int a = b - 2 * kMaxB, w = a - 2 * kAStages, d = w - 2 * kMaxRaw;
            const int count = a < 0 ? 1 : w < 0 ? (a >= kAStages ? 1 : kOwnStages ? kDecodeWarps / kDecodeGroups : kDecodeWarps)
                              : d < 0 ? (w >= kMaxRaw ? kDecodeWarps : 1) : d >= 2 ? kEpilogueThreads / 32 : p.dual ? 2 : 1;
            mbar_init(smem_u32(sm) + 8 * b, count);
        }
        if (lane == 0) sm->gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    } else if (warp == kXWarp && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
    } else if (warp == kRawWarp && lane < (row_phased(WT) ? (KIND == kGateUp ? 2 * kPhases : kPhases) : KIND == kGateUp ? 2 : 1)) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&w_maps.m[lane]) : "memory");
    }
    TileIter<KIND> iter;
    if (KIND == kDense) iter.init(p);   // (its parameters arrive cold, so before the barrier, which waits for some anyway)
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(&sm->tmem_base), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // The kernel may start while the one before it in the stream drains: weights are never written by a kernel in
    // flight, so their copies go ahead (dense form); X, the expert list and Y wait for that grid.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (KIND != kDense) asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tmem_base = sm->tmem_base;
    // Accumulators in tensor memory: a tile has one, or one per MMA warp; narrow tiles alternate between two sets.
    const int n_acc = p.tile_m <= kMaxTileM / (p.dual ? 4 : 2) ? 2 : 1;
    const int d_other = p.tile_m <= kMaxTileM / 4 ? 64 : 128;   // second accumulator of a tile, columns on from the first

    if (KIND != kDense) iter.init(p);
    Tile it;

    if (warp < kDecodeWarps) {
        // ===== decode warps: threads r and r + 128 of a group <-> weight row r = TMEM lane r, 32 values each. The groups
        // fill alternate A stages: four warps a scheduler hide each other's latencies =====
        const int r = tid & 127, half = (warp >> 2) & 1, grp = warp / (kDecodeWarps / kDecodeGroups);
        const int trow = tile_row<WT, KIND>(r) & (KIND == kGateUp ? 63 : 127), tslot = tile_slot<WT, KIND>(r);
        // how far the row's first byte lies off a 16-byte boundary (a tile starts a multiple of 8 rows into its matrix)
        const int row_lead = row_phased(WT) ? (int)(((size_t)trow * p.row_bytes) & 15) : 0;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + kTmemA + 16 * half;
        int sa = kOwnStages ? grp : 0, sr = 0;
        uint32_t pa = 0, pr = 0;
        while (iter.next(p, it)) {
            // Rows past n_out need no care here: their staged bytes are zero (the tensor maps fill what lies
            // outside the matrix with zeros), and a zero block decodes to zeros.
            Raw<WT> cur;
            for (int ks = 4 * it.kb0; ks < 4 * it.kb1; ks += Raw<WT>::kSteps) {
                wait_phase(smem_u32(&sm->raw_full[sr]), pr, gave_up, p.status);
                if constexpr (row_phased(WT)) cur.lead = (row_lead + (ks >> 2) * block_bytes(WT)) & 15;
                cur.load_block(raw_ring + (size_t)sr * kStageBytes + tslot * kSeg, half, ks, grp);
                // The group's two K steps fill one tensor-memory stage (Q8_0: its one step half of it); the second is
                // converted while the first's store is in flight.
                uint32_t v[16];
                if (half) cur.template convert<1>(0, v);
                else cur.template convert<0>(0, v);
                // The stage is given back when its bytes ARE in registers: an arrival does not wait for loads in flight, and
                // while the MMAs and the copies of X keep shared memory busy those took longer than a refill (Q8_0, tiles of
                // 96 tokens and more: rows of a later stage in the first ones). Hence the address that needs them, every lane's.
                const int pending = __any_sync(0xFFFFFFFFu, (cur.loaded() & p.zero) != 0u);
                if (lane == 0) mbar_arrive(smem_u32(&sm->raw_empty[sr]) + pending);
                if (++sr == p.n_raw) {
                    sr = 0;
                    pr ^= 1;
                }
                wait_phase(smem_u32(&sm->a_empty[sa]), pa ^ 1, gave_up, p.status);
                tc_fence_after();
                tmem_st16(lane_addr + 64 * sa + (kOwnStages ? 0 : 32 * grp), v);
                if constexpr (kOwnStages) {
                    uint32_t u[16];
                    if (half) cur.template convert<1>(1, u);
                    else cur.template convert<0>(1, u);
                    tmem_st16(lane_addr + 64 * sa + 32, u);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sm->a_full[sa]));
                if ((sa += kOwnStages ? kDecodeGroups : 1) >= kAStages) {
                    sa -= kAStages;
                    pa ^= 1;
                }
            }
        }
    } else if (warp < kDecodeWarps + kEpilogueWarps) {
        // ===== epilogue warps: TMEM lane = weight row, column = token =====
        // The accumulator is read 32 tokens at a time, written to shared memory as [token][weight row] and stored
        // from there, so it is free again as soon as it has been read.
        const int ew = warp - kDecodeWarps, et = tid - kDecodeThreads;
        const uint32_t lane_d = tmem_base + ((uint32_t)(32 * ew) << 16);
        const int my_row = tile_row<WT, KIND>(32 * ew + lane);
        int ybuf = 0, da = 0, first = 0;   // first: as in the MMA warps
        uint32_t ph = 0;
        int n_blk = 0;
        // 32 tokens of the accumulator; of both, where two MMA warps shared the tile's super-blocks (of a single one, only one
        // did anything)
        auto read = [&](uint32_t addr, uint32_t (&v)[32]) {
            if (!p.dual || n_blk == 1) {
                tmem_ld32(addr + (p.dual && (first & 1) ? (uint32_t)d_other : 0u), v);
                tmem_ld_wait();
                return;
            }
            uint32_t w[32];
            tmem_ld32(addr, v);
            tmem_ld32(addr + (uint32_t)d_other, w);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
        };
        asm volatile("griddepcontrol.wait;" ::: "memory");
        while (iter.next(p, it)) {
            wait_phase(smem_u32(&sm->d_full[da]), ph, gave_up, p.status);
            tc_fence_after();
            const uint32_t d_addr = lane_d + 128 * da;
            const int tokens = tile_tokens<KIND>(p, it);
            n_blk = it.kb1 - it.kb0;
            if (KIND == kDense && it.piece) {
                // a piece of K: the whole accumulator goes to shared memory over the drained X ring (every MMA that
                // read it is done); the cluster adds the pieces up below
                float *part = reinterpret_cast<float *>(smem);
                for (int c0 = 0; c0 < tokens; c0 += kYChunk) {
                    uint32_t v[32];
                    read(d_addr + (uint32_t)c0, v);
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (c0 + j < tokens) part[(c0 + j) * kTileN + my_row] = __uint_as_float(v[j]);
                }
                break;   // the last
            }
            for (int c0 = 0; c0 < tokens; c0 += kYChunk) {
                uint32_t v[32];
                read(d_addr + (uint32_t)c0, v);
                if (KIND == kDense && !p.y_tma) {   // a Y the tensor map cannot describe: straight out
                    const int64_t n = it.n0 + my_row, m_first = it.x_row + c0;
                    if (n < p.n_out) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (m_first + j < p.rows) p.y[(m_first + j) * p.n_out + n] = __uint_as_float(v[j]);
                    }
                    continue;
                }
                if (KIND == kDense && et == 0) tma_store_wait_read<1>();   // the store that read this buffer two chunks ago is done with it
                asm volatile("bar.sync 2, %0;" ::"n"(kEpilogueThreads) : "memory");
                float *buf = ystage + ybuf * (kYChunk * kTileN);
#pragma unroll
                for (int j = 0; j < 32; j++) buf[j * kTileN + my_row] = __uint_as_float(v[j]);
                if (KIND == kDense) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("bar.sync 2, %0;" ::"n"(kEpilogueThreads) : "memory");
                if (KIND == kDense) {
                    if (et == 0) {   // rows past the end of Y are clipped by the tensor map
                        tma_store_2d(&y_map, it.n0, it.x_row + c0, smem_u32(buf));
                        tma_store_commit();
                    }
                } else if (KIND == kGateUp) {
                    // four threads a token, 16 outputs each: columns 0..63 of the buffer are gates, 64..127 ups. The
                    // result is rounded to f16 as the GEMM that reads it would round it (finite values saturate).
                    const int tok = et >> 2, col = 16 * (et & 3);
                    if (c0 + tok < it.m) {
                        uint32_t o[8];
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const float2 g = *reinterpret_cast<const float2 *>(buf + tok * kTileN + col + 2 * i);
                            const float2 u = *reinterpret_cast<const float2 *>(buf + tok * kTileN + 64 + col + 2 * i);
                            o[i] = h2_bits(__halves2half2(half_sat(g.x / (1.0f + expf(-g.x)) * u.x), half_sat(g.y / (1.0f + expf(-g.y)) * u.y)));
                        }
                        uint4 *dst = reinterpret_cast<uint4 *>(p.h + (int64_t)(it.x_row + c0 + tok) * p.n_out + it.n0 + col);
                        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
                        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kYChunk / 4; i++) {
                        const int tok = 4 * i + ew;   // a warp per token: 512 contiguous bytes
                        if (c0 + tok < it.m)
                            *reinterpret_cast<float4 *>(p.y + (int64_t)(it.x_row + c0 + tok) * p.n_out + it.n0 + 4 * lane) =
                                *reinterpret_cast<const float4 *>(buf + tok * kTileN + 4 * lane);
                    }
                }
                ybuf ^= 1;
            }
            first += n_blk;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sm->d_empty[da]));   // the accumulator is free again
            if (++da == n_acc) {
                da = 0;
                ph ^= 1;
            }
        }
        // the staging buffers must outlive the stores that read them
        if (KIND == kDense && et == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else if (warp == kXWarp) {
        // ===== TMA producer of X tiles: like the MMA issuer a whole warp, one elected lane issues (from a one-lane branch
        // a copy took some 250 clocks to issue, which bound the formats staged as eight boxes) =====
        const uint32_t elected = elect_one();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        iter.n = __shfl_sync(0xFFFFFFFFu, iter.n, 0);
        int sb = 0;
        uint32_t pb = 0;
        while (iter.next(p, it)) {
            const int boxes = __shfl_sync(0xFFFFFFFFu, (tile_tokens<KIND>(p, it) + kGroupBox - 1) / kGroupBox, 0);
            const int x_row = __shfl_sync(0xFFFFFFFFu, it.x_row, 0);
            for (int ks = 4 * it.kb0; ks < 4 * it.kb1; ks += p.xk) {
                wait_phase(smem_u32(&sm->b_empty[sb]), pb ^ 1, gave_up, p.status);
                const uint32_t bar = smem_u32(&sm->b_full[sb]), dst = smem_u32(smem) + (uint32_t)(sb * b_stage);
                // (dense: one box per K step; else only the boxes that hold tokens of the group)
                mbar_arrive_expect_tx(bar, (uint32_t)(p.xk * (KIND == kDense ? b_bytes : boxes * kGroupBox * 128)), elected);
                for (int j = 0; j < p.xk; j++) {
                    if (KIND == kDense) {
                        tma_load_2d(dst + j * b_bytes, &x_map, (ks + j) * kBK, x_row, bar, elected);
                    } else {
                        for (int b = 0; b < boxes; b++)
                            tma_load_2d(dst + j * b_bytes + b * kGroupBox * 128, &x_map, (ks + j) * kBK, x_row + b * kGroupBox, bar, elected);
                    }
                }
                if (++sb == p.n_b) {
                    sb = 0;
                    pb ^= 1;
                }
            }
        }
    } else if (warp == kRawWarp) {
        // ===== TMA producer of raw block columns =====
        constexpr int kHalves = KIND == kGateUp ? 2 : 1;   // matrices in a weight tile
        constexpr int kPer = Raw<WT>::kSteps;              // K steps per stage
        const uint32_t elected = elect_one();
        iter.n = __shfl_sync(0xFFFFFFFFu, iter.n, 0);
        int sr = 0;
        uint32_t pr = 0;
        while (iter.next(p, it)) {
            const int w_row = __shfl_sync(0xFFFFFFFFu, it.w_row, 0);
            for (int blk = 4 * it.kb0 / kPer; blk < 4 * it.kb1 / kPer; blk++) {
                wait_phase(smem_u32(&sm->raw_empty[sr]), pr ^ 1, gave_up, p.status);
                const uint32_t bar = smem_u32(&sm->raw_full[sr]);
                const uint32_t stage = smem_u32(raw_ring) + (uint32_t)(sr * kStageBytes);
                mbar_arrive_expect_tx(bar, (uint32_t)kStageBytes, elected);
                if constexpr (row_phased(WT)) {
                    constexpr int kBoxRows = kTileN / kPhases / kHalves;
#pragma unroll
                    for (int c = 0; c < kPhases; c++) {
                        // map c starts (c * row_bytes) % 16 bytes before row c; the block's granules from there
                        const int x0 = (((c * p.row_bytes) & 15) + blk * block_bytes(WT)) & ~15;
                        // a matrix of fewer than eight rows has no row c: read outside the map, which fills zeros
                        const int y0 = (KIND != kDense || c < p.n_out) ? w_row / kPhases : (1 << 24);
#pragma unroll
                        for (int hf = 0; hf < kHalves; hf++)
                            tma_load_2d(stage + (hf * (kTileN / 2) + c * kBoxRows) * kSeg, &w_maps.m[hf * kPhases + c], x0, y0, bar, elected);
                    }
                } else {
                    const int x0 = WT == KRK_CUDA_Q8_0 ? 136 * blk - 8 * (blk & 1) : blk * kSeg;   // a multiple of 16
#pragma unroll
                    for (int hf = 0; hf < kHalves; hf++)
                        tma_load_2d(stage + hf * (kTileN / 2) * kSeg, &w_maps.m[hf], x0, w_row, bar, elected);
                }
                if (++sr == p.n_raw) {
                    sr = 0;
                    pr ^= 1;
                }
            }
        }
    } else {
        // ===== MMA issuers: the whole warp walks the loop, one elected lane issues (see umma_f16_ts_step). Their loop shares
        // a scheduler with decode warps, and for narrow tiles its chain of waits, address arithmetic and commits is what
        // a super-block takes (290 clocks a K step against 126 alone). So two warps take super-blocks in turn, each into
        // an accumulator of its own, which the read-out adds. Every ring holds an even number of super-blocks (the A ring
        // two), so that a warp meets each of its slots on every lap and a parity cannot be taken for that of the lap before. =====
        const int who = warp - kMmaWarp, step = p.dual ? 2 : 1;
        const uint32_t elected = elect_one();
        constexpr uint32_t tmem = 0;   // an allocation of all 512 columns starts at the first
        iter.n = __shfl_sync(0xFFFFFFFFu, iter.n, 0);
        const int per_blk = 4 / p.xk;     // X stages per super-block
        int blk = who;                    // this warp's next super-block of the CTA's sequence
        int first = 0;                    // the sequence number of the tile's first super-block
        int sb = (who * per_blk) % p.n_b, sa = 2 * who, da = 0;
        uint32_t pa = 0, pb = 0, pd = 0;
        while ((who == 0 || p.dual) && iter.next(p, it)) {
            const uint32_t idesc = instr_desc(kTileN, __shfl_sync(0xFFFFFFFFu, tile_tokens<KIND>(p, it), 0));
            wait_phase(smem_u32(&sm->d_empty[da]), pd ^ 1, gave_up, p.status);   // the epilogue has drained the accumulator
            tc_fence_after();
            const uint32_t d_tmem = tmem + 128 * da + (who ? d_other : 0);
            const int n_blk = it.kb1 - it.kb0;
            uint32_t fresh = 1u;
            for (; blk < first + n_blk; blk += step) {
                uint32_t b_lo = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const bool new_b = (j & (p.xk - 1)) == 0, new_a = (j & 1) == 0;
                    const uint32_t b_bar = smem_u32(&sm->b_full[sb]), a_bar = smem_u32(&sm->a_full[sa]);
                    if (new_b) {   // both waits in flight together
                        const bool okb = mbar_try_wait(b_bar, pb), oka = !new_a || mbar_try_wait(a_bar, pa);
                        if (!okb) wait_phase(b_bar, pb, gave_up, p.status);
                        if (!oka) wait_phase(a_bar, pa, gave_up, p.status);
                        tc_fence_after();
                        b_lo = smem_desc_lo(smem_u32(smem) + (uint32_t)(sb * b_stage));
                    } else if (new_a) {
                        wait_phase(a_bar, pa, gave_up, p.status);
                        tc_fence_after();
                    }
                    umma_f16_ts_step(d_tmem, tmem + kTmemA + 64 * sa + 32 * (j & 1), b_lo, kSmemDescHi, idesc, j == 0 ? fresh : 0u, elected);
                    b_lo += (uint32_t)b_bytes >> 4;
                    if (((j + 1) & (p.xk - 1)) == 0) {
                        umma_commit(smem_u32(&sm->b_empty[sb]), elected);   // a stage is free once the MMAs that read it are done
                        if (++sb == p.n_b) {
                            sb = 0;
                            pb ^= 1;
                        }
                    }
                    if (j & 1) {
                        umma_commit(smem_u32(&sm->a_empty[sa]), elected);
                        if (++sa == kAStages) {
                            sa = 0;
                            pa ^= 1;
                        }
                    }
                }
                fresh = 0u;
                if (p.dual) {   // past the other warp's super-block
                    sb += per_blk;
                    if (sb >= p.n_b) {
                        sb -= p.n_b;
                        pb ^= 1;
                    }
                    sa += 2;
                    if (sa >= kAStages) {
                        sa -= kAStages;
                        pa ^= 1;
                    }
                }
            }
            first += n_blk;
            umma_commit(smem_u32(&sm->d_full[da]), elected);
            if (++da == n_acc) {
                da = 0;
                pd ^= 1;
            }
        }
    }

    // A shared tile's pieces meet: CTA `rank` adds its share of the tokens over all CTAs of the cluster, in K order. The
    // decode warps do that, who have the time to work out where while the last super-blocks are multiplied.
    const bool sums = KIND == kDense && p.split > 1 && warp < kDecodeWarps;
    int tok = 0, tok_end = 0, col = 0;
    int64_t m = 0, n = 0;
    if (sums) {
        const int rank = cluster_rank(), at = p.n_full + cluster_id();
        const int nt = tile_group(p, at), mt = at - nt * p.n_tiles_m;
        tok = rank * p.sum_tokens + tid / (kTileN / 4), col = 4 * (tid % (kTileN / 4));
        m = (int64_t)mt * p.tile_m + tok, n = (int64_t)nt * kTileN + col;
        tok_end = nt < p.n_tiles_n && n < p.n_out ? min((rank + 1) * p.sum_tokens, p.tile_m) : 0;   // (not: a cluster without a tile)
        tok_end = (int)min((int64_t)tok_end, tok + p.rows - m);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
        __syncwarp();
    }
    if (KIND == kDense && p.split > 1) {
        cluster_sync();
        if (sums) {
            float *y = p.y + m * p.n_out + n;
            for (; tok < tok_end; tok += kDecodeThreads / (kTileN / 4), y += (kDecodeThreads / (kTileN / 4)) * p.n_out) {
                const uint32_t at = smem_u32(smem) + (uint32_t)(tok * kTileN + col) * 4u;
                float4 v[kMaxSplit];   // all in flight together: one after the other they took some 250 ns each
#pragma unroll
                for (int q = 0; q < kMaxSplit; q++)
                    if (q < p.split) v[q] = ld_peer(at, q);
                float4 s = v[0];
#pragma unroll
                for (int q = 1; q < kMaxSplit; q++)
                    if (q < p.split) s.x += v[q].x, s.y += v[q].y, s.z += v[q].z, s.w += v[q].w;
                if (p.y_tma) {   // 16-byte aligned, n_out a multiple of four
                    *reinterpret_cast<float4 *>(y) = s;
                } else {
                    y[0] = s.x;
                    if (n + 1 < p.n_out) y[1] = s.y;
                    if (n + 2 < p.n_out) y[2] = s.z;
                    if (n + 3 < p.n_out) y[3] = s.w;
                }
            }
        }
        // Nobody leaves while its shared memory is being read. Relaxed: what was read has been used by the stores above, and a
        // release would wait for those (700 ns).
        asm volatile("barrier.cluster.arrive.relaxed.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");
    }
}

// A thread takes QUADS quads, a block's width apart and all in flight together. Four, where one each is more than 64 blocks: fewer
// blocks leave more SMs to the GEMM's CTAs, which start beside them, and fit at a time (passes back to back; alone it gives nothing: Q6_K 4096 x 11008 at 37
// tokens 20.8 -> 19.1 us, Q8_0 4096 x 4096 at 64 tokens 12.4 -> 11.2, Q3_K 11008 x 4096 at 300 tokens 50.4 -> 48.3). Below, the
// longer thread only takes longer (16 tokens of 4096 values 8.7 against 9.05).
constexpr int kConvertThreads = 256, kConvertFewBlocks = 64;
template <int QUADS>
__global__ void __launch_bounds__(kConvertThreads) f32_to_f16_kernel(__half *__restrict__ out, const float *__restrict__ in, int64_t n4) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int kBlock = kConvertThreads * QUADS;
    for (int64_t i0 = (int64_t)blockIdx.x * kBlock + threadIdx.x; i0 < n4; i0 += (int64_t)gridDim.x * kBlock) {
        float4 v[QUADS];
#pragma unroll
        for (int j = 0; j < QUADS; j++) {
            const int64_t i = i0 + j * kConvertThreads;
            v[j] = reinterpret_cast<const float4 *>(in)[i < n4 ? i : i0];
        }
#pragma unroll
        for (int j = 0; j < QUADS; j++) {
            const int64_t i = i0 + j * kConvertThreads;
            if (i < n4)
                reinterpret_cast<uint2 *>(out)[i] = make_uint2(h2_bits(__halves2half2(half_sat(v[j].x), half_sat(v[j].y))),
                                                               h2_bits(__halves2half2(half_sat(v[j].z), half_sat(v[j].w))));
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    return fn;
}

// A row-major matrix as a 2-d tensor map (no fill but zeros outside it).
bool encode_2d(CUtensorMap *map, CUtensorMapDataType type, const void *base, int64_t cols, int64_t rows, size_t pitch, int box_cols,
               int box_rows, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promo) {
    EncodeTiledFn encode = encode_tiled();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, type, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promo,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The division-free parameters of GemmParams.
void set_divisions(GemmParams &p, int group, int64_t tiles) {
    const uint64_t most = (uint64_t)tiles + 256, m = (uint64_t)group;   // (clusters without a tile look past the last)
    p.group = group;
    // at * per is at / m * 2^32 and less than at more: the quotient is exact while at * m < 2^32
    p.per_group = m > 1 && most * m < (1ull << 32) ? (uint32_t)(((1ull << 32) + m - 1) / m) : 0u;
    p.k_blocks = (int)(p.n_in / 256);
    p.kb_each = p.k_blocks / p.split;
    p.kb_more = p.k_blocks % p.split;
    p.sum_tokens = (p.tile_m + p.split - 1) / p.split;
}

// The maps over the raw weight bytes of one matrix ([n_out][row_bytes] bytes), for boxes that bring `tile_rows` rows.
// Formats staged as one box: box = one stage's bytes of a row x the rows. Phased formats: map c covers the rows c,
// c + 8, c + 16, ... from the 16-byte boundary at or before row c: inner extent = the lead bytes + one row (so nothing
// past a row's own end is ever read, and what the box holds beyond it is zero fill), pitch = eight rows. A c with no
// row at all (fewer than eight rows in the matrix) repeats map 0; its staged rows are never used.
template <int WT>
bool encode_w_maps(CUtensorMap *maps, const uint8_t *w, int64_t n_out, int row_bytes, int tile_rows) {
    if constexpr (!row_phased(WT)) {
        return encode_2d(maps, CU_TENSOR_MAP_DATA_TYPE_UINT8, w, row_bytes, n_out, row_bytes, raw_seg(WT), tile_rows,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    } else {
        for (int c = 0; c < kPhases; c++) {
            const int cc = c < n_out ? c : 0;
            const size_t start = (size_t)cc * row_bytes, lead = start & 15;
            if (!encode_2d(&maps[c], CU_TENSOR_MAP_DATA_TYPE_UINT8, w + (start - lead), (int64_t)(lead + row_bytes), (n_out - cc + kPhases - 1) / kPhases,
                           (size_t)kPhases * row_bytes, raw_seg(WT), tile_rows / kPhases, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
                return false;
        }
        return true;
    }
}

// Ring depths and the shared-memory map of a launch. The raw ring wants as many K steps in flight as the X ring;
// both grow in turn while they fit.
template <int WT>
size_t layout(GemmParams &p, bool one_tile) {   // one_tile: no CTA has a second one
    const int stage = kTileN * raw_seg(WT), steps = Raw<WT>::kSteps;
    p.xk = p.tile_m <= 64 ? 4 : p.tile_m <= 128 ? 2 : 1;   // X stages of at most 32 KB
    const int xb = p.tile_m * 128 * p.xk;
    const int y_bytes = 2 * kYChunk * kTileN * (int)sizeof(float);
    const int room = kSmemMax - 1024 - y_bytes - (int)sizeof(GemmBars);
    // Tiles of 65..128 tokens have room for two accumulators only: for two MMA warps, or for the read-out beside the next
    // tile, which is worth more where a CTA has several tiles of short K (Q8_0 experts of K = 2048: 34.7 against 40.8 us).
    p.dual = p.tile_m <= kMaxTileM / 4 || (p.tile_m <= kMaxTileM / 2 && p.n_in >= (one_tile ? 2048 : 4096));
    const int unit_b = p.dual ? 2 * (4 / p.xk) : 1;   // the X ring grows by this many stages (see the MMA warps)
    p.n_b = p.dual ? unit_b : kMinB;
    p.n_raw = kMinRaw;
    for (;;) {
        const int left = room - p.n_b * xb - p.n_raw * stage;
        const bool want_b = p.n_b + unit_b <= kMaxB && p.n_b * p.xk < steps * p.n_raw;
        if (want_b && left >= unit_b * xb) p.n_b += unit_b;
        else if (p.n_raw < kMaxRaw && left >= stage) p.n_raw++;
        else if (p.n_b + unit_b <= kMaxB && left >= unit_b * xb) p.n_b += unit_b;
        else break;
    }
    p.raw_off = p.n_b * xb;
    p.y_off = p.raw_off + p.n_raw * stage;
    p.bar_off = p.y_off + y_bytes;
    return (size_t)p.bar_off + sizeof(GemmBars) + 1024;
}

template <int WT, int KIND>
int launch_kernel(const GemmParams &p, const CUtensorMap &x_map, const WMaps<KIND> &w_maps, const CUtensorMap &y_map, int grid, size_t smem,
                  cudaStream_t st) {
    static bool configured[64] = {};
    auto kernel = gemm_tc_kernel<WT, KIND>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        if (e != cudaSuccess) {
            note_cuda_error(e);
            return KRK_CUDA_ELAUNCH;
        }
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.split > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p, x_map, w_maps, y_map);
    note_launch(1, KRK_CUDA_FAMILY_GEMM_TC);
    if (e != cudaSuccess) {
        note_cuda_error(e);
        (void)cudaGetLastError();
        return KRK_CUDA_ELAUNCH;
    }
    return KRK_CUDA_OK;
}

// How many clusters of 1..kMaxSplit CTAs (one per SM) the current device holds at a time; looked up once per device.
const int *cluster_counts(int sms) {
    static std::mutex mu;
    static int counts[64][kMaxSplit + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    std::lock_guard<std::mutex> lk(mu);
    int *c = counts[dev];
    if (c[1] == 0) {
        auto kernel = gemm_tc_kernel<KRK_CUDA_Q4_K, kDense>;   // every dense form fills an SM alike
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        for (int s = 2; s <= kMaxSplit; s++) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(sms / s * s));
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kSmemMax;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)s;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) n = 0;   // none: tiles are not shared
            // Odd sizes do not pack that densely while the CTAs of the kernel before leave, and a cluster that comes late
            // costs a wave, so three of them are not counted on. Of 60 drawn products 58 choose the same either way; Q8_0
            // 2816 x 5120 at 439 tokens takes 28.4 us with all 45 clusters of three and 21.1 with this choice (74 of two),
            // Q6_K 9968 x 10496 at 318 tokens 74.8 and 74.4, and Q3_K 11008 x 4096 at 300 tokens 66 and 50.
            c[s] = (s & 1) ? (n > 3 ? n - 3 : 0) : n;
        }
        (void)cudaGetLastError();
        c[1] = sms;
    }
    return c;
}

template <int WT>
int launch_dense(GemmParams &p, const GemmPlan &g, const uint8_t *w, const __half *xh, cudaStream_t st, const float *x_f32) {
    CUtensorMap x_map, y_map;
    WMaps<kDense> w_maps;
    set_divisions(p, g.n_tiles_m, (int64_t)g.n_tiles_n * g.n_tiles_m);
    const size_t smem = layout<WT>(p, g.n_full == 0 || (g.n_full <= g.grid && g.split == 1));
    if (!encode_2d(&x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, xh, p.n_in, p.rows, (size_t)p.n_in * sizeof(__half), kBK, p.tile_m,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !encode_w_maps<WT>(w_maps.m, w, p.n_out, p.row_bytes, kTileN))
        return KRK_CUDA_ELAUNCH;
    // Y as a [rows][n_out] f32 matrix, box = 128 weight rows x kYChunk tokens, for the stores of the read-out. A Y that
    // is not 16-byte aligned with 16-byte-multiple rows cannot be described: the kernel then stores directly.
    if (p.y_tma && !encode_2d(&y_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.y, p.n_out, p.rows, (size_t)p.n_out * sizeof(float), kTileN, kYChunk,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE))
        return KRK_CUDA_ELAUNCH;
    if (!p.y_tma) y_map = x_map;   // never used
    // every map is encoded: from here on only a launch can fail
    if (x_f32) {
        const int rc = launch_f32_to_f16(const_cast<__half *>(xh), x_f32, p.rows * p.n_in, st);
        if (rc != KRK_CUDA_OK) return rc;
    }
    return launch_kernel<WT, kDense>(p, x_map, w_maps, y_map, g.grid, smem, st);
}

int run_dense(float *y, const void *x, int x_dtype, const uint8_t *w, int wt, int64_t n_out, int64_t n_in, int64_t rows, __half *x_copy,
              int *status, int sms, cudaStream_t st) {
    const GemmPlan g = plan_gemm(n_out, n_in, rows, sms, cluster_counts(sms));
    GemmParams p{};
    p.y = y;
    p.n_out = n_out;
    p.n_in = n_in;
    p.rows = rows;
    p.tile_m = g.tile_m;
    p.n_tiles_n = g.n_tiles_n;
    p.n_tiles_m = g.n_tiles_m;
    p.split = g.split;
    p.n_full = g.n_full;
    p.row_bytes = (int)row_bytes(wt, n_in);
    p.y_tma = ((reinterpret_cast<uintptr_t>(y) & 15) == 0 && (n_out % 4) == 0) ? 1 : 0;
    p.status = status;
    const bool f32 = x_dtype == KRK_CUDA_X_F32;
    const __half *xh = f32 ? x_copy : static_cast<const __half *>(x);
    int rc = KRK_CUDA_EDTYPE;
    KRK_DISPATCH_WT(wt, rc = launch_dense<WT>(p, g, w, xh, st, f32 ? static_cast<const float *>(x) : nullptr));
    return rc;
}

template <int WT, int KIND>
int launch_experts(GemmParams &p, const ExpertGemm &e, cudaStream_t st) {
    CUtensorMap x_map;
    WMaps<KIND> w_maps;
    constexpr int kRows = KIND == kGateUp ? kTileN / 2 : kTileN;   // rows of one matrix in a weight tile
    p.row_bytes = (int)row_bytes(WT, e.n_in);
    set_divisions(p, p.n_tiles_n, (int64_t)e.max_groups * p.n_tiles_n);
    const size_t smem = layout<WT>(p, false);
    if (!encode_2d(&x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, e.x, e.n_in, e.x_rows, (size_t)e.n_in * sizeof(__half), kBK, kGroupBox,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !encode_w_maps<WT>(w_maps.m, e.w, e.bank_rows, p.row_bytes, kRows) ||
        (KIND == kGateUp && !encode_w_maps<WT>(w_maps.m + (row_phased(WT) ? kPhases : 1), e.w_up, e.bank_rows, p.row_bytes, kRows)))
        return KRK_CUDA_ELAUNCH;
    const long long tiles = (long long)e.max_groups * p.n_tiles_n;
    const int sms = sm_count();
    return launch_kernel<WT, KIND>(p, x_map, w_maps, x_map, (int)(tiles < sms ? tiles : sms), smem, st);
}

template <int KIND>
int run_experts(GemmParams &p, const ExpertGemm &e, cudaStream_t st) {
    p.n_out = e.n_out;
    p.n_in = e.n_in;
    p.rows = e.x_rows;
    p.tile_m = e.tile_m;
    p.n_tiles_n = (int)(e.n_out / (KIND == kGateUp ? kTileN / 2 : kTileN));
    p.n_tiles_m = 1;
    p.split = 1;
    p.groups = e.groups;
    p.n_groups = e.n_groups;
    p.status = device_status_word();
    if (!p.status) return KRK_CUDA_EDEVICE;
    int rc = KRK_CUDA_EDTYPE;
    KRK_DISPATCH_WT(e.wt, rc = (launch_experts<WT, KIND>(p, e, st)));
    return rc;
}

} // namespace

int launch_gemm_experts_gate_up(__half *h, const ExpertGemm &e, cudaStream_t st) {
    GemmParams p{};
    p.h = h;
    return run_experts<kGateUp>(p, e, st);
}
int launch_gemm_experts_down(float *y, const ExpertGemm &e, cudaStream_t st) {
    GemmParams p{};
    p.y = y;
    return run_experts<kDown>(p, e, st);
}

// f16 copy of n activations (n a multiple of 4), finite values beyond the f16 range saturated (half_sat).
int launch_f32_to_f16(__half *out, const float *in, int64_t n, cudaStream_t st) {
    const int64_t n4 = n / 4, few = (n4 + kConvertThreads - 1) / kConvertThreads, many = (n4 + 4 * kConvertThreads - 1) / (4 * kConvertThreads);
    if (few <= kConvertFewBlocks) return launched(launch_overlapped(f32_to_f16_kernel<1>, dim3((unsigned)few), dim3(kConvertThreads), st, out, in, n4));
    const int64_t most = (int64_t)sm_count() * (2048 / kConvertThreads);
    return launched(launch_overlapped(f32_to_f16_kernel<4>, dim3((unsigned)(many < most ? many : most)), dim3(kConvertThreads), st, out, in, n4));
}

size_t gemm_workspace_bytes(int x_dtype, int64_t, int64_t n_in, int64_t rows) {
    return x_dtype == KRK_CUDA_X_F32 ? (((size_t)rows * (size_t)n_in * sizeof(__half) + 255) & ~(size_t)255) : 0;
}

int launch_gemm_tc(float *y, const void *x, int x_dtype, const uint8_t *w, int wt, int64_t n_out, int64_t n_in,
                   int64_t rows, void *workspace, cudaStream_t st) {
    if (rows > (1 << 24) || n_out > (1 << 30) || n_in > (1 << 24)) return KRK_CUDA_ESHAPE;
    int *status = device_status_word();
    if (!status) return KRK_CUDA_EDEVICE;
    return run_dense(y, x, x_dtype, w, wt, n_out, n_in, rows, static_cast<__half *>(workspace), status, sm_count(), st);
}

// ---- prefill GEMM for callers that must not allocate --------------------------------------------------
// The f32-activation form of the prefill GEMM needs an f16 copy of X. krk_cuda_gemm takes that space
// from the caller; this entry takes it from a fixed array that lives in the library's device image, so
// that a host which has already committed all device memory (an engine that sizes weights and KV cache
// against a budget at load time and allocates nothing afterwards), or which cannot tolerate the implicit
// device synchronisation of an allocation in the middle of a decode loop, can still run it.

constexpr int64_t kStaticHalves = 4ll << 20;   // rows * n_in <= 4 Mi values (8 MiB of f16), e.g. 1024 x 4096
static __device__ __align__(256) unsigned char g_static_scratch[kStaticHalves * 2 + 256];   // f16 X, then a status word
std::mutex g_static_mu;
unsigned char *g_static_addr[64] = {};   // device address of the array, per device, once looked up
int g_static_sms[64] = {};

} // namespace krk_cuda

using namespace krk_cuda;

extern "C" int krk_cuda_gemm_f32_static(void *y_f32, const void *x_f32, const void *w, int wt, int64_t n_out, int64_t n_in,
                                        int64_t rows, void *stream) {
    if (!krk_cuda_dtype_ok(wt) || !gemm_tc_takes(wt)) return KRK_CUDA_EDTYPE;
    if (n_out < 0 || rows < 0 || !krk_cuda_gemm_k_ok(wt, n_in) || n_in % 256 != 0) return KRK_CUDA_ESHAPE;
    if (rows > (1 << 24) || n_out > (1 << 30) || n_in > (1 << 24)) return KRK_CUDA_ESHAPE;
    if (n_out == 0 || rows == 0) return KRK_CUDA_OK;
    if (!y_f32 || !x_f32 || !w) return KRK_CUDA_ENULL;
    if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(x_f32) & 15) || (reinterpret_cast<uintptr_t>(y_f32) & 3))
        return KRK_CUDA_EALIGN;
    if (rows * n_in > kStaticHalves) return KRK_CUDA_ETOOBIG;   // larger than the fixed array: use krk_cuda_gemm

    // Once per device, with that device current: the device address of the array. In host code the
    // array's name is only a handle for this query, never a pointer a kernel may be given.
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return KRK_CUDA_EDEVICE;
    unsigned char *scratch = nullptr;
    int sms = 0;
    {
        // first use on this device, under a lock so that a second host thread never sees half of it
        std::lock_guard<std::mutex> lk(g_static_mu);
        if (!g_static_addr[dev]) {
            void *ptr = nullptr;
            int n_sm = 0;
            e = cudaGetSymbolAddress(&ptr, g_static_scratch);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess || !ptr || n_sm <= 0) {
                if (e != cudaSuccess) note_cuda_error(e);
                return KRK_CUDA_EDEVICE;
            }
            g_static_sms[dev] = n_sm;
            g_static_addr[dev] = static_cast<unsigned char *>(ptr);
        }
        scratch = g_static_addr[dev];
        sms = g_static_sms[dev];
    }
    // Every call overwrites the part of the array it uses before reading it (the conversion kernel), so nothing of
    // the previous call's contents is ever consumed.
    return run_dense(static_cast<float *>(y_f32), x_f32, KRK_CUDA_X_F32, static_cast<const uint8_t *>(w), wt, n_out, n_in, rows,
                     reinterpret_cast<__half *>(scratch), reinterpret_cast<int *>(scratch + kStaticHalves * 2), sms,
                     static_cast<cudaStream_t>(stream));
}

extern "C" int krk_cuda_gemm_f32_static_status(void) {
    // The word behind the f16 area: 0, or the code a bounded wait of this entry's kernels left there.
    // Read and cleared through the symbol itself (copies, no allocation); synchronises the device.
    int v = 0;
    const size_t at = (size_t)kStaticHalves * 2;
    if (cudaDeviceSynchronize() != cudaSuccess) return KRK_CUDA_ELAUNCH;
    if (cudaMemcpyFromSymbol(&v, g_static_scratch, sizeof v, at) != cudaSuccess) return KRK_CUDA_EDEVICE;
    if (v != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_static_scratch, &zero, sizeof zero, at);
    }
    return v;
}
