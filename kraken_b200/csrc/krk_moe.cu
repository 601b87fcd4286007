// Router and routed-expert FFN: one token, decode batches and prefill.
//
// The routing result stays on the device: expert ids are read by the kernels themselves,
// so no logits or ids cross PCIe (the reference downloads the logits and routes on the
// host, src/engine.cpp:11678-11920, or reads device ids in its opt-in moe_dispatch,
// src/hip/kernels/moe_table.hpp:67-180).
#include "krk_chunk.cuh"

namespace krk_cuda {

namespace {

constexpr int kMaxExperts = 1024;
constexpr int kMaxK = 32;

// The sum of v[0..n) in index order (the order the host adds them in), by a whole warp: each lane fetches one value
// of every 32 and the running sum takes them lane by lane through shuffles, so the chain is 4-cycle additions
// instead of one shared-memory round trip per term. Every lane returns the sum.
__device__ __forceinline__ float ordered_sum(const float *v, int n, int lane) {
    float sum = 0.0f;
    for (int base = 0; base < n; base += 32) {
        const float mine = base + lane < n ? v[base + lane] : 0.0f;
        const int m = min(32, n - base);
#pragma unroll 8
        for (int i = 0; i < m; i++) sum = __fadd_rn(sum, __shfl_sync(0xFFFFFFFFu, mine, i));
    }
    return sum;
}

// The k largest of prob[0..n) in slot order by one warp: strict '>' so equal values keep the lower index
// (src/engine.cpp:11857-11886). Lane s (s < k) returns slot s's index (-1: none left) and value; `sum` is the sum of
// the picked values in slot order. Up to 128 entries live in registers (four per lane) and a round is two warp
// reductions: the maximum over the bit patterns of the (non-negative) values, then the lowest index among the lanes
// that hold it. More entries take rounds over shared memory (prob is then modified: -2 marks a taken entry).
__device__ __forceinline__ void topk_warp(float *prob, int n, int k, int lane, int &my_id, float &my_w, float &sum) {
    my_id = -1;
    my_w = 0.0f;
    sum = 0.0f;
    if (n <= 128) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = lane + 32 * j < n ? prob[lane + 32 * j] : -2.0f;
        for (int s = 0; s < k; s++) {
            float bp = -1.0f;
            int be = 0x7FFFFFFF;
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (v[j] > bp) {
                    bp = v[j];
                    be = lane + 32 * j;
                }
            const unsigned key = bp >= 0.0f ? __float_as_uint(bp) + 1u : 0u;   // bit patterns of values >= 0 order like the values
            const unsigned top = __reduce_max_sync(0xFFFFFFFFu, key);
            const unsigned win = __reduce_min_sync(0xFFFFFFFFu, (key == top && top != 0u) ? (unsigned)be : 0x7FFFFFFFu);
            const bool ok = top != 0u;
            const float w = ok ? __uint_as_float(top - 1u) : 0.0f;
            sum = __fadd_rn(sum, w);
            if (lane == s) {
                my_id = ok ? (int)win : -1;
                my_w = w;
            }
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (ok && lane + 32 * j == (int)win) v[j] = -2.0f;
        }
        return;
    }
    for (int s = 0; s < k; s++) {
        float bp = -1.0f;
        int be = 0x7FFFFFFF;
        for (int e = lane; e < n; e += 32) {
            const float pe = prob[e];
            if (pe > bp) {
                bp = pe;
                be = e;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float op = __shfl_xor_sync(0xFFFFFFFFu, bp, o);
            const int oe = __shfl_xor_sync(0xFFFFFFFFu, be, o);
            if (op > bp || (op == bp && oe < be)) {
                bp = op;
                be = oe;
            }
        }
        const bool ok = be < n && bp >= 0.0f;
        const float w = ok ? bp : 0.0f;
        sum = __fadd_rn(sum, w);
        if (lane == s) {
            my_id = ok ? be : -1;
            my_w = w;
        }
        if (ok && lane == 0) prob[be] = -2.0f;
        __syncwarp();
    }
}

// One warp per token. Softmax as the reference computes it: subtract the maximum, sum the
// exponentials in expert order, multiply by the reciprocal (src/engine.cpp:11704-11713);
// then k picks of the largest probability, strict '>' so equal probabilities keep the lower
// id (:11857-11886); then the picked weights are divided by their slot-order sum
// (:11913-11918).
__device__ __forceinline__ void route_token(int32_t *__restrict__ ids, float *__restrict__ wts, const float *__restrict__ lg,
                                            int n_expert, int k, float *prob, int *sid, int lane) {
    float mx = -INFINITY;
    for (int e = lane; e < n_expert; e += 32) mx = fmaxf(mx, lg[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    for (int e = lane; e < n_expert; e += 32) prob[e] = exp_as_host(__fsub_rn(lg[e], mx));
    __syncwarp();
    const float sum = ordered_sum(prob, n_expert, lane);
    const float inv = sum > 0.0f ? __fdiv_rn(1.0f, sum) : 0.0f;
    for (int e = lane; e < n_expert; e += 32) prob[e] = __fmul_rn(prob[e], inv);
    __syncwarp();

    int my_id;
    float my_w, ksum;
    topk_warp(prob, n_expert, k, lane, my_id, my_w, ksum);
    const float kinv = ksum > 0.0f ? __fdiv_rn(1.0f, ksum) : 0.0f;
    if (lane < k) {
        ids[lane] = my_id;
        wts[lane] = __fmul_rn(my_w, kinv);
        if (sid) sid[lane] = my_id;
    }
}

__global__ void __launch_bounds__(32)
route_kernel(int32_t *__restrict__ ids, float *__restrict__ wts, const float *__restrict__ logits,
             int n_expert, int k) {
    __shared__ float prob[kMaxExperts];
    const int64_t t = blockIdx.x;
    route_token(ids + t * k, wts + t * k, logits + t * n_expert, n_expert, k, prob, nullptr, threadIdx.x);
}

// The router in the three steps Backend exposes (include/krk/backend.hpp:934-986): probabilities,
// selection, expert-major plan. Same arithmetic as route_token, split where the interface splits it.
__global__ void __launch_bounds__(32)
router_softmax_kernel(float *__restrict__ probs, const float *__restrict__ logits, int n_expert) {
    const float *lg = logits + (int64_t)blockIdx.x * n_expert;
    float *pr = probs + (int64_t)blockIdx.x * n_expert;
    const int lane = threadIdx.x;
    float mx = -INFINITY;
    for (int e = lane; e < n_expert; e += 32) mx = fmaxf(mx, lg[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    for (int e = lane; e < n_expert; e += 32) pr[e] = exp_as_host(__fsub_rn(lg[e], mx));
    __syncwarp();
    const float sum = ordered_sum(pr, n_expert, lane);   // in expert order, as the host adds them
    const float inv = sum > 0.0f ? __fdiv_rn(1.0f, sum) : 0.0f;
    for (int e = lane; e < n_expert; e += 32) pr[e] = __fmul_rn(pr[e], inv);
}

// k picks of the largest probability per row (strict '>': a tie keeps the lower id), weights = the picked
// probabilities, divided by their slot-order sum when `normalize`, times `scale`.
__global__ void __launch_bounds__(32)
router_topk_kernel(const float *__restrict__ probs, int n_expert, int k, int32_t *__restrict__ ids, float *__restrict__ wts,
                   int normalize, float scale) {
    __shared__ float prob[kMaxExperts];
    const float *pr = probs + (int64_t)blockIdx.x * n_expert;
    const int lane = threadIdx.x;
    for (int e = lane; e < n_expert; e += 32) prob[e] = pr[e];
    __syncwarp();
    int my_id;
    float my_w, ksum;
    topk_warp(prob, n_expert, k, lane, my_id, my_w, ksum);
    const float kinv = normalize ? (ksum > 0.0f ? __fdiv_rn(1.0f, ksum) : 0.0f) : 1.0f;
    if (lane < k) {
        float w = normalize ? __fmul_rn(my_w, kinv) : my_w;
        if (scale != 1.0f) w = __fmul_rn(w, scale);
        ids[(int64_t)blockIdx.x * k + lane] = my_id;
        wts[(int64_t)blockIdx.x * k + lane] = w;
    }
}

// The expert-major plan of a layer from the selected ids: off[n_expert + 1] prefix offsets, rows[n * k] the
// token of each entry and wt[n * k] its weight, entries of one expert in (token, slot) order: the order of the
// host's plan (src/engine.cpp:12215-12248; device twin src/hip/kernels/router.hpp:252-289). Thread e walks
// the pairs in order for expert e, so the order is prescribed, not left to scheduling. One block.
__global__ void __launch_bounds__(1024)
moe_plan_build_kernel(const int32_t *__restrict__ ids, int n_rows, int k, int n_expert, int32_t *__restrict__ off,
                      int32_t *__restrict__ rows, float *__restrict__ wt, const float *__restrict__ wts) {
    __shared__ int count[kMaxExperts + 1];
    const int nk = n_rows * k;
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) {
        int c = 0;
        for (int i = 0; i < nk; i++) c += ids[i] == e;
        count[e] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int e = 0; e < n_expert; e++) {
            const int c = count[e];
            count[e] = run;
            off[e] = run;
            run += c;
        }
        off[n_expert] = run;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) {
        int at = count[e];
        for (int i = 0; i < nk; i++)
            if (ids[i] == e) {
                rows[at] = i / k;
                wt[at] = wts ? wts[i] : 0.0f;
                at++;
            }
    }
}

struct MoeParams {
    const uint8_t *gate, *up, *down;
    const float *x;        // [n_tok][n_embd]
    const int32_t *ids;    // [n_tok][k]
    const float *wts;      // [n_tok][k]
    float *h;              // [n_tok*k][n_ff]   silu(gate) * up per pick
    float *d;              // [n_tok*k][n_embd] down projection per pick
    float *y;              // [n_tok][n_embd]
    int64_t n_embd, n_ff;
    int n_local, expert_base, k, n_tok;
    const int32_t *pos;    // row of d that holds a pick (null: the pick's own number)
    int vec;               // y takes float4 stores
};

__device__ __forceinline__ int local_expert(const MoeParams &p, int pick) {
    const int e = p.ids[pick] - p.expert_base;
    return (e >= 0 && e < p.n_local) ? e : -1;
}

// h[pick][row] = silu(Wgate_e[row] . x_t) * (Wup_e[row] . x_t); one warp per (pick, row).
template <int WT>
__global__ void __launch_bounds__(256)
moe_gate_up_kernel(const __grid_constant__ MoeParams p) {
    const int pick = blockIdx.y;
    const int e = local_expert(p, pick);
    if (e < 0) return;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= p.n_ff) return;
    const size_t rb = row_bytes(WT, p.n_embd);
    const uint8_t *g = p.gate + ((size_t)e * p.n_ff + row) * rb;
    const uint8_t *u = p.up + ((size_t)e * p.n_ff + row) * rb;
    const float *x = p.x + (int64_t)(pick / p.k) * p.n_embd;
    float sg = 0.0f, su = 0.0f;
    for (int64_t c = lane; c < (p.n_embd >> 5); c += 32) {
        sg += chunk_dot<WT>(g, c, x);
        su += chunk_dot<WT>(u, c, x);
    }
    sg = warp_sum(sg);
    su = warp_sum(su);
    if (lane == 0)
        p.h[(int64_t)pick * p.n_ff + row] = __fmul_rn(__fdiv_rn(sg, __fadd_rn(1.0f, exp_as_host(-sg))), su);
}

// d[pick][row] = Wdown_e[row] . h[pick]
template <int WT>
__global__ void __launch_bounds__(256)
moe_down_kernel(const __grid_constant__ MoeParams p) {
    const int pick = blockIdx.y;
    const int e = local_expert(p, pick);
    if (e < 0) return;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= p.n_embd) return;
    const uint8_t *w = p.down + ((size_t)e * p.n_embd + row) * row_bytes(WT, p.n_ff);
    const float *h = p.h + (int64_t)pick * p.n_ff;
    float s = 0.0f;
    for (int64_t c = lane; c < (p.n_ff >> 5); c += 32) s += chunk_dot<WT>(w, c, h);
    s = warp_sum(s);
    if (lane == 0) p.d[(int64_t)pick * p.n_embd + row] = s;
}

// y[t][j] = sum over the picks of token t held here, ascending expert id, of w * d[pick][j]
// starting from zero: the order and the arithmetic of the reference's per-expert
// scatter_axpy_rows chain (src/engine.cpp:12353-, src/backend_cpu.cpp:3193-3220).
constexpr int kCombineThreads = 128;
__global__ void __launch_bounds__(kCombineThreads)
moe_combine_kernel(const __grid_constant__ MoeParams p) {
    __shared__ int s_row[kMaxK];
    __shared__ float s_w[kMaxK];
    __shared__ int s_n;
    // programmatic dependent launch: this grid may start while the one before it drains (it reads nothing before
    // that grid is complete), and lets the one after it start the same way
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = blockIdx.x;
    if (threadIdx.x < 32) {
        // lane s looks at slot s of this token: its place among the slots held here, by expert id
        const int s = threadIdx.x;
        int id = 0x7FFFFFFF, e = -1;
        if (s < p.k) {
            id = p.ids[t * p.k + s];
            e = local_expert(p, t * p.k + s);
        }
        int rank = 0, n = 0;
        for (int j = 0; j < p.k; j++) {
            const int idj = __shfl_sync(0xFFFFFFFFu, id, j), ej = __shfl_sync(0xFFFFFFFFu, e, j);
            if (ej >= 0) {
                n++;
                rank += (idj < id || (idj == id && j < s)) ? 1 : 0;
            }
        }
        if (e >= 0) {
            s_row[rank] = p.pos ? p.pos[t * p.k + s] : t * p.k + s;
            s_w[rank] = p.wts[t * p.k + s];
        }
        if (s == 0) s_n = n;
    }
    __syncthreads();
    const int n = s_n;
    const int64_t n4 = p.n_embd >> 2;   // rows are whole 32-value blocks
    for (int64_t j = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; j < n4; j += (int64_t)gridDim.y * blockDim.x) {
        // the loads of a batch of eight go out together; the additions keep their order
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int i0 = 0; i0 < n; i0 += 8) {
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                v[i] = i0 + i < n ? reinterpret_cast<const float4 *>(p.d + (int64_t)s_row[i0 + i] * p.n_embd)[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (i0 + i < n) {
                    const float w = s_w[i0 + i];
                    acc.x = __fadd_rn(acc.x, __fmul_rn(w, v[i].x));
                    acc.y = __fadd_rn(acc.y, __fmul_rn(w, v[i].y));
                    acc.z = __fadd_rn(acc.z, __fmul_rn(w, v[i].z));
                    acc.w = __fadd_rn(acc.w, __fmul_rn(w, v[i].w));
                }
        }
        float *y = p.y + (int64_t)t * p.n_embd + 4 * j;
        if (p.vec) *reinterpret_cast<float4 *>(y) = acc;
        else y[0] = acc.x, y[1] = acc.y, y[2] = acc.z, y[3] = acc.w;
    }
}

// Builds the two device-side matrix tables of the streaming path from the routed expert ids: one
// gate/up pair and one down matrix per pick this bank holds, ordered by expert id so that an expert
// picked by several tokens is streamed by neighbouring CTAs at about the same time (its second read
// comes from L2). One block; picks <= kPlanThreads.
// With `logits` the routing itself runs first, one warp per token (n_tok <= 8), writing p.ids / p.wts.
constexpr int kPlanThreads = 256;
constexpr int kPlanRouteExperts = 1024;   // experts the fused routing holds in shared memory, per token
__global__ void __launch_bounds__(kPlanThreads)
moe_plan_kernel(const __grid_constant__ MoeParams p, StreamTable *gate_up, StreamTable *down, int wt_gate_up, int wt_down,
                size_t rb_gate_up, size_t rb_down, const float *logits, int n_expert) {
    __shared__ int key[kPlanThreads];
    __shared__ float prob[KRK_CUDA_MAX_ROWS][kPlanRouteExperts];
    __shared__ int sid[KRK_CUDA_MAX_ROWS][kMaxK];   // the ids the fused routing picked, for the plan below
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // (see moe_combine_kernel)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (logits) {
        const int t = threadIdx.x >> 5;
        if (t < p.n_tok)
            route_token(const_cast<int32_t *>(p.ids) + t * p.k, const_cast<float *>(p.wts) + t * p.k,
                        logits + (int64_t)t * n_expert, n_expert, p.k, prob[t], sid[t], threadIdx.x & 31);
        __syncthreads();   // the ids written above are read below by other threads of this block
    }
    const int n_pick = p.n_tok * p.k, pick = threadIdx.x;
    int e = -1;
    if (pick < n_pick) {
        // (with the routing fused the ids come out of shared memory, not back from global memory)
        const int id = logits ? sid[pick / p.k][pick % p.k] : p.ids[pick];
        const int le = id - p.expert_base;
        e = (le >= 0 && le < p.n_local) ? le : -1;
    }
    key[pick] = e >= 0 ? e * kPlanThreads + pick : 0x7FFFFFFF;
    const int n = __syncthreads_count(e >= 0);
    if (e >= 0) {
        int rank = 0;
        for (int j = 0; j < n_pick; j++) rank += key[j] < key[pick];
        const float *x = p.x + (int64_t)(pick / p.k) * p.n_embd;
        float *h = p.h + (int64_t)pick * p.n_ff;
        GemvMat g, u, d;
        g.w = p.gate + (size_t)e * p.n_ff * rb_gate_up;
        u.w = p.up + (size_t)e * p.n_ff * rb_gate_up;
        g.x = u.x = x;
        g.y = u.y = h;            // the pair's fold writes silu(gate) * up through the gate's pointer
        g.n_out = u.n_out = p.n_ff;
        g.wt = u.wt = wt_gate_up;
        d.w = p.down + (size_t)e * p.n_embd * rb_down;
        d.x = h;
        d.y = p.d + (int64_t)pick * p.n_embd;
        d.n_out = p.n_embd;
        d.wt = wt_down;
        gate_up->mat[2 * rank] = g;
        gate_up->mat[2 * rank + 1] = u;
        down->mat[rank] = d;
    }
    if (threadIdx.x == 0) gate_up->n_entries = down->n_entries = n;
}

// ---- more than one token ------------------------------------------------------------------------------------
// Expert-major (the reference's grouped form, src/engine.cpp:12353-12690), planned and run on the device without the
// host ever seeing the counts. Experts that more than kFewRows tokens picked run on the tensor cores: their tokens'
// rows are gathered into one f16 block, groups of up to tile_m rows of it are the token tiles of the expert GEMMs.
// Experts with fewer rows keep f32 activations on the streaming kernel, `cap` rows of an expert per table entry, so
// that an expert's weights are streamed once per `cap` of its tokens (entries of one expert are neighbours: a second
// read comes from level 2). One table, one launch: the host picks `cap` from the expected rows per expert.
constexpr int kFewRows = KRK_CUDA_MAX_ROWS;
constexpr int kRouteFloats = kMaxExperts * kFewRows;   // router probabilities that fit beside the plan
struct GroupedParams {
    const uint8_t *gate, *up, *down;
    size_t rb_gate_up, rb_down;
    int wt_gate_up, wt_down;
    const float *x;        // [n_tok][n_embd]
    const int32_t *ids;    // [n_tok][k]
    const float *wts;      // [n_tok][k]
    const float *logits;   // set: the routing runs first and writes ids and wts ([n_tok][n_expert], at most kRouteFloats)
    int n_expert;
    int64_t n_embd, n_ff;
    int n_local, expert_base, k, n_tok, tile_m, cap, cap_log2;
    int *n_groups;         // null (no tensor-core experts): at most kFewRows tokens
    GemmGroup *groups;
    StreamTable *table_gu, *table_dn;
    int32_t *x_rows;       // [entries][cap]: the tokens of an entry (cap 1: the entry's own x pointer says it)
    __half *xg;            // [picks][n_embd]: gathered rows of the tensor-core experts
    float *hs;             // [entries * cap][n_ff]
    float *d;              // [picks + entries * cap][n_embd]: down projections, tensor-core rows first
    int32_t *pos;          // [n_tok][k]: a pick's row of d (-1: held elsewhere)
};

// Exclusive sum over the block's threads (whole warps); `total` is the sum of all.
__device__ __forceinline__ int block_scan(int v, int *warp_sums, int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();   // the sums of the scan before are read
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    const int w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
    int winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, winc, o);
        if (lane >= o) winc += u;
    }
    total = __shfl_sync(0xFFFFFFFFu, winc, 31);
    return inc - v + __shfl_sync(0xFFFFFFFFu, winc - w, warp);
}

// One block of at least n_local threads; thread e looks after expert e, and after the picks e, e + blockDim, ... Picks
// take places in their expert's rows through shared-memory counters; a few-row expert's picks are then put in token order
// (a row's place decides which limb columns it rides in, and with them the rounding order of its sums; a tensor-core
// row's place changes nothing). What a call of few tokens costs here is latency, so nothing is read back from global
// memory: the ids come out of the routing's shared copy, a thread's first pick stays in registers.
constexpr int kPlanIds = 1024;
__global__ void __launch_bounds__(kMaxExperts)
moe_group_plan_kernel(const __grid_constant__ GroupedParams p) {
    __shared__ int cnt[kMaxExperts], base[kMaxExperts], sid[kPlanIds], warp_sums[32];
    __shared__ union {
        float prob[kRouteFloats];
        int list[kMaxExperts * kFewRows];
    } u;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int e = threadIdx.x, n_pick = p.n_tok * p.k;
    cnt[e] = 0;
    if (p.logits) {   // a warp per token (n_pick <= kPlanIds: up to 32 tokens of up to 32 picks)
        for (int t = e >> 5; t < p.n_tok; t += blockDim.x >> 5)
            route_token(const_cast<int32_t *>(p.ids) + t * p.k, const_cast<float *>(p.wts) + t * p.k, p.logits + (int64_t)t * p.n_expert,
                        p.n_expert, p.k, u.prob + t * p.n_expert, sid + t * p.k, e & 31);
    }
    __syncthreads();
    auto local = [&](int i) {   // pick i's expert in the bank, or -1
        const int le = (p.logits ? sid[i] : p.ids[i]) - p.expert_base;
        return le >= 0 && le < p.n_local ? le : -1;
    };
    const int le0 = e < n_pick ? local(e) : -1;
    const int slot0 = le0 >= 0 ? atomicAdd(&cnt[le0], 1) : 0;
    for (int i = e + blockDim.x; i < n_pick; i += blockDim.x) {
        const int le = local(i);
        if (le >= 0) p.pos[i] = atomicAdd(&cnt[le], 1);   // its place, until the pass below
    }
    __syncthreads();
    const int m = cnt[e];
    const bool many = p.n_groups && m > kFewRows, few = m > 0 && !many;   // (ids of the caller may repeat within a token)
    const int n_ent = few ? (m + p.cap - 1) >> p.cap_log2 : 0;
    int total, many_off = 0;
    if (p.n_groups) {
        many_off = block_scan(many ? m : 0, warp_sums, total);
        const int group_off = block_scan(many ? (m + p.tile_m - 1) / p.tile_m : 0, warp_sums, total);
        if (e == 0) *p.n_groups = total;
        if (many)
            for (int g = 0; g * p.tile_m < m; g++) p.groups[group_off + g] = GemmGroup{e, many_off + g * p.tile_m, min(p.tile_m, m - g * p.tile_m)};
    }
    const int ent0 = block_scan(n_ent, warp_sums, total);
    if (e == 0) p.table_gu->n_entries = p.table_dn->n_entries = total;
    base[e] = many ? many_off : n_pick + ent0 * p.cap;
    __syncthreads();
    for (int i = e; i < n_pick; i += blockDim.x) {
        const int le = i == e ? le0 : local(i);
        if (le < 0) {
            p.pos[i] = -1;
            continue;
        }
        const int slot = i == e ? slot0 : p.pos[i], b = base[le];
        if (b < n_pick) p.pos[i] = b + slot;
        else u.list[b - n_pick + slot] = i;
    }
    __syncthreads();
    for (int i = e; i < n_pick; i += blockDim.x) {
        const int le = i == e ? le0 : local(i);
        if (le < 0 || base[le] < n_pick) continue;
        const int row0 = base[le] - n_pick, n = cnt[le], token = i / p.k;
        int rank = 0;
        for (int q = 0; q < n; q++) rank += u.list[row0 + q] < i;
        const int row = row0 + rank;
        p.pos[i] = n_pick + row;
        if (p.cap > 1) {   // (rows past the expert's last repeat it; nobody reads what they give)
            p.x_rows[row] = token;
            if (rank == n - 1)
                for (int q = row + 1; q & (p.cap - 1); q++) p.x_rows[q] = token;
        }
        if ((rank & (p.cap - 1)) == 0) {   // the first pick of an entry writes it
            const int ent = row >> p.cap_log2;
            GemvMat g, up, d;
            g.w = p.gate + (size_t)le * p.n_ff * p.rb_gate_up;
            up.w = p.up + (size_t)le * p.n_ff * p.rb_gate_up;
            g.x = up.x = p.x + (p.cap > 1 ? 0 : (int64_t)token * p.n_embd);
            g.y = up.y = p.hs + (int64_t)row * p.n_ff;   // the pair's fold writes silu(gate) * up through the gate's pointer
            g.n_out = up.n_out = p.n_ff;
            g.wt = up.wt = p.wt_gate_up;
            d.w = p.down + (size_t)le * p.n_embd * p.rb_down;
            d.x = g.y;
            d.y = p.d + (int64_t)(n_pick + row) * p.n_embd;
            d.n_out = p.n_embd;
            d.wt = p.wt_down;
            p.table_gu->mat[2 * ent] = g;
            p.table_gu->mat[2 * ent + 1] = up;
            p.table_dn->mat[ent] = d;
        }
    }
}

// The activation rows of the tensor-core experts' picks to their places as f16, rounded as the dense GEMM rounds f32
// activations. One block per pick; a token's row comes out of L2 for all picks but the first.
constexpr int kGatherThreads = 128;
__global__ void __launch_bounds__(kGatherThreads)
moe_gather_kernel(const __grid_constant__ GroupedParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int pick = blockIdx.x, row = p.pos[pick], n_pick = p.n_tok * p.k;
    if (row < 0 || row >= n_pick) return;
    const float4 *src = reinterpret_cast<const float4 *>(p.x + (int64_t)(pick / p.k) * p.n_embd);
    const int n4 = (int)(p.n_embd >> 2);
    uint2 *dst = reinterpret_cast<uint2 *>(p.xg + (int64_t)row * p.n_embd);
#pragma unroll 4
    for (int j = threadIdx.x; j < n4; j += kGatherThreads) {
        const float4 v = src[j];
        const __half2 a = __halves2half2(half_sat(v.x), half_sat(v.y)), b = __halves2half2(half_sat(v.z), half_sat(v.w));
        dst[j] = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
    }
}

} // namespace

int launch_route(int32_t *ids, float *wts, const float *logits, int64_t n_tok, int n_expert, int k,
                 cudaStream_t st) {
    if (n_expert <= 0 || n_expert > kMaxExperts || k <= 0 || k > kMaxK || k > n_expert)
        return KRK_CUDA_EARG;
    if (n_tok == 0) return KRK_CUDA_OK;
    route_kernel<<<(unsigned)n_tok, 32, 0, st>>>(ids, wts, logits, n_expert, k);
    note_launch();
    return check_launch();
}

int launch_router_softmax(float *probs, const float *logits, int64_t n_rows, int n_expert, cudaStream_t st) {
    if (n_expert <= 0 || n_expert > kMaxExperts) return KRK_CUDA_EARG;
    if (n_rows == 0) return KRK_CUDA_OK;
    router_softmax_kernel<<<(unsigned)n_rows, 32, 0, st>>>(probs, logits, n_expert);
    note_launch();
    return check_launch();
}

int launch_router_topk(const float *probs, int64_t n_rows, int n_expert, int k, int32_t *ids, float *wts, int normalize,
                       float scale, cudaStream_t st) {
    if (n_expert <= 0 || n_expert > kMaxExperts || k <= 0 || k > kMaxK || k > n_expert) return KRK_CUDA_EARG;
    if (n_rows == 0) return KRK_CUDA_OK;
    router_topk_kernel<<<(unsigned)n_rows, 32, 0, st>>>(probs, n_expert, k, ids, wts, normalize, scale);
    note_launch();
    return check_launch();
}

int launch_moe_plan_build(const int32_t *ids, int64_t n_rows, int k, int n_expert, int32_t *off, int32_t *rows, float *wt,
                          const float *wts, cudaStream_t st) {
    if (n_expert <= 0 || n_expert > kMaxExperts || k <= 0 || n_rows < 0 || n_rows * k > (1 << 24)) return KRK_CUDA_EARG;
    moe_plan_build_kernel<<<1, n_expert < 1024 ? ((n_expert + 31) / 32) * 32 : 1024, 0, st>>>(ids, (int)n_rows, k, n_expert, off, rows,
                                                                                              wt, wts);
    note_launch();
    return check_launch();
}

static size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

// n_tok <= 8: per-pick h and d rows, then the two matrix tables of the streaming path
static size_t moe_float_bytes(const krk_cuda_expert_bank *bank, int k, int64_t n_tok) {
    return up256(sizeof(float) * (size_t)(n_tok * k) * (size_t)(bank->n_ff + bank->n_embd));
}

// More than one token, shapes that the streaming kernel (and above eight tokens the tensor-core kernel) addresses: the
// workspace of launch_moe_ffn_grouped. Calls of many tokens go in chunks, so that it stays bounded: 28 KB a pick at 4096 x 1536,
// 1.84 GB for a whole chunk. (Smaller chunks would decode every expert's weights more often.)
constexpr int64_t kChunkPicks = 65536;
struct GroupedLayout {
    size_t head, groups, pos, table_gu, table_dn, x_rows, xg, h, hs, d, total;
    int64_t chunk;   // tokens per chunk
    int max_groups;
};
constexpr int kMinTileM = 32;
static GroupedLayout grouped_layout(const krk_cuda_expert_bank *bank, int k, int64_t n_tok) {
    GroupedLayout L;
    L.chunk = kChunkPicks / k < n_tok ? kChunkPicks / k : n_tok;
    const size_t picks = (size_t)(L.chunk * k);
    const bool many = n_tok > kFewRows;
    // entries and their rows, whichever rows per entry are chosen: no entry is empty, and beside tensor-core experts an
    // expert has at most kFewRows
    size_t entries = 0, rows = 0;
    for (size_t cap = 1; cap <= kFewRows; cap *= 2) {
        const size_t most = (size_t)bank->n_local * (kFewRows / cap), n = many && most < picks ? most : picks;
        entries = n > entries ? n : entries;
        rows = n * cap > rows ? n * cap : rows;
    }
    L.max_groups = many ? (int)(picks / kMinTileM) + bank->n_local : 0;
    size_t at = 0;
    auto take = [&at](size_t bytes) { const size_t o = at; at += up256(bytes); return o; };
    L.head = take(sizeof(int));
    L.groups = take(sizeof(GemmGroup) * (size_t)L.max_groups);
    L.pos = take(sizeof(int32_t) * picks);
    L.table_gu = take(stream_table_bytes(2 * entries));
    L.table_dn = take(stream_table_bytes(entries));
    L.x_rows = take(sizeof(int32_t) * rows);
    L.xg = take(many ? sizeof(__half) * picks * bank->n_embd : 0);
    L.h = take(many ? sizeof(__half) * picks * bank->n_ff : 0);
    L.hs = take(sizeof(float) * rows * bank->n_ff);
    L.d = take(sizeof(float) * ((many ? picks : 0) + rows) * bank->n_embd);
    L.total = at;
    return L;
}
static bool grouped_takes(const krk_cuda_expert_bank *bank, int64_t n_tok) {
    if (n_tok <= kFewRows && bank->n_local > kMaxExperts) return false;   // more than the plan has threads
    return n_tok > 1 && (n_tok <= kFewRows || (bank->n_embd % 256 == 0 && bank->n_ff % 256 == 0)) &&
           stream_takes(bank->wt_gate_up, bank->n_embd, kFewRows) && stream_takes(bank->wt_down, bank->n_ff, kFewRows);
}

// The other shapes: one expert after the other, the tokens of an expert as one matrix.
struct LoopLayout {
    size_t off, rows, wt, xg, g, u, dg, gemm, total;
};
// rung for a [m x n_in] . W^T product by row count: streaming / shape-agnostic GEMV up to 8 rows, tensor cores above
static size_t loop_gemm_bytes(const krk_cuda_expert_bank *bank, int64_t n_tok) {
    size_t a = 0, b = 0;
    if (bank->n_embd % 256 == 0) a = gemm_workspace_bytes(KRK_CUDA_X_F32, bank->n_ff, bank->n_embd, n_tok);
    if (bank->n_ff % 256 == 0) b = gemm_workspace_bytes(KRK_CUDA_X_F32, bank->n_embd, bank->n_ff, n_tok);
    return a > b ? a : b;
}
static LoopLayout loop_layout(const krk_cuda_expert_bank *bank, int k, int64_t n_tok) {
    LoopLayout L;
    const size_t picks = (size_t)(n_tok * k);
    size_t at = 0;
    auto take = [&at](size_t bytes) { const size_t o = at; at += up256(bytes); return o; };
    L.off = take(sizeof(int32_t) * (kMaxExperts + 1));
    L.rows = take(sizeof(int32_t) * picks);
    L.wt = take(sizeof(float) * picks);
    L.xg = take(sizeof(float) * (size_t)n_tok * bank->n_embd);
    L.g = take(sizeof(float) * (size_t)n_tok * bank->n_ff);
    L.u = take(sizeof(float) * (size_t)n_tok * bank->n_ff);
    L.dg = take(sizeof(float) * (size_t)n_tok * bank->n_embd);
    L.gemm = take(loop_gemm_bytes(bank, n_tok));
    L.total = at;
    return L;
}

size_t moe_workspace_bytes(const krk_cuda_expert_bank *bank, int k, int64_t n_tok) {
    const size_t grouped = grouped_takes(bank, n_tok) ? grouped_layout(bank, k, n_tok).total : 0;
    if (n_tok > KRK_CUDA_MAX_ROWS) return grouped ? grouped : loop_layout(bank, k, n_tok).total;
    const size_t picks = (size_t)(n_tok * k);
    const size_t by_pick = moe_float_bytes(bank, k, n_tok) + stream_table_bytes(2 * picks) + stream_table_bytes(picks);
    return grouped > by_pick ? grouped : by_pick;
}

static int launch_combine(const MoeParams &p, cudaStream_t st) {
    // tokens in x: a chunk of one pick each has 65,536 of them, and y ends at 65,535 (more columns than that are strided over)
    const int64_t n4 = p.n_embd / 4, cols = (n4 + kCombineThreads - 1) / kCombineThreads;
    return launched(launch_overlapped(moe_combine_kernel, dim3((unsigned)p.n_tok, (unsigned)(cols < 65535 ? cols : 65535)), dim3(kCombineThreads), st, p));
}

static MoeParams moe_params(float *y, const float *x, const int32_t *ids, const float *wts, const krk_cuda_expert_bank *bank, int k, int64_t n_tok) {
    MoeParams p;
    p.gate = static_cast<const uint8_t *>(bank->gate);
    p.up = static_cast<const uint8_t *>(bank->up);
    p.down = static_cast<const uint8_t *>(bank->down);
    p.x = x;
    p.ids = ids;
    p.wts = wts;
    p.h = p.d = nullptr;
    p.y = y;
    p.n_embd = bank->n_embd;
    p.n_ff = bank->n_ff;
    p.n_local = bank->n_local;
    p.expert_base = bank->expert_base;
    p.k = k;
    p.n_tok = (int)n_tok;
    p.pos = nullptr;
    p.vec = (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    return p;
}

// Few weight bytes over all picks: reading an expert again costs less than the longer preparation of four and eight rows (two
// against four, 18 MB 27.2 against 32.3 us, 28 MB 23.8 against 30.6), or than the longer plan (an entry per pick).
constexpr double kFewBytes = 64e6, kByPickBytes = 25e6;
// Rows per entry of the few-row experts, from the rows an expert can expect: two cost what one does, four and eight 1.5
// and 2.2 times.
static int entry_rows_log2(int64_t picks, int n_expert) {
    return 5 * picks < 2 * n_expert ? 0 : picks < 2 * n_expert ? 1 : picks < 5 * n_expert ? 2 : 3;
}

// Weight bytes of all picks' experts.
static double pick_bytes(const krk_cuda_expert_bank *bank, int64_t picks) {
    return (double)picks * (2.0 * bank->n_ff * row_bytes(bank->wt_gate_up, bank->n_embd) + (double)bank->n_embd * row_bytes(bank->wt_down, bank->n_ff));
}

static int moe_ffn_chunk(const GroupedLayout &L, uint8_t *ws, float *y, const float *x, const int32_t *ids, const float *wts,
                         const krk_cuda_expert_bank *bank, int k, int64_t n_tok, const float *logits, int n_expert, cudaStream_t st) {
    const bool many = L.max_groups > 0;   // some expert may go to the tensor cores
    GroupedParams p;
    p.gate = static_cast<const uint8_t *>(bank->gate);
    p.up = static_cast<const uint8_t *>(bank->up);
    p.down = static_cast<const uint8_t *>(bank->down);
    p.rb_gate_up = row_bytes(bank->wt_gate_up, bank->n_embd);
    p.rb_down = row_bytes(bank->wt_down, bank->n_ff);
    p.wt_gate_up = bank->wt_gate_up;
    p.wt_down = bank->wt_down;
    p.x = x;
    p.ids = ids;
    p.wts = wts;
    p.logits = logits;
    p.n_expert = n_expert;
    p.n_embd = bank->n_embd;
    p.n_ff = bank->n_ff;
    p.n_local = bank->n_local;
    p.expert_base = bank->expert_base;
    p.k = k;
    p.n_tok = (int)n_tok;
    // From the rows an expert can expect: the token tile (an expert's rows should fit one, since every further tile
    // decodes its weights again; up to 64 tokens two accumulators alternate), and the rows per entry of the few-row experts.
    // Over five banks of 8 to 128 experts, tiles of 128 take 1.03 of the time of tiles of 64 at 60 mean rows and 0.89 at 72;
    // tiles of 256 take 1.12 of the time of tiles of 128 at 112, 1.01 at 128 and 0.96 at 160.
    const int64_t picks = n_tok * k, mean = picks / n_expert;
    p.tile_m = mean <= 60 ? 64 : mean <= 120 ? 128 : 256;
    p.cap_log2 = entry_rows_log2(picks, n_expert);
    if (!many && p.cap_log2 > 1 && pick_bytes(bank, picks) < kFewBytes) p.cap_log2 = 1;
    p.cap = 1 << p.cap_log2;
    p.n_groups = many ? reinterpret_cast<int *>(ws + L.head) : nullptr;
    p.groups = reinterpret_cast<GemmGroup *>(ws + L.groups);
    p.pos = reinterpret_cast<int32_t *>(ws + L.pos);
    p.table_gu = reinterpret_cast<StreamTable *>(ws + L.table_gu);
    p.table_dn = reinterpret_cast<StreamTable *>(ws + L.table_dn);
    p.x_rows = reinterpret_cast<int32_t *>(ws + L.x_rows);
    p.xg = reinterpret_cast<__half *>(ws + L.xg);
    p.hs = reinterpret_cast<float *>(ws + L.hs);
    p.d = reinterpret_cast<float *>(ws + L.d);
    if (!many) p.d -= picks * p.n_embd;   // rows of d count from the picks on
    __half *h = reinterpret_cast<__half *>(ws + L.h);

    // threads: one per expert, a warp per token to route, one per pick
    int64_t threads = bank->n_local > picks ? bank->n_local : picks;
    if (logits && 32 * n_tok > threads) threads = 32 * n_tok;
    threads = threads < kMaxExperts ? (threads + 31) / 32 * 32 : kMaxExperts;
    int rc = launched(launch_overlapped(moe_group_plan_kernel, dim3(1), dim3((unsigned)threads), st, p));
    if (rc != KRK_CUDA_OK) return rc;
    ExpertGemm gu, dn;
    gu.x = p.xg;
    gu.x_rows = dn.x_rows = picks;
    gu.w = p.gate;
    gu.w_up = p.up;
    gu.bank_rows = (int64_t)bank->n_local * bank->n_ff;
    gu.wt = bank->wt_gate_up;
    gu.n_out = bank->n_ff;
    gu.n_in = bank->n_embd;
    dn.x = h;
    dn.w = p.down;
    dn.w_up = nullptr;
    dn.bank_rows = (int64_t)bank->n_local * bank->n_embd;
    dn.wt = bank->wt_down;
    dn.n_out = bank->n_embd;
    dn.n_in = bank->n_ff;
    gu.tile_m = dn.tile_m = p.tile_m;
    gu.groups = dn.groups = p.groups;
    gu.n_groups = dn.n_groups = p.n_groups;
    gu.max_groups = dn.max_groups = L.max_groups;
    StreamBanks gu_banks, dn_banks;
    gu_banks.base[0] = p.gate;
    gu_banks.base[1] = p.up;
    gu_banks.rows = gu.bank_rows;
    dn_banks.base[0] = p.down;
    dn_banks.base[1] = nullptr;
    dn_banks.rows = dn.bank_rows;
    if (many) {
        if ((rc = launched(launch_overlapped(moe_gather_kernel, dim3((unsigned)picks), dim3(kGatherThreads), st, p))) != KRK_CUDA_OK) return rc;
        if ((rc = launch_gemm_experts_gate_up(h, gu, st)) != KRK_CUDA_OK) return rc;
    }
    if ((rc = launch_gemv_stream_table(p.table_gu, p.cap > 1 ? p.x_rows : nullptr, bank->wt_gate_up, bank->n_ff, bank->n_embd, p.cap, 1, &gu_banks, st)) < 0) return rc;
    if (many && (rc = launch_gemm_experts_down(p.d, dn, st)) != KRK_CUDA_OK) return rc;
    if ((rc = launch_gemv_stream_table(p.table_dn, nullptr, bank->wt_down, bank->n_embd, bank->n_ff, p.cap, 0, &dn_banks, st)) < 0) return rc;

    MoeParams cp = moe_params(y, x, ids, wts, bank, k, n_tok);
    cp.d = p.d;
    cp.pos = p.pos;
    return launch_combine(cp, st);
}

static int launch_moe_ffn_grouped(float *y, const float *x, const int32_t *ids, const float *wts, const krk_cuda_expert_bank *bank,
                                  int k, int64_t n_tok, const float *logits, int n_expert, void *workspace, cudaStream_t st) {
    const int last = bank->expert_base + bank->n_local;   // ids at or above this are held elsewhere
    if (n_tok > kFewRows && last > kMaxExperts) return KRK_CUDA_EARG;
    const GroupedLayout L = grouped_layout(bank, k, n_tok);
    // up to a router row per warp of its block: the plan kernel routes them itself
    if (logits && (n_tok > kMaxExperts / 32 || n_tok * n_expert > kRouteFloats || n_tok * k > kPlanIds)) {
        const int rc = launch_route(const_cast<int32_t *>(ids), const_cast<float *>(wts), logits, n_tok, n_expert, k, st);
        if (rc != KRK_CUDA_OK) return rc;
        logits = nullptr;
    }
    if (n_expert < last) n_expert = last;
    if (n_expert < 1) n_expert = 1;
    for (int64_t t0 = 0; t0 < n_tok; t0 += L.chunk) {
        const int64_t n = n_tok - t0 < L.chunk ? n_tok - t0 : L.chunk;
        const int rc = moe_ffn_chunk(L, static_cast<uint8_t *>(workspace), y + t0 * bank->n_embd, x + t0 * bank->n_embd, ids + t0 * k,
                                     wts + t0 * k, bank, k, n, logits, n_expert, st);
        if (rc != KRK_CUDA_OK) return rc;
    }
    return KRK_CUDA_OK;
}

static int grouped_matmul(float *y, const float *x, const uint8_t *w, int wt, int64_t n_out, int64_t n_in, int64_t m, void *ws,
                          cudaStream_t st) {
    if (m > KRK_CUDA_MAX_ROWS && n_in % 256 == 0)
        return launch_gemm_tc(y, x, KRK_CUDA_X_F32, w, wt, n_out, n_in, m, ws, st);
    for (int64_t r0 = 0; r0 < m; r0 += KRK_CUDA_MAX_ROWS) {
        const int64_t nr = m - r0 < KRK_CUDA_MAX_ROWS ? m - r0 : KRK_CUDA_MAX_ROWS;
        GemvMat mat;
        mat.w = w;
        mat.x = x + r0 * n_in;
        mat.y = y + r0 * n_out;
        mat.n_out = n_out;
        mat.wt = wt;
        int rc = launch_gemv_stream(&mat, 1, n_in, (int)nr, 0, 0, st);
        if (rc < 0) return rc;
        if (rc == 0) rc = launch_gemv_generic(&mat, 1, n_in, (int)nr, 0, 0, st);
        if (rc != KRK_CUDA_OK && rc != 1) return rc;
    }
    return KRK_CUDA_OK;
}

// y[n_tok][n_embd] = sum over the picks this bank holds, experts in ascending id, of w * down(silu(gate x) * up x).
// One device-to-host copy of the plan's offsets (a stream synchronisation) tells the host how many rows each
// expert has, as the reference's host plan does.
static int launch_moe_ffn_loop(float *y, const float *x, const int32_t *ids, const float *wts, const krk_cuda_expert_bank *bank,
                               int k, int64_t n_tok, void *workspace, cudaStream_t st) {
    const int n_expert = bank->expert_base + bank->n_local;   // ids at or above this are held elsewhere
    if (n_expert > kMaxExperts) return KRK_CUDA_EARG;
    const LoopLayout L = loop_layout(bank, k, n_tok);
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    int32_t *off = reinterpret_cast<int32_t *>(ws + L.off), *rows = reinterpret_cast<int32_t *>(ws + L.rows);
    float *wt = reinterpret_cast<float *>(ws + L.wt), *xg = reinterpret_cast<float *>(ws + L.xg);
    float *g = reinterpret_cast<float *>(ws + L.g), *u = reinterpret_cast<float *>(ws + L.u), *dg = reinterpret_cast<float *>(ws + L.dg);
    int rc = launch_moe_plan_build(ids, n_tok, k, n_expert, off, rows, wt, wts, st);
    if (rc != KRK_CUDA_OK) return rc;
    static thread_local int32_t h_off[kMaxExperts + 1];
    cudaError_t e = cudaMemcpyAsync(h_off, off, sizeof(int32_t) * (size_t)(n_expert + 1), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaMemsetAsync(y, 0, sizeof(float) * (size_t)n_tok * bank->n_embd, st);
    if (e != cudaSuccess) {
        note_cuda_error(e);
        return KRK_CUDA_ELAUNCH;
    }
    const size_t rb_gu = row_bytes(bank->wt_gate_up, bank->n_embd), rb_dn = row_bytes(bank->wt_down, bank->n_ff);
    for (int ex = bank->expert_base; ex < n_expert; ex++) {
        const int64_t m = h_off[ex + 1] - h_off[ex];
        if (m <= 0) continue;
        const int local = ex - bank->expert_base;
        const int32_t *er = rows + h_off[ex];
        const float *ew = wt + h_off[ex];
        const uint8_t *wg = static_cast<const uint8_t *>(bank->gate) + (size_t)local * bank->n_ff * rb_gu;
        const uint8_t *wu = static_cast<const uint8_t *>(bank->up) + (size_t)local * bank->n_ff * rb_gu;
        const uint8_t *wd = static_cast<const uint8_t *>(bank->down) + (size_t)local * bank->n_embd * rb_dn;
        if ((rc = launch_gather_rows(xg, x, er, m, bank->n_embd, st)) != KRK_CUDA_OK) return rc;
        if ((rc = grouped_matmul(g, xg, wg, bank->wt_gate_up, bank->n_ff, bank->n_embd, m, ws + L.gemm, st)) != KRK_CUDA_OK) return rc;
        if ((rc = grouped_matmul(u, xg, wu, bank->wt_gate_up, bank->n_ff, bank->n_embd, m, ws + L.gemm, st)) != KRK_CUDA_OK) return rc;
        if ((rc = launch_silu_mul(g, g, u, m * bank->n_ff, st)) != KRK_CUDA_OK) return rc;
        if ((rc = grouped_matmul(dg, g, wd, bank->wt_down, bank->n_embd, bank->n_ff, m, ws + L.gemm, st)) != KRK_CUDA_OK) return rc;
        if ((rc = launch_scatter_axpy_rows(y, dg, er, ew, m, bank->n_embd, st)) != KRK_CUDA_OK) return rc;
    }
    return KRK_CUDA_OK;
}

// Widths that are not whole super-blocks and few weight bytes: the warp-per-row kernels (4 MB 13.1 us against 18.7 streaming,
// 8 MB 22.6 against 25.7, 11.6 MB 29.5 against 34.6; 14.6 MB 33.5 against 25.6).
constexpr double kOddBytes = 12e6;
int launch_moe_ffn_generic(float *y, const float *x, const int32_t *ids, const float *wts,
                           const krk_cuda_expert_bank *bank, int k, int64_t n_tok, void *workspace,
                           cudaStream_t st, const float *logits, int n_expert) {
    // `logits` set: route first (ids / wts are outputs). The streaming path folds the routing into its plan
    // kernel; every other path runs the routing kernel on its own.
    // (few picks, or so thinly spread that entries would hold one row each: an entry per pick, and the shorter plan)
    const int last = bank->expert_base + bank->n_local;
    const bool by_pick = n_tok <= KRK_CUDA_MAX_ROWS && (n_tok * k <= 8 || entry_rows_log2(n_tok * k, n_expert > last ? n_expert : last) == 0 || pick_bytes(bank, n_tok * k) < kByPickBytes);
    const bool small_odd = n_tok <= KRK_CUDA_MAX_ROWS && (bank->n_embd % 256 != 0 || bank->n_ff % 256 != 0) && pick_bytes(bank, n_tok * k) < kOddBytes;
    if (!by_pick && !small_odd && grouped_takes(bank, n_tok)) return launch_moe_ffn_grouped(y, x, ids, wts, bank, k, n_tok, logits, n_expert, workspace, st);
    bool routed = logits == nullptr;
    if (n_tok > KRK_CUDA_MAX_ROWS) {
        if (!routed) {
            const int rc = launch_route(const_cast<int32_t *>(ids), const_cast<float *>(wts), logits, n_tok, n_expert, k, st);
            if (rc != KRK_CUDA_OK) return rc;
        }
        return launch_moe_ffn_loop(y, x, ids, wts, bank, k, n_tok, workspace, st);
    }
    MoeParams p = moe_params(y, x, ids, wts, bank, k, n_tok);
    p.h = static_cast<float *>(workspace);
    p.d = p.h + (size_t)(n_tok * k) * bank->n_ff;
    const int picks = (int)(n_tok * k);
    // Streaming path: the same kernel as the dense decode GEMV, fed from device-side tables.
    // gate and up experts are rows of two stacked banks: their table launch stages weights out of one tensor map each
    StreamBanks gu_banks;
    gu_banks.base[0] = p.gate;
    gu_banks.base[1] = p.up;
    gu_banks.rows = (int64_t)bank->n_local * bank->n_ff;
    if (!small_odd && picks <= kPlanThreads && stream_takes(bank->wt_gate_up, bank->n_embd, 1) && stream_takes(bank->wt_down, bank->n_ff, 1)) {
        const bool fuse_route = !routed && n_expert <= kPlanRouteExperts && n_tok * 32 <= kPlanThreads;
        if (!routed && !fuse_route) {
            const int rc = launch_route(const_cast<int32_t *>(ids), const_cast<float *>(wts), logits, n_tok, n_expert, k, st);
            if (rc != KRK_CUDA_OK) return rc;
        }
        uint8_t *tables = static_cast<uint8_t *>(workspace) + moe_float_bytes(bank, k, n_tok);
        StreamTable *ta = reinterpret_cast<StreamTable *>(tables);
        StreamTable *tb = reinterpret_cast<StreamTable *>(tables + stream_table_bytes(2 * (size_t)picks));
        int rc = launched(launch_overlapped(moe_plan_kernel, dim3(1), dim3(kPlanThreads), st, p, ta, tb, bank->wt_gate_up, bank->wt_down,
                                            row_bytes(bank->wt_gate_up, bank->n_embd), row_bytes(bank->wt_down, bank->n_ff),
                                            fuse_route ? logits : (const float *)nullptr, n_expert));
        if (rc != KRK_CUDA_OK) return rc;
        rc = launch_gemv_stream_table(ta, nullptr, bank->wt_gate_up, bank->n_ff, bank->n_embd, 1, 1, &gu_banks, st);
        if (rc < 0) return rc;
        rc = launch_gemv_stream_table(tb, nullptr, bank->wt_down, bank->n_embd, bank->n_ff, 1, 0, nullptr, st);
        if (rc < 0) return rc;
        return launch_combine(p, st);
    }
    if (!routed) {
        const int rc = launch_route(const_cast<int32_t *>(ids), const_cast<float *>(wts), logits, n_tok, n_expert, k, st);
        if (rc != KRK_CUDA_OK) return rc;
    }
    {
        dim3 grid((unsigned)((bank->n_ff + 7) / 8), (unsigned)picks);
        KRK_DISPATCH_WT(bank->wt_gate_up, moe_gate_up_kernel<WT><<<grid, 256, 0, st>>>(p));
        note_launch();
        const int rc = check_launch();
        if (rc != KRK_CUDA_OK) return rc;
    }
    {
        dim3 grid((unsigned)((bank->n_embd + 7) / 8), (unsigned)picks);
        KRK_DISPATCH_WT(bank->wt_down, moe_down_kernel<WT><<<grid, 256, 0, st>>>(p));
        note_launch();
        const int rc = check_launch();
        if (rc != KRK_CUDA_OK) return rc;
    }
    return launch_combine(p, st);
}

} // namespace krk_cuda
