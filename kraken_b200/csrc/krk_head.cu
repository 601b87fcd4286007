// The two steps either side of the output-head GEMV: the embedding gather before the first layer and the
// top-k of the logits row after the head, both on the device so that neither token rows nor the 513 KB
// logits row cross PCIe per token.
//
// embed: out[t] = decoded row tokens[t] of the (quantized) embedding table; an id outside [0, n_vocab)
// gives a zero row (src/backend_cpu.cpp:746-778). Bit-exact with the host decoders.
//
// logits_topk: Backend::logits_topk (include/krk/backend.hpp:902-922; CPU twin src/backend_cpu.cpp:862-912):
// key(i) = logits[i], clamped to +-softcap when softcap > 0, then divided (positive) or multiplied
// (negative) by rep_pen where the token's bit is set in pen_mask; the k largest keys in descending order,
// ties toward the lower id; ids past the row's length are -1 / -FLT_MAX; mass = sum over the whole row of
// exp((key - max) / temp). Two kernels. The first is a radix select: up to four passes over 8-bit digits of the
// order-preserving integer form of the keys find the k-th largest (as soon as a digit decides, no further), everything above it (and the
// lowest ids among its equals) is collected. Every block selects from its 2048-key slice of the row and leaves the slice's (max, sum
// of exp). The one block of the second kernel ranks what of the slices' candidates is above a bound (see rank_select; the radix select
// again where many keys are equal or there are more than 512 slices) and folds the sums. What bounds it is latency: about a dozen barriers and two passes through level 2. (Pulling the k best
// out one at a time, by warp arg-max and list merges, took 52 us at k = 40 on 128,256 logits.)
#include "krk_common.cuh"

#include <cfloat>

namespace krk_cuda {

namespace {

template <int WT>
__global__ void __launch_bounds__(256)
embed_kernel(float *__restrict__ out, const uint8_t *__restrict__ table, const int32_t *__restrict__ tokens,
             int64_t n_vocab, int64_t n_embd, int64_t n_tok, size_t rb) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t total = n_tok * n_embd;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = i / n_embd, k = i - t * n_embd;
        const int32_t id = tokens[t];
        out[i] = (id < 0 || (int64_t)id >= n_vocab) ? 0.0f : decode_value<WT>(table + (size_t)id * rb, k);
    }
}

constexpr int kTopkThreads = 512;
constexpr int kTopkMaxK = 64;
constexpr int kTopkSlice = 2048;        // keys of a block of the first kernel
constexpr int kTopkPer = kTopkSlice / kTopkThreads;
constexpr int kMergeThreads = 1024;
constexpr int kRankBlocks = 512;         // lists up to which the second kernel ranks, see rank_select
constexpr int kMergeHeld = 8192;        // candidates the second kernel keeps in shared memory

struct TopkParams {
    const float *logits;
    const uint32_t *pen_mask;
    float rep_pen, softcap, inv_temp;
    int64_t n;
    int k;
};

// A NaN key ranks last, as -infinity does.
__device__ __forceinline__ float topk_key(const TopkParams &p, int64_t i) {
    float v = p.logits[i];
    if (p.softcap > 0.0f) v = v > p.softcap ? p.softcap : (v < -p.softcap ? -p.softcap : v);
    if (p.pen_mask && p.rep_pen > 0.0f && p.rep_pen != 1.0f && ((p.pen_mask[(uint32_t)i >> 5] >> ((uint32_t)i & 31)) & 1u))
        v = v > 0.0f ? __fdiv_rn(v, p.rep_pen) : __fmul_rn(v, p.rep_pen);
    return v == v ? v : -INFINITY;
}
// Order-preserving unsigned form (both zeros alike); 0 is "nothing" and loses to every key, -infinity included.
__device__ __forceinline__ uint32_t order(float v) {
    const uint32_t b = __float_as_uint(v + 0.0f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}

constexpr int kNone = 0x7FFFFFFF;

// By a whole block: the k-th largest of the keys that `each(f)` hands to f (each thread its own; zeros are ignored), and
// how many of its equals belong to the k largest. Fewer than k keys: threshold 0, nothing taken from its equals.
// k = 1 (kGreatest): one pass and one barrier in place of four passes of three; compiled apart, since the other form
// loses 1.2 us beside the extra code (42,146 logits and their head: 34.2 -> 29.2 us at k = 1). A few (kFew): the distinct
// keys from the greatest down, each with its number, a pass and a barrier each (32,000 logits, few against radix: k = 2 7.3
// against 11.4 us, k = 6 10.4 against 11.7, k = 8 12.0 against 11.7).
enum SelectMode { kRadix, kGreatest, kFew };
constexpr int kFewK = 7;
template <SelectMode MODE, class Each>
__device__ __forceinline__ void radix_select(Each &&each, int k, uint32_t &threshold, int &of_equals) {
    __shared__ int hist[256];
    __shared__ uint32_t s_prefix;
    __shared__ int s_left, s_all;
    if constexpr (MODE == kGreatest) {
        uint32_t most = 0u;
        each([&](uint32_t u) { most = max(most, u); });
        most = __reduce_max_sync(0xFFFFFFFFu, most);
        if ((threadIdx.x & 31) == 0) hist[threadIdx.x >> 5] = (int)most;
        __syncthreads();
        const int lane = threadIdx.x & 31;
        threshold = __reduce_max_sync(0xFFFFFFFFu, lane < (int)blockDim.x / 32 ? (uint32_t)hist[lane] : 0u);
        of_equals = threshold != 0u ? 1 : 0;
        return;
    }
    if constexpr (MODE == kFew) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x / 32;
        uint32_t below = 0xFFFFFFFFu;   // (no key has this value: it would be a NaN's)
        int want = k;
        for (int pass = 0;; pass ^= 1) {
            uint32_t most = 0u;
            each([&](uint32_t u) { most = max(most, u < below ? u : 0u); });
            most = __reduce_max_sync(0xFFFFFFFFu, most);
            int same = 0;
            each([&](uint32_t u) { same += u == most; });
            same = __reduce_add_sync(0xFFFFFFFFu, same);
            // (two halves in turn: a warp may be a pass ahead of the last reader, never two)
            if (lane == 0) {
                hist[128 * pass + 2 * warp] = (int)most;
                hist[128 * pass + 2 * warp + 1] = same;
            }
            __syncthreads();
            const uint32_t m = lane < n_warps ? (uint32_t)hist[128 * pass + 2 * lane] : 0u;
            const int c = lane < n_warps ? hist[128 * pass + 2 * lane + 1] : 0;
            below = __reduce_max_sync(0xFFFFFFFFu, m);
            const int n = __reduce_add_sync(0xFFFFFFFFu, m == below ? c : 0);
            if (below == 0u || n >= want) {   // fewer than k keys, or the k-th is among these
                threshold = below;
                of_equals = below == 0u ? 0 : want;
                return;
            }
            want -= n;
        }
    }
    uint32_t prefix = 0u, mask = 0u;
    int left = k;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        each([&](uint32_t u) {
            if (u != 0u && (u & mask) == prefix) atomicAdd(&hist[(u >> shift) & 255u], 1);
        });
        __syncthreads();
        if (threadIdx.x < 32) {
            // lane l holds bins 255 - 8l .. 248 - 8l, descending; the digit is where the running count reaches `left`
            const int lane = threadIdx.x;
            int c[8], sum = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) sum += c[j] = hist[255 - 8 * lane - j];
            int above = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xFFFFFFFFu, above, o);
                if (lane >= o) above += v;
            }
            const int total = __shfl_sync(0xFFFFFFFFu, above, 31);
            above -= sum;
            if (total < left) {   // (only in the first pass: fewer keys than k)
                if (lane == 0) s_left = -1;
            } else if (above < left && above + sum >= left) {
                int j = 0;
#pragma unroll
                for (int q = 0; q < 7; q++)
                    if (j == q && above + c[q] < left) {
                        above += c[q];
                        j++;
                    }
                int in_bin = c[7];
#pragma unroll
                for (int q = 0; q < 7; q++)
                    if (j == q) in_bin = c[q];
                s_prefix = prefix | ((uint32_t)(255 - 8 * lane - j) << shift);
                s_left = left - above;
                s_all = in_bin == left - above;
            }
        }
        __syncthreads();
        left = s_left;
        if (left < 0) {
            threshold = 0u;
            of_equals = 0;
            return;
        }
        prefix = s_prefix;
        mask |= 255u << shift;
        // all of the bin belong to the k largest: the later digits do not matter (most slices, after two digits: 128,256 logits at
        // k = 40 11.8 -> 11.1 us)
        if (s_all && prefix != 0u && shift != 0) {
            threshold = prefix - 1u;
            of_equals = 0;
            return;
        }
    }
    threshold = prefix;
    of_equals = left;
}

// The selected of a block in shared memory, in no order: keys above the threshold, and of its equals the lowest ids.
struct Selected {
    uint32_t u[kTopkMaxK];
    int id[kTopkMaxK];
    int n, n_equal;
};

// cand_u / cand_i: [blocks][k] in no order; part: [blocks][2] = (slice max, slice sum of exp((key - slice max) * inv_temp))
template <SelectMode MODE>
__global__ void __launch_bounds__(kTopkThreads)
topk_slices_kernel(const __grid_constant__ TopkParams p, uint32_t *__restrict__ cand_u, int *__restrict__ cand_i,
                   float *__restrict__ part) {
    constexpr int kWarps = kTopkThreads / 32;
    __shared__ Selected sel;
    __shared__ int equal[kTopkSlice];
    __shared__ float red[kWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) sel.n = sel.n_equal = 0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t lo = (int64_t)blockIdx.x * kTopkSlice;
    const int cnt = (int)min((int64_t)kTopkSlice, p.n - lo);
    float v[kTopkPer];
    uint32_t u[kTopkPer];
#pragma unroll
    for (int j = 0; j < kTopkPer; j++) {
        const int i = j * kTopkThreads + tid;
        v[j] = i < cnt ? topk_key(p, lo + i) : -INFINITY;
        u[j] = i < cnt ? order(v[j]) : 0u;
    }
    float mx = -FLT_MAX;
#pragma unroll
    for (int j = 0; j < kTopkPer; j++) mx = fmaxf(mx, v[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    if (lane == 0) red[warp] = mx;
    uint32_t threshold;
    int of_equals;
    radix_select<MODE>([&](auto &&f) {
#pragma unroll
        for (int j = 0; j < kTopkPer; j++) f(u[j]);
    }, p.k, threshold, of_equals);   // (its barriers publish red[])
    float sum = 0.0f;
    mx = red[0];
    for (int w = 1; w < kWarps; w++) mx = fmaxf(mx, red[w]);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kTopkPer; j++)
        if (u[j] != 0u) sum += expf((v[j] - mx) * p.inv_temp);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) red[warp] = sum;
#pragma unroll
    for (int j = 0; j < kTopkPer; j++) {
        const int i = j * kTopkThreads + tid;
        if (u[j] > threshold) {
            const int at = atomicAdd(&sel.n, 1);
            sel.u[at] = u[j];
            sel.id[at] = (int)(lo + i);
        } else if (u[j] == threshold && of_equals > 0) {
            equal[atomicAdd(&sel.n_equal, 1)] = (int)(lo + i);
        }
    }
    __syncthreads();
    const int n_above = sel.n, n_equal = sel.n_equal;
    for (int i = tid; i < n_equal; i += kTopkThreads) {
        const int id = equal[i];
        int rank = i;
        if (n_equal > of_equals) {
            rank = 0;
            for (int q = 0; q < n_equal; q++) rank += equal[q] < id;
        }
        if (rank < of_equals) {
            sel.u[n_above + rank] = threshold;
            sel.id[n_above + rank] = id;
        }
    }
    __syncthreads();
    for (int i = tid; i < p.k; i += kTopkThreads) {
        const bool ok = i < n_above + of_equals;
        cand_u[(size_t)blockIdx.x * p.k + i] = ok ? sel.u[i] : 0u;
        cand_i[(size_t)blockIdx.x * p.k + i] = ok ? sel.id[i] : kNone;
    }
    if (tid == 0) {
        float s = 0.0f;
        for (int w = 0; w < kWarps; w++) s += red[w];
        part[2 * blockIdx.x] = mx;
        part[2 * blockIdx.x + 1] = s;
    }
}

// Ranks of n distinct keys among each other, eight threads to a key: f(key, rank).
template <class F>
__device__ __forceinline__ void rank_keys(const unsigned long long *keys, int n, F &&f) {
    const int part = threadIdx.x & 7;
    for (int base = 0; base < n; base += kMergeThreads / 8) {
        const int i = base + (int)(threadIdx.x >> 3);
        const unsigned long long mine = keys[min(i, n - 1)];
        int rank = 0;
#pragma unroll 4
        for (int q = part; q < n; q += 8) rank += keys[q] > mine;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) rank += __shfl_xor_sync(0xFFFFFFFFu, rank, o);
        if (part == 0 && i < n) f(mine, rank);
    }
}
// By a whole block: the k best of n_blocks lists of k keys each, without radix passes. The best few of every list, k in all at
// least, have a k-th largest, and k keys are not below that: what is below is out, and what is left, about twice k, is ranked key
// against key (ties to the lower id). False, in every thread, where more are left than the block has threads: many equal keys.
// (Candidates are all near the top, so that the radix select's first digits put them in one bin: 128,256 logits, k = 40, 16.0 -> 11.8
// us with the first kernel, k = 64 18.0 -> 12.8, 32,000 logits k = 5 10.1 -> 7.4.)
template <class EachAt>
__device__ __forceinline__ bool rank_select(EachAt &&each_at, const TopkParams &p, const uint32_t *__restrict__ cand_u, const int *__restrict__ cand_i,
                                            int n_blocks, int32_t *__restrict__ ids, float *__restrict__ vals) {
    static_assert(kTopkMaxK <= 64 && kRankBlocks + kTopkMaxK <= kMergeThreads, "two keys of a list a lane");
    __shared__ unsigned long long keys[kMergeThreads];   // a key's order, then what is the greater the lower the index or the id
    __shared__ uint32_t s_bound;
    __shared__ int s_left;
    const int tid = threadIdx.x, lane = tid & 31, k = p.k, each = (k + n_blocks - 1) / n_blocks;
    if (tid == 0) s_left = 0;
    for (int b = tid >> 5; b < n_blocks; b += kMergeThreads / 32) {
        const uint32_t *list = cand_u + (size_t)b * k;
        uint32_t u0 = lane < k ? list[lane] : 0u, u1 = lane + 32 < k ? list[lane + 32] : 0u;
        for (int r = 0; r < each; r++) {
            const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, max(u0, u1));
            const bool first = lane == __ffs(__ballot_sync(0xFFFFFFFFu, u0 == most || u1 == most)) - 1;   // one of equals
            const int at = b * each + r;
            if (lane == 0) keys[at] = (unsigned long long)most << 32 | (uint32_t)~at;
            if (first && u0 == most) u0 = 0u;
            else if (first) u1 = 0u;
        }
    }
    __syncthreads();
    // (k of them at least, k + n_blocks - 1 at most)
    rank_keys(keys, n_blocks * each, [&](unsigned long long key, int rank) {
        if (rank == k - 1) s_bound = max((uint32_t)(key >> 32), 1u);   // (a zero is no key)
    });
    __syncthreads();
    const uint32_t bound = s_bound;
    each_at([&](uint32_t u, int64_t i) {
        if (u >= bound) {
            const int at = atomicAdd(&s_left, 1);
            if (at < kMergeThreads) keys[at] = (unsigned long long)u << 32 | (uint32_t)~cand_i[i];
        }
    });
    __syncthreads();
    const int n = s_left;
    if (n > kMergeThreads) return false;
    rank_keys(keys, n, [&](unsigned long long key, int rank) {
        if (rank < k) {
            const int id = (int)~(uint32_t)key;
            ids[rank] = id;
            vals[rank] = topk_key(p, id);
        }
    });
    if (tid >= n && tid < k) {   // fewer than k keys
        ids[tid] = -1;
        vals[tid] = -FLT_MAX;
    }
    return true;
}

template <SelectMode MODE>
__global__ void __launch_bounds__(kMergeThreads)
topk_merge_kernel(const __grid_constant__ TopkParams p, const uint32_t *__restrict__ cand_u, const int *__restrict__ cand_i,
                  const float *__restrict__ part, int n_blocks, int32_t *__restrict__ ids, float *__restrict__ vals,
                  float *__restrict__ mass_out) {
    __shared__ uint32_t held[kMergeHeld];
    __shared__ Selected sel;
    const int tid = threadIdx.x, lane = tid & 31, k = p.k;
    if (tid == 0) sel.n = 0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int64_t total = (int64_t)n_blocks * k;
    const bool in_smem = total <= kMergeHeld;
    if (in_smem)
        for (int i = tid; i < (int)total; i += kMergeThreads) held[i] = cand_u[i];
    if (mass_out && tid >= kMergeThreads - 32) {   // the last warp: the slices' sums
        float mx = -FLT_MAX;
        for (int b = lane; b < n_blocks; b += 32) mx = fmaxf(mx, part[2 * b]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        float m = 0.0f;
        for (int b = lane; b < n_blocks; b += 32)
            if (part[2 * b + 1] > 0.0f) m += part[2 * b + 1] * expf((part[2 * b] - mx) * p.inv_temp);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xFFFFFFFFu, m, o);
        if (lane == 0) *mass_out = m;
    }
    __syncthreads();
    auto each_at = [&](auto &&f) {
        for (int64_t i = tid; i < total; i += kMergeThreads) f(in_smem ? held[i] : cand_u[i], i);
    };
    if constexpr (MODE != kGreatest)
        if (n_blocks <= kRankBlocks && rank_select(each_at, p, cand_u, cand_i, n_blocks, ids, vals)) return;
    uint32_t threshold;
    int of_equals;
    radix_select<MODE>([&](auto &&f) { each_at([&](uint32_t u, int64_t) { f(u); }); }, k, threshold, of_equals);
    each_at([&](uint32_t u, int64_t i) {
        if (u > threshold) {
            const int at = atomicAdd(&sel.n, 1);
            sel.u[at] = u;
            sel.id[at] = cand_i[i];
        }
    });
    __syncthreads();
    int n_sel = sel.n;
    // the equals of the threshold, lowest ids first: one at a time, each above the one before (rarely more than one)
    int last = -1;
    for (int q = 0; q < of_equals; q++) {
        __shared__ int s_min;
        if (tid == 0) s_min = kNone;
        __syncthreads();
        int best = kNone;
        each_at([&](uint32_t u, int64_t i) {
            if (u == threshold) {
                const int id = cand_i[i];
                if (id > last) best = min(best, id);
            }
        });
        best = __reduce_min_sync(0xFFFFFFFFu, best);
        if (lane == 0 && best != kNone) atomicMin(&s_min, best);
        __syncthreads();
        last = s_min;
        if (tid == 0) {
            sel.u[n_sel] = threshold;
            sel.id[n_sel] = last;
        }
        n_sel++;
        __syncthreads();
    }
    __syncthreads();
    if (tid < k) {
        if (tid < n_sel) {
            const uint32_t u = sel.u[tid];
            const int id = sel.id[tid];
            int rank = 0;
            for (int q = 0; q < n_sel; q++) rank += sel.u[q] > u || (sel.u[q] == u && sel.id[q] < id);
            ids[rank] = id;
            vals[rank] = topk_key(p, id);
        } else {
            ids[tid] = -1;
            vals[tid] = -FLT_MAX;
        }
    }
}

int topk_blocks(int64_t n) { return (int)((n + kTopkSlice - 1) / kTopkSlice); }

} // namespace

int launch_embed(float *out, const uint8_t *table, int wt, int64_t n_vocab, int64_t n_embd, const int32_t *tokens,
                 int64_t n_tok, cudaStream_t st) {
    const int64_t total = n_tok * n_embd;
    if (total == 0) return KRK_CUDA_OK;
    const int64_t want = (total + 255) / 256;
    const int grid = (int)(want < (int64_t)sm_count() * 16 ? want : (int64_t)sm_count() * 16);
    const size_t rb = row_bytes(wt, n_embd);
    int rc = KRK_CUDA_EDTYPE;
    KRK_DISPATCH_WT(wt, rc = launched(launch_overlapped(embed_kernel<WT>, dim3((unsigned)grid), dim3(256), st, out, table, tokens, n_vocab, n_embd, n_tok, rb)));
    return rc;
}

size_t logits_topk_workspace_bytes(int64_t n, int k) {
    const size_t blocks = (size_t)topk_blocks(n);
    return blocks * (size_t)k * 8 + blocks * 8 + 256;
}

int launch_logits_topk(const float *logits, int64_t n, int k, const uint32_t *pen_mask, float rep_pen, float softcap,
                       float temp, int32_t *ids, float *vals, float *mass_out, void *workspace, cudaStream_t st) {
    if (k < 1 || k > kTopkMaxK || n < 1) return KRK_CUDA_EARG;
    if (n > INT32_MAX) return KRK_CUDA_ESHAPE;   // ids are 32-bit
    const int blocks = topk_blocks(n);
    const SelectMode mode = k == 1 ? kGreatest : k <= kFewK ? kFew : kRadix;
    uint32_t *cand_u = static_cast<uint32_t *>(workspace);
    int *cand_i = reinterpret_cast<int *>(cand_u + (size_t)blocks * k);
    float *part = reinterpret_cast<float *>(cand_i + (size_t)blocks * k);
    TopkParams p;
    p.logits = logits;
    p.pen_mask = pen_mask;
    p.rep_pen = rep_pen;
    p.softcap = softcap;
    p.inv_temp = temp > 0.0f ? 1.0f / temp : 1.0f;
    p.n = n;
    p.k = k;
    int rc = launched(launch_overlapped(mode == kGreatest ? topk_slices_kernel<kGreatest> : mode == kFew ? topk_slices_kernel<kFew> : topk_slices_kernel<kRadix>, dim3((unsigned)blocks), dim3(kTopkThreads), st, p, cand_u, cand_i, part));
    if (rc != KRK_CUDA_OK) return rc;
    return launched(launch_overlapped(mode == kGreatest ? topk_merge_kernel<kGreatest> : mode == kFew ? topk_merge_kernel<kFew> : topk_merge_kernel<kRadix>, dim3(1), dim3(kMergeThreads), st, p, cand_u, cand_i, part, blocks, ids, vals, mass_out));
}

} // namespace krk_cuda
