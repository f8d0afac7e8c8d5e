// Routing of the one-rank layer: device side, for the routing kernels (local_layer.cu) and for the kernel that routes by itself (local_few.cu).
#pragma once
#include "gemm_common.cuh"
#include "layer.h"
#include "local_layer.h"

namespace tmoe {
namespace detail {

constexpr int kRouteThreads = 256;
constexpr int kRouteWarps = kRouteThreads / 32;
constexpr int kDirectEntries = 4096;                                      // most entries that every block counts itself

__device__ __forceinline__ int load_expert(const void* idx, int is64, long i, int E) {
    const long long e = is64 ? reinterpret_cast<const long long*>(idx)[i] : (long long) reinterpret_cast<const int*>(idx)[i];
    return e >= 0 && e < E ? (int)e : -1;
}

// Experts of entries k0 .. k0 + 7 of token t, -1 where there is none: all loads are under way at a time
__device__ __forceinline__ void load_experts(const void* idx, int is64, long t, int K, int E, int k0, bool there, int (&e)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = there && k0 + j < K ? load_expert(idx, is64, t * K + k0 + j, E) : -1;
}

// -------------------------------------------------------------------------------------------------
// Routing.  A chunk is 256 tokens (a warp per 32); slots are ordered by (expert, 32-token group, k, lane) as in routing.cu.
// count: histograms of a chunk's entries over experts and of its tokens over their LAST expert; clears the counters of the layer.
// assign: every block adds up all chunk histograms, which gives it the segment table and its own bases, so no block waits for
// another and no scan kernel sits in between.  With few entries (kDirectEntries) every block counts all of them itself and
// clears a share of the counters: one launch instead of two.  us on the GPU, one launch / two with the gap between them (32 experts, top-8), by
// entries: 1024 6.1 / 10.8, 4096 8.8 / 12.9, 8192 10.6 / 13.3, 24008 17.2 / 14.2.  (So one launch is ahead up to 12 thousand or so; the
// line stands where the test of a call's launches has it.)
// What bounds them is a chain of latencies, so a chunk's slots and the work lists are written by different blocks, a token's indices and weights
// are requested together before anything else, and what follows from the schedule alone is computed on the host.  Before (one block after the
// other, an index and a weight at a time behind a match.any of 550 to 700 cycles, 64-bit divisions), assign, us, forward / with backward's lists:
// 32 tokens 8.4 -> 5.1 / 12.3 -> 5.7, 512 14.1 -> 8.8 / 16.1 -> 8.8, 8192 11.6 -> 8.7 / 14.5 -> 8.7, 16384 14.0 -> 9.7 / 18.5 -> 11.7.
// -------------------------------------------------------------------------------------------------
constexpr int kRouteTableBlocks = 8;                                        // where there are no lists

struct RouteArgs {
    LocalLayerPlan p;
    int* ws;
    const void* topk_idx;
    int is64;
    const float* topk_w;
    int nb1[2], nb2[2], mu_wd, nb_wd, mu_wg, nb_wg;
    int group_units;                         // units per batch
    int lag[2], head[2];                     // per direction: batches that the second GEMM is behind, tiles of the first GEMM before it in a block
    int id_bits;                             // of an expert's number, or E
};

// with blocks of kRouteThreads
__device__ __forceinline__ void clear_counters(const RouteArgs& a) {
    int4* z = reinterpret_cast<int4*>(a.ws);
    for (long i = (long)blockIdx.x * kRouteThreads + threadIdx.x; i < a.p.zero_words / 4; i += (long)gridDim.x * kRouteThreads) z[i] = make_int4(0, 0, 0, 0);
}

// largest e with base[e] <= v < base[e + 1]
__device__ __forceinline__ int find_segment(const int* base, int E, int v) {
    int lo = 0, hi = E;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (base[mid] <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The lanes that have the same number, for N numbers at a time, by votes on their bits.  (match.any takes 550 to 700 cycles where the numbers differ.)
template <int N>
__device__ __forceinline__ void match_lanes(const int (&v)[N], int bits, uint32_t (&same)[N]) {
#pragma unroll
    for (int j = 0; j < N; ++j) same[j] = 0xffffffffu;
    for (int b = 0; b < bits; ++b) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const bool one = (v[j] >> b) & 1;
            const uint32_t ones = __ballot_sync(0xffffffffu, one);
            same[j] &= one ? ones : ~ones;
        }
    }
}

// [E] entries per expert, [E + 1] tokens by their last expert, added to what is there; those of tokens below `below` also to `before`
__device__ __forceinline__ void count_entries(const RouteArgs& a, int* totals, int* before, int below) {
    const int E = a.p.E, K = a.p.K;
    for (int t = threadIdx.x; t < a.p.T; t += kRouteThreads) {
        const bool earlier = before != nullptr && t < below;
        int m = -1;
        for (int k0 = 0; k0 < K; k0 += 8) {
            int e[8];
            load_experts(a.topk_idx, a.is64, t, K, E, k0, true, e);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                m = max(m, e[j]);
                if (e[j] < 0) continue;
                atomicAdd(&totals[e[j]], 1);
                if (earlier) atomicAdd(&before[e[j]], 1);
            }
        }
        atomicAdd(&totals[E + m + 1], 1);
        if (earlier) atomicAdd(&before[E + m + 1], 1);
    }
}

// Blocks 0 .. chunks - 1 write the slots of their tokens, the others the rest of the tables and the work lists: with keep in turn forward's,
// backward's and that of the weight gradients.
template <bool DIRECT>
__device__ __forceinline__ void route_assign(const RouteArgs& a, int* sh, int (&bound)[4], int block, int blocks) {
    const int E = a.p.E, K = a.p.K, T = a.p.T, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int* seg = sh;                           // [E + 1] first slot
    int* ub = seg + E + 1;                   // [E + 1] first unit
    int* ob = ub + E + 1;                    // [E + 1] first place in the token order, by last expert
    int* cnt = ob + E + 1;                   // [warps][E] next slot
    int* lst = cnt + kRouteWarps * E;        // [warps][E + 1] next place in the token order
    int* totals = lst + kRouteWarps * (E + 1);   // [E] entries, [E + 1] tokens by their last expert: of all chunks ...
    int* before_own = totals + 2 * E + 1;        // ... and of those before this block's
    const int* last_hist = totals + E;
    int* few_word = before_own + 2 * E + 1;      // local_few.cu takes the call
    const bool own = block < a.p.chunks;
    // this thread's token: its first eight entries, requested before anything else
    const int t = own ? block * kRouteThreads + tid : T;
    int first[8];
    float first_w[8];
    load_experts(a.topk_idx, a.is64, t, K, E, 0, t < T, first);
#pragma unroll
    for (int j = 0; j < 8; ++j) first_w[j] = t < T && j < K ? a.topk_w[(long)t * K + j] : 0.f;
    for (int i = tid; i < kRouteWarps * (2 * E + 1) + 2 * (2 * E + 1); i += kRouteThreads) cnt[i] = 0;      // (and lst, totals, before_own)
    __syncthreads();
    if (DIRECT) {
        count_entries(a, totals, own ? before_own : nullptr, block * kRouteThreads);
    } else {
        // the chunks' histograms, several threads per bin
        const int* ch = a.ws + a.p.chunk_hist;
        const int* cl = a.ws + a.p.chunk_last;
        const int bins = 2 * E + 1, parts = min(8, (a.p.chunks + 7) / 8);
        for (int v = tid; v < bins * parts; v += kRouteThreads) {
            const int part = v / bins, i = v - part * bins;
            const int* h = i < E ? ch + i : cl + (i - E);
            const int cols = i < E ? E : E + 1;
            int run = 0, before = 0;
#pragma unroll 8
            for (int c = part; c < a.p.chunks; c += parts) {
                const int n = h[(long)c * cols];
                run += n;
                if (c < block) before += n;
            }
            atomicAdd(&totals[i], run);
            if (own) atomicAdd(&before_own[i], before);
        }
    }
    // of this block's tokens: entries per warp and expert, tokens per warp and last expert
    int m = -1;
    for (int k0 = 0; own && k0 < K; k0 += 8) {
        int e[8];
        if (k0 == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = first[j];
        } else {
            load_experts(a.topk_idx, a.is64, t, K, E, k0, t < T, e);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (e[j] >= 0) atomicAdd(&cnt[warp * E + e[j]], 1);
            m = max(m, e[j]);
        }
    }
    if (t < T) atomicAdd(&lst[warp * (E + 1) + m + 1], 1);
    __syncthreads();
    if (warp == 0) {
        int run_s = 0, run_u = 0, run_r = 0, hit = 0, few_units = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            const int blocks = e < E ? (totals[e] + 127) / 128 : 0;
            hit += __popc(__ballot_sync(0xffffffffu, blocks != 0));
            few_units += __reduce_add_sync(0xffffffffu, e < E ? (totals[e] + a.p.few_unit - 1) / a.p.few_unit : 0);
            int s = blocks * 128, u = (blocks + 1) / 2;
            const int s_own = s, u_own = u;
            for (int o = 1; o < 32; o <<= 1) {
                const int sv = __shfl_up_sync(0xffffffffu, s, o), uv = __shfl_up_sync(0xffffffffu, u, o);
                if (lane >= o) {
                    s += sv;
                    u += uv;
                }
            }
            if (e < E) {
                seg[e] = run_s + s - s_own;
                ub[e] = run_u + u - u_own;
            }
            run_s += __shfl_sync(0xffffffffu, s, 31);
            run_u += __shfl_sync(0xffffffffu, u, 31);
            run_r += __reduce_add_sync(0xffffffffu, e < E ? (totals[e] + BK - 1) / BK * BK : 0);
        }
        if (block == 0 && lane == 0) a.ws[a.p.meta + kMetaRows] = run_r;      // rows of whole 64-row steps
        if (lane == 0) {
            seg[E] = run_s;
            ub[E] = run_u;
            // Units beyond an expert's first, each of which takes its weights again, from L2: 1 / few_again of the experts with rows at most.  (As many of units of 64
            // rows with up to 16 rows on average.  us, general kernel / local_few.cu, 64 experts, top-4, H=7168 I=768, all tokens on four experts, where every call of 128
            // and of 256 tokens has one and three per expert: 88 / 76, 95 / 115.  The other shares: local_layer_plan.)
            *few_word = a.p.few == 1 || (a.p.few == 2 && (few_units - hit) * a.p.few_again <= hit);
        }
    }
    if (warp == 1) {
        int run = 0;
        for (int e0 = 0; e0 <= E; e0 += 32) {
            const int mine = e0 + lane <= E ? last_hist[e0 + lane] : 0;
            int v = mine;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            if (e0 + lane <= E) ob[e0 + lane] = run + v - mine;
            run += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    int* meta = a.ws + a.p.meta;
    int* slot_tk = a.ws + a.p.slot_tk;
    float* slot_w = reinterpret_cast<float*>(a.ws + a.p.slot_w);
    if (!own) {
        const int U = ub[E];
        const int helper = block - a.p.chunks, helpers = blocks - a.p.chunks;
        // ---- tables
        if (helper == 0) {
            for (int e = tid; e < E; e += kRouteThreads) a.ws[a.p.counts + e] = totals[e];
            if (tid == 0) {
                meta[kMetaUnits] = U;
                meta[kMetaSlots] = seg[E];
                meta[kMetaFew] = *few_word;
            }
        }
        for (int e = helper; e < E; e += helpers)
            for (int s = seg[e] + totals[e] + tid; s < seg[e + 1]; s += kRouteThreads) {
                slot_tk[s] = -1;
                slot_w[s] = 0.f;
            }
        if (*few_word) return;
        // ---- work lists: the order that layer.cu's scheduler writes (see there), with units in slot order.  A batch ends where an expert does, if
        // one does within half a batch of its nominal end: an expert whose units are split over two batches has its weights read from memory
        // for each of them, and every byte from memory counts against the power cap (a plain copy reaches it).  Batches of 8 units, forward +
        // backward: 8192 tokens, H=7168 I=2048, 32 experts of 8.5 units 15.37 -> 14.86 ms (the forward alone 5.65 -> 5.32 J); 8192, H=2048 I=3072,
        // 16 experts of 12.5 units 5.04 -> 4.97; experts of three units, forward only (3001 tokens, H=7168) 1.98 -> 1.92.
        const int lists = a.p.keep ? 3 : 1, list = helper % lists, at0 = helper / lists, step = (helpers - list + lists - 1) / lists;
        if (list < 2) {
            const int dir = list;
            const int SG = a.group_units, NG = (U + SG - 1) / SG;
            auto first_unit = [&](int g) {
                const long v = (long)max(g, 0) * SG;
                if (v >= U) return U;
                const int e = find_segment(ub, E, (int)v), before = (int)v - ub[e], behind = ub[e + 1] - (int)v;
                if (before <= behind) return 2 * before <= SG ? ub[e] : (int)v;
                return 2 * behind < SG ? ub[e + 1] : (int)v;
            };
            int4* work = reinterpret_cast<int4*>(a.ws + a.p.work[dir]);
            const int cap = a.p.work_cap[dir], nb1 = a.nb1[dir], nb2 = a.nb2[dir], lg = a.lag[dir];
            // block g of the list: the first `head` tiles of batch g's first GEMM, the second GEMM of batch g - lg, the rest of the first
            struct Part { int u0, units; };
            auto emit = [&](int pos, int kind, const Part& p, int r) {
                const int n_blk = r / p.units, u = p.u0 + (r - n_blk * p.units);
                const int e = find_segment(ub, E, u);
                const int blk0 = seg[e] / 128 + 2 * (u - ub[e]);
                const int two = (blk0 + 1) * 128 < seg[e + 1] ? 1 : 0;
                // rows that have to be in place; backward, whole 64-row steps of K of the weight gradients
                const int end = seg[e] + (dir == 1 ? (totals[e] + BK - 1) / BK * BK : totals[e]);
                const int need0 = max(0, min(128, end - blk0 * 128)), need1 = two ? max(0, min(128, end - (blk0 + 1) * 128)) : 0;
                // rows of zeros among them, in the last unit of an expert
                const int pad = (dir == 1 && (blk0 + 2) * 128 >= end) ? end - seg[e] - totals[e] : 0;
                if (pos < cap) work[pos] = make_int4(kind | (two << 4) | (e << 8) | (pad << 24), u, n_blk | (need0 << 16) | (need1 << 24), blk0);
            };
            for (int g = at0; g < NG + lg && NG > 0; g += step) {
                // first units of batches g and g - lg, and of the ones behind them
                if (tid < 4) bound[tid] = first_unit(g + (tid & 1) - (tid >= 2 ? lg : 0));
                __syncthreads();
                const Part p1{bound[0], bound[1] - bound[0]}, p2{bound[2], g >= lg ? bound[3] - bound[2] : 0};
                __syncthreads();
                const int off = p1.u0 * nb1 + p2.u0 * nb2, n1 = p1.units * nb1, n2 = p2.units * nb2, head = min(n1, a.head[dir]);
                for (int i = tid; i < n1 + n2; i += kRouteThreads) {
                    if (i < head) emit(off + i, kWorkGemm1, p1, i);
                    else if (i < head + n2) emit(off + i, kWorkGemm2, p2, i - head);
                    else emit(off + i, kWorkGemm1, p1, i - n2);
                }
            }
            if (at0 == 0 && tid == 0) {
                const int wgrads = dir == 1 ? E * (a.mu_wd * a.nb_wd + a.mu_wg * a.nb_wg) : 0;
                meta[kMetaWork + dir] = min(U * (nb1 + nb2) + wgrads, cap);
            }
        } else {
            int4* work = reinterpret_cast<int4*>(a.ws + a.p.work[1]);
            const int cap = a.p.work_cap[1], items = U * (a.nb1[1] + a.nb2[1]);      // (of the two GEMMs, which come before)
            const int per_wd = a.mu_wd * a.nb_wd, per_e = per_wd + a.mu_wg * a.nb_wg;
            for (int i = at0 * kRouteThreads + tid; i < E * per_e; i += step * kRouteThreads) {
                const bool down = i < E * per_wd;
                const int j = down ? i : i - E * per_wd, per = down ? per_wd : per_e - per_wd, nb = down ? a.nb_wd : a.nb_wg;
                const int e = j / per, r = j - e * per, m_blk = r / nb;
                if (items + i < cap)
                    work[items + i] = make_int4((down ? kWorkWgradDown : kWorkWgradGateup) | (e << 8), seg[e], (r - m_blk * nb) | (m_blk << 16),
                                         (totals[e] + UK - 1) / UK);       // (in 16 rows: padding adds nothing)
            }
        }
        return;
    }
    // ---- slots of this chunk's entries, places of its tokens in the token order
    for (int i = tid; i < 2 * E + 1; i += kRouteThreads) {
        const bool slots = i < E;
        const int e = slots ? i : i - E, cols = slots ? E : E + 1;
        int run = (slots ? seg[e] : ob[e]) + before_own[i];
        int* w = slots ? cnt : lst;
        for (int v = 0; v < kRouteWarps; ++v) {
            const int n = w[v * cols + e];
            w[v * cols + e] = run;
            run += n;
        }
    }
    __syncthreads();
    const uint32_t before = (1u << lane) - 1u;
    int* my = cnt + warp * E;
    long place = 0;
    {
        const int bucket[1] = {m + 1};
        uint32_t same[1];
        match_lanes(bucket, a.id_bits, same);
        const uint32_t earlier = same[0] & __ballot_sync(0xffffffffu, t < T) & before;
        if (t < T) {
            place = lst[warp * (E + 1) + m + 1] + __popc(earlier);
            a.ws[a.p.token_order + place] = t;
        }
    }
    for (int k0 = 0; k0 < K; k0 += 8) {
        int e8[8], id[8];
        float w8[8];
        uint32_t same[8];
        if (k0 == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                e8[j] = first[j];
                w8[j] = first_w[j];
            }
        } else {
            load_experts(a.topk_idx, a.is64, t, K, E, k0, t < T, e8);
#pragma unroll
            for (int j = 0; j < 8; ++j) w8[j] = t < T && k0 + j < K ? a.topk_w[(long)t * K + k0 + j] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) id[j] = e8[j] < 0 ? E : e8[j];
        match_lanes(id, a.id_bits, same);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j >= K) break;
            const int e = e8[j];
            int slot = -1;
            if (e >= 0) {
                slot = my[e] + __popc(same[j] & before);
                slot_tk[slot] = t * K + k0 + j;
                slot_w[slot] = w8[j];
            }
            __syncwarp();
            if (e >= 0 && (same[j] & before) == 0) my[e] += __popc(same[j]);
            __syncwarp();
            if (t < T) a.ws[a.p.order_slot + place * K + k0 + j] = slot;
        }
    }
}

// where route_assign leaves the entries per expert in its shared memory
__host__ __device__ constexpr int route_totals(int E) { return 3 * (E + 1) + kRouteWarps * (2 * E + 1); }
// ints of shared memory that it wants
__host__ __device__ constexpr int route_words(int E) { return 3 * (E + 1) + (kRouteWarps + 2) * (2 * E + 1) + 1; }

}  // namespace detail

detail::RouteArgs local_route_args(const LocalLayerParams& q);      // (local_layer.cu)

}  // namespace tmoe
