// Un-fused dispatch / combine on one rank, see local.h.
//
//   local_route     counts per expert and the row of every token: up to 1024 tokens one block, up to 128 K entries a cluster of eight that add up
//                   each other's counts, neither of which needs cleared counters; above, a memset and one block per 128 tokens, of which the
//                   last to finish scans the chunks
//   local_dispatch  rows, expert ids and weights of the tokens that go anywhere, in token order
//   local_move      the repeat of a dispatch with a known layout, and the combine
//
// All are bound by memory traffic: every row is read once and written once.  A warp moves 2 KB of a row (four 16-byte loads in
// flight per lane), so that a few hundred rows already fill the SMs.  Through the symmetric arena the same dispatch took a
// push into the arena, a copy out of it, nine table copies and two waits of the host.  Measured through the API, hidden 7168,
// top-8, 32 experts: layout + dispatch + combine + cached dispatch + combine with weights at 4096 tokens 1216 -> 96 us (77 launches
// before), layout + FP8 dispatch + combine at 1003 tokens 736 -> 42 us.
// The latter is host work: four allocations and four launches, and the wait for the counts, for which the host watches the pinned
// words that the route kernel writes (an event behind it was seen a few microseconds later).
#include "local.h"

#include <cooperative_groups.h>

#include "ptx.cuh"

namespace tmoe {

namespace {

constexpr uint32_t kSegBytes = 2048;
constexpr int kLocalOneBlock = 1024;     // most tokens that one block routes
constexpr int kLocalCluster = 8;         // blocks that route more,
constexpr long kLocalClusterEntries = 128 * 1024;   // and most entries that they do
static_assert(kLocalOneBlock == 1024, "a warp adds up the counts of 32 warps");

struct Parts {
    LocalPart p[kLocalMaxParts];
    int n;
    int segs[kLocalMaxParts];
    int total_segs;
};

__device__ __forceinline__ long long load_entry(const void* idx, int is64, long i) {
    return is64 ? reinterpret_cast<const long long*>(idx)[i] : (long long) reinterpret_cast<const int*>(idx)[i];
}

// A count for the host, with the number of the call in the upper half: every word says by itself whether it is there, so the kernel
// ends without a fence over the bus (2 us with one and a flag behind it).
__device__ __forceinline__ void publish(volatile unsigned long long* word, int seq, int count) {
    *word = ((unsigned long long)(uint32_t)seq << 32) | (uint32_t)count;
}

// counts a token's valid entries; true if there are any.  (Eight indices are on their way at a time.)
__device__ __forceinline__ bool count_token(const void* topk_idx, int is64, long t, int K, int E, int* hist) {
    bool any = false;
    for (int k0 = 0; k0 < K; k0 += 8) {
        long long e[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = k0 + j < K ? load_entry(topk_idx, is64, t * K + k0 + j) : -1;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (e[j] < 0 || e[j] >= E) continue;
            atomicAdd(&hist[(int)e[j]], 1);
            any = true;
        }
    }
    return any;
}

// Every block of the cluster takes a run of chunks, eight at a time, and keeps its counts; then each reads what the others have.  With more
// entries (local_route_many_kernel) counters in memory are cleared by a memset and added to by a block per chunk: two more steps of the stream, each
// of which takes 2 us and more however little is done in it.  us of layout + dispatch through the API, so / here: 2000 tokens, top-8, 32 experts 50.5 / 41.0,
// 4096 49.8 / 41.5, 16384, 256 experts 52.3 / 50.1 (the kernel 8.5 / 11.6, an atomic per entry in few SMs); 100000, 32 experts 73 / 126.
__global__ void __cluster_dims__(kLocalCluster, 1, 1) __launch_bounds__(kLocalOneBlock)
local_route_kernel(const void* topk_idx, int is64, int T, int K, int E, int* totals, int* row_local, int* chunk_base, uint8_t* in_rank,
                   unsigned long long* host_out, int host_seq) {
    extern __shared__ int hist[];
    __shared__ int warp_rows[kLocalOneBlock / 32];
    __shared__ int rows_here;
    constexpr int kChunkWarps = kLocalChunk / 32, kAtATime = kLocalOneBlock / kLocalChunk;
    const auto cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, first = warp / kChunkWarps * kChunkWarps, rank = (int)cluster.block_rank();
    const int chunks = (T + kLocalChunk - 1) / kLocalChunk, share = (chunks + kLocalCluster - 1) / kLocalCluster;
    const int begin = min(rank * share, chunks), end = min(begin + share, chunks);
    for (int e = tid; e < E; e += kLocalOneBlock) hist[e] = 0;
    __syncthreads();
    int run = 0;
    for (int c0 = begin; c0 < end; c0 += kAtATime) {
        const int chunk = c0 + warp / kChunkWarps, t = chunk * kLocalChunk + (tid & (kLocalChunk - 1));
        const bool live = chunk < end && t < T;
        const bool any = live && count_token(topk_idx, is64, t, K, E, hist);
        if (live && in_rank != nullptr) in_rank[t] = any ? 1 : 0;
        const uint32_t b = __ballot_sync(0xffffffffu, any);
        if (lane == 0) warp_rows[warp] = __popc(b);
        __syncthreads();
        const int own = warp_rows[lane];
        const int earlier = __reduce_add_sync(0xffffffffu, lane < first ? own : 0);
        const int before = __reduce_add_sync(0xffffffffu, lane >= first && lane < warp ? own : 0);
        const int rows = __reduce_add_sync(0xffffffffu, own);
        if (live) row_local[t] = any ? before + __popc(b & ((1u << lane) - 1u)) : -1;
        if (chunk < end && warp == first && lane == 0) chunk_base[chunk] = run + earlier;
        run += rows;
        __syncthreads();
    }
    if (tid == 0) rows_here = run;
    cluster.sync();
    int base = 0, all = 0;
#pragma unroll
    for (int j = 0; j < kLocalCluster; ++j) {
        const int n = *cluster.map_shared_rank(&rows_here, j);
        if (j < rank) base += n;
        all += n;
    }
    if (base != 0)
        for (int c = begin + tid; c < end; c += kLocalOneBlock) chunk_base[c] += base;
    for (int e = rank * kLocalOneBlock + tid; e < E; e += kLocalCluster * kLocalOneBlock) {
        int n = 0;
#pragma unroll
        for (int j = 0; j < kLocalCluster; ++j) n += cluster.map_shared_rank(hist, j)[e];
        totals[e] = n;
        if (host_out != nullptr) publish(host_out + 1 + e, host_seq, n);
    }
    if (rank == 0 && tid == 0) {
        totals[E] = all;
        if (host_out != nullptr) publish(host_out, host_seq, all);
    }
    cluster.sync();                          // (no block may end while another reads its counts)
}

__global__ void __launch_bounds__(kLocalChunk)
local_route_many_kernel(const void* topk_idx, int is64, int T, int K, int E, int* totals, int* row_local, int* chunk_base, uint8_t* in_rank,
                        unsigned long long* host_out, int host_seq) {
    extern __shared__ int hist[];
    __shared__ int warp_rows[kLocalChunk / 32];
    __shared__ int last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < E; e += kLocalChunk) hist[e] = 0;
    __syncthreads();
    const int t = blockIdx.x * kLocalChunk + tid;
    const bool any = t < T && count_token(topk_idx, is64, t, K, E, hist);
    if (t < T && in_rank != nullptr) in_rank[t] = any ? 1 : 0;
    const uint32_t b = __ballot_sync(0xffffffffu, any);
    if (lane == 0) warp_rows[warp] = __popc(b);
    __syncthreads();
    int before = 0, rows = 0;
    for (int w = 0; w < kLocalChunk / 32; ++w) {
        if (w < warp) before += warp_rows[w];
        rows += warp_rows[w];
    }
    if (t < T) row_local[t] = any ? before + __popc(b & ((1u << lane) - 1u)) : -1;
    for (int e = tid; e < E; e += kLocalChunk)
        if (hist[e] != 0) atomicAdd(totals + e, hist[e]);
    if (tid == 0) {
        chunk_base[blockIdx.x] = rows;
        atomicAdd(totals + E, rows);
    }
    // the last block to arrive sees every count: it turns the chunk counts into chunk bases
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(totals + E + 1, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (warp == 0) {
        int run = 0;
        for (int c0 = 0; c0 < (int)gridDim.x; c0 += 32) {
            const int c = c0 + lane;
            const int v = c < (int)gridDim.x ? __ldcg(chunk_base + c) : 0;
            int incl = v;
            for (int s = 1; s < 32; s <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, s);
                if (lane >= s) incl += u;
            }
            if (c < (int)gridDim.x) chunk_base[c] = run + incl - v;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    if (host_out != nullptr) {
        if (tid == 0) publish(host_out, host_seq, __ldcg(totals + E));
        for (int e = tid; e < E; e += kLocalChunk) publish(host_out + 1 + e, host_seq, __ldcg(totals + e));
    }
}

__global__ void __launch_bounds__(kLocalOneBlock)
local_route_small_kernel(const void* topk_idx, int is64, int T, int K, int E, int* totals, int* row_local, int* chunk_base, uint8_t* in_rank,
                         unsigned long long* host_out, int host_seq) {
    extern __shared__ int hist[];
    __shared__ int warp_rows[kLocalOneBlock / 32];
    constexpr int kChunkWarps = kLocalChunk / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, first = warp / kChunkWarps * kChunkWarps;
    for (int e = t; e < E; e += kLocalOneBlock) hist[e] = 0;
    __syncthreads();
    const bool any = t < T && count_token(topk_idx, is64, t, K, E, hist);
    if (t < T && in_rank != nullptr) in_rank[t] = any ? 1 : 0;
    const uint32_t b = __ballot_sync(0xffffffffu, any);
    if (lane == 0) warp_rows[warp] = __popc(b);
    __syncthreads();
    // rows of the warps before this one: of its chunk, and of the chunks before
    const int own = warp_rows[lane];
    const int chunks = __reduce_add_sync(0xffffffffu, lane < first ? own : 0);
    const int before = __reduce_add_sync(0xffffffffu, lane >= first && lane < warp ? own : 0);
    const int rows = __reduce_add_sync(0xffffffffu, own);
    if (t < T) {
        row_local[t] = any ? before + __popc(b & ((1u << lane) - 1u)) : -1;
        if (t % kLocalChunk == 0) chunk_base[t / kLocalChunk] = chunks;
    }
    for (int e = t; e < E; e += kLocalOneBlock) {
        totals[e] = hist[e];
        if (host_out != nullptr) publish(host_out + 1 + e, host_seq, hist[e]);
    }
    if (t == 0) {
        totals[E] = rows;
        if (T == 0) chunk_base[0] = 0;
        if (host_out != nullptr) publish(host_out, host_seq, rows);
    }
}

// up to kSegBytes of one row, by one warp; src == nullptr writes zeros
__device__ __forceinline__ void move_segment(uint8_t* dst, const uint8_t* src, uint32_t bytes, int lane) {
    const uintptr_t align = (reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src) | bytes) & 15u;
    if (align == 0) {
        const int nvec = (int)(bytes / 16);
        int4* d = reinterpret_cast<int4*>(dst);
        const int4* s = reinterpret_cast<const int4*>(src);
        int4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = make_int4(0, 0, 0, 0);
            if (src != nullptr && lane + 32 * i < nvec) v[i] = ld_nc_v4(s + lane + 32 * i);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (lane + 32 * i < nvec) d[lane + 32 * i] = v[i];
    } else {
        for (uint32_t i = lane; i < bytes; i += 32) dst[i] = src != nullptr ? src[i] : (uint8_t)0;
    }
}

__device__ __forceinline__ void move_row_segment(const Parts& ps, int seg, long dst_row, long src_row, int lane) {
    int i = 0;
    if (ps.n > 1 && seg >= ps.segs[0]) {
        seg -= ps.segs[0];
        i = 1;
    }
    const LocalPart& p = ps.p[i];
    const uint32_t off = (uint32_t)seg * kSegBytes;
    const uint32_t bytes = min(kSegBytes, p.row_bytes - off);
    const uint8_t* src = src_row < 0 ? nullptr : static_cast<const uint8_t*>(p.src) + (size_t)src_row * p.row_bytes + off;
    move_segment(static_cast<uint8_t*>(p.dst) + (size_t)dst_row * p.row_bytes + off, src, bytes, lane);
}

__global__ void __launch_bounds__(256)
local_dispatch_kernel(const __grid_constant__ Parts ps, const void* topk_idx, int is64, const float* topk_w, int T, int K, int E,
                      const int* totals, const int* row_local, const int* chunk_base, int* send_row, void* recv_idx, float* recv_w,
                      int worst_rows) {
    const int lane = threadIdx.x & 31;
    const long warps = (long)gridDim.x * (blockDim.x >> 5);
    const int filled = worst_rows > 0 ? min(totals[E], worst_rows) : 0;
    const long work = (long)(T + (worst_rows > 0 ? worst_rows - filled : 0)) * ps.total_segs;
    for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < work; i += warps) {
        const long t = i / ps.total_segs;
        const int seg = (int)(i - t * ps.total_segs);
        long row, src = t;
        if (t < T) {
            const int r = row_local[t];
            row = r >= 0 ? (long)chunk_base[t / kLocalChunk] + r : -1;
            if (seg == 0 && lane == 0) send_row[t] = (int)row;
            if (row < 0) continue;
        } else {
            row = filled + (t - T);
            src = -1;
        }
        move_row_segment(ps, seg, row, src, lane);
        if (seg == 0 && lane < K) {
            long long e = -1;
            if (src >= 0) e = load_entry(topk_idx, is64, t * K + lane);
            if (e >= E) e = -1;
            if (is64) static_cast<long long*>(recv_idx)[row * K + lane] = e < 0 ? -1 : e;
            else static_cast<int*>(recv_idx)[row * K + lane] = e < 0 ? -1 : (int)e;
            recv_w[row * K + lane] = e < 0 ? 0.f : topk_w[t * K + lane];
        }
    }
}

__global__ void __launch_bounds__(256)
local_move_kernel(const __grid_constant__ Parts ps, const int* send_row, int T, long rows, int to_rows, const void* topk_idx, int is64, int K, int E,
                  const float* weights, float* weights_out) {
    const int lane = threadIdx.x & 31;
    const long warps = (long)gridDim.x * (blockDim.x >> 5);
    const long work = (long)T * ps.total_segs;
    for (long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < work; i += warps) {
        const long t = i / ps.total_segs;
        const int seg = (int)(i - t * ps.total_segs);
        const int sent = send_row[t];
        const long row = sent < rows ? sent : -1;
        if (to_rows) {
            if (row >= 0) move_row_segment(ps, seg, row, t, lane);
            continue;
        }
        move_row_segment(ps, seg, t, row, lane);
        if (weights != nullptr && seg == 0 && lane < K) {
            const long long e = load_entry(topk_idx, is64, t * K + lane);
            weights_out[t * K + lane] = (row >= 0 && e >= 0 && e < E) ? weights[row * K + lane] : 0.f;
        }
    }
}

bool make_parts(const LocalPart* parts, int n, Parts& ps) {
    if (n < 1 || n > kLocalMaxParts) return false;
    ps.n = n;
    ps.total_segs = 0;
    for (int i = 0; i < n; ++i) {
        if (parts[i].row_bytes == 0) return false;
        ps.p[i] = parts[i];
        ps.segs[i] = (int)((parts[i].row_bytes + kSegBytes - 1) / kSegBytes);
        ps.total_segs += ps.segs[i];
    }
    return true;
}

// A block per eight segments, up to 16 blocks for each of a B200's 148 SMs, with more than `many` segments 64; warps stride over the rest.  us by blocks per
// SM: 16384 rows of 14 KB (115 K segments), repeat of a dispatch 2 78.6, 4 76.2, 8 79.0, 16 77.7, 32 74.0, 64 72.6, dispatch 16 74.1, 64 72.5, with FP8 rows and
// scales (82 K) 16 40.3, 64 41.6; 10000 rows (70 K), repeat 16 47.4, 64 45.2; combine with weights at 4096 rows (29 K) 2 23.1, 4 16.7, 8 16.4, 16 15.4, 64
// 16.5.  Segments of 1 and 4 KB, or 32 bytes per lane and load, are slower (dispatch + repeat at 4096 rows 38.5; 1 KB 40.0, 4 KB 45.4, 32 bytes 40.6).
int move_grid(long rows, int segs, long many) {
    const long most = 148 * (rows * segs > many ? 64 : 16), blocks = (rows * segs + 7) / 8;
    return (int)(blocks < 1 ? 1 : blocks > most ? most : blocks);
}

}  // namespace

cudaError_t local_route(const void* topk_idx, int is64, int T, int K, int E, int* totals, int* row_local, int* chunk_base, uint8_t* in_rank,
                        unsigned long long* host_out, int host_seq, cudaStream_t stream) {
    const size_t smem = (size_t)E * sizeof(int);
    if (E < 1 || smem > 40 * 1024) return cudaErrorInvalidValue;
    if (T <= kLocalOneBlock) {
        local_route_small_kernel<<<1, kLocalOneBlock, smem, stream>>>(topk_idx, is64, T, K, E, totals, row_local, chunk_base, in_rank, host_out, host_seq);
        return cudaGetLastError();
    }
    if ((long)T * K <= kLocalClusterEntries) {
        local_route_kernel<<<kLocalCluster, kLocalOneBlock, smem, stream>>>(topk_idx, is64, T, K, E, totals, row_local, chunk_base, in_rank, host_out, host_seq);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(totals, 0, (size_t)(E + 2) * sizeof(int), stream);
    if (e != cudaSuccess) return e;
    const int chunks = (T + kLocalChunk - 1) / kLocalChunk;
    local_route_many_kernel<<<chunks, kLocalChunk, smem, stream>>>(topk_idx, is64, T, K, E, totals, row_local, chunk_base, in_rank, host_out, host_seq);
    return cudaGetLastError();
}

cudaError_t local_dispatch(const LocalPart* parts, int num_parts, const void* topk_idx, int is64, const float* topk_w, int T, int K, int E,
                           const int* totals, const int* row_local, const int* chunk_base, int* send_row, void* recv_idx, float* recv_w,
                           int worst_rows, cudaStream_t stream) {
    Parts ps{};
    if (!make_parts(parts, num_parts, ps) || K > 32) return cudaErrorInvalidValue;
    const long rows = T > worst_rows ? T : worst_rows;
    if (rows == 0) return cudaSuccess;
    local_dispatch_kernel<<<move_grid(rows, ps.total_segs, 96 * 1024), 256, 0, stream>>>(ps, topk_idx, is64, topk_w, T, K, E, totals, row_local, chunk_base,
                                                                             send_row, recv_idx, recv_w, worst_rows);
    return cudaGetLastError();
}

cudaError_t local_move(const LocalPart* parts, int num_parts, const int* send_row, int T, long rows, int to_rows, const void* topk_idx, int is64, int K,
                       int E, const float* weights, float* weights_out, cudaStream_t stream) {
    Parts ps{};
    if (!make_parts(parts, num_parts, ps) || K > 32) return cudaErrorInvalidValue;
    if (T == 0) return cudaSuccess;
    local_move_kernel<<<move_grid(T, ps.total_segs, 64 * 1024), 256, 0, stream>>>(ps, send_row, T, rows, to_rows, topk_idx, is64, K, E, weights, weights_out);
    return cudaGetLastError();
}

}  // namespace tmoe
