// The MoE layer on one rank, see local_layer.h.  Roles of the persistent kernel (74 CTA pairs, 16 warps per CTA):
//
//   producer   claims items of the work list, hands them to the pair, loads operand tiles by TMA
//   issuer     tcgen05 cta_group::2, 256x256 or 256x512 tiles (128 rows for a unit of one block), two accumulators in tensor memory
//   loaders    4 warps: bring the operands that are made of token rows from the caller's tensor (load_rows).  An instance of the kernel
//              has none: there all warps but the first two copy rows into slot order (copy role), and the producer loads them
//   epilogue   8 warps: SwiGLU / dSwiGLU / store.  A warp packs 32 rows x 64 columns into shared memory (128-byte swizzle) and
//              hands them to one TMA store; the pre-activation goes straight between registers and memory (preact_at).
//   gather     warps 2 and 3, joined by the epilogue warps at the end of the list: keep a copy of x (forward), and sum every
//              token's expert rows as soon as the units that hold them are finished.
//              Tokens are visited in the order of their last expert, which is the order in which they become ready.
//
// The work list and the order of every sum are those of layer.cu, with three exceptions, none of which changes a result: batches of the list
// end where experts do (see there); K of a weight gradient ends after the 16 rows that hold the last one, as what layer.cu adds beyond is
// zeros; and a weight gradient's tiles are listed along a row of the result: the tiles in flight at a time then write whole rows (7 %
// faster where the stores bound it, 57 rows per expert).
// What is different because there is one rank: token rows are loaded or copied by slot instead of pushed by entry, expert rows stay in slot
// order (one TMA box per 32 rows instead of 32 bulk copies to landing rows), the sum of a token waits for its own units
// instead of for every rank's completion flag, counters have GPU scope, and no host read, table copy or padding kernel is
// left around the kernel.
//
// Forward + backward through the API, several-rank kernels (30 to 38 launches and one host wait per step) -> these:
//   512 tokens, H=512 I=256, 4 experts, top-2            873 ->    96 us   (was host work and launches)
//   4096, H=2048 I=2048, 16 experts, top-8              2914 ->  2206 us
//   8192, H=2048 I=3072, 16 experts, top-6              6192 ->  4780 us
//   8192, H=7168 I=2048, 32 experts, top-8             16737 -> 14385 us
//   16384, H=7168 I=512, 32 experts, top-8             10388 ->  8166 us
// Large layers are bound by the power cap: the SM clock drops to 1.0 to 1.3 GHz, and time is energy (0.86 pJ per FLOP at H=7168 I=2048, of
// which cuBLAS alone takes 0.74).
#include "local_layer.h"

#include <algorithm>
#include <type_traits>

#include "gemm_common.cuh"
#include "launch_count.h"
#include "layer.h"
#include "local_route.cuh"

namespace tmoe {

using namespace detail;

namespace {

// A stage holds 64 columns of K of a tile: this CTA's 128 rows of A and, for each 256 columns of the tile, its 128 rows of B.
// Tiles are 256 rows by 512 columns where a layer is large enough (local_layer_plan), else 256 by 256: the wide tile reads a
// quarter fewer operand bytes from L2 per FLOP, and moving operands is what the power cap leaves least for.  A launch with a
// wide GEMM has four stages of 48 KB, any other six of 32 KB: where few rows share a weight the loads come from HBM, and four
// stages of a narrow tile (1.4 us) do not cover its latency (15 to 20 % slower).
constexpr int kMaxStages = 6;
constexpr int kBHalfBytesP = (BN / 2) * BK * 2;
constexpr int kNarrowStageBytes = kAStageBytes + kBHalfBytesP;            // 32 KB
constexpr int kWideStageBytes = kAStageBytes + 2 * kBHalfBytesP;          // 48 KB
constexpr int kPipeBytesP = 6 * kNarrowStageBytes;                        // 192 KB
static_assert(kPipeBytesP == 4 * kWideStageBytes, "both divisions use the same memory");
constexpr int kBoxBytes = 32 * 128;                                       // 32 rows x 64 bf16 columns
constexpr int kEpiBytes = kEpiWarps * kBoxBytes;                          // 32 KB: one box per epilogue warp
constexpr int kBarOffsetP = kPipeBytesP + kEpiBytes;
constexpr int kSmemBytesP = kBarOffsetP + 512 + 1024;
constexpr int kCopyRows = 8;                                              // rows a gather warp claims at a time (divides a block)
constexpr int kFirstRows = 1;                                             // with copies: slots every warp copies before anything else
constexpr int kGatherWarps = 2 + kEpiWarps;                               // warps of a CTA that sum in the end
constexpr int kLoadWarps = 4;
constexpr int kLayerThreads = kThreads + 32 * kLoadWarps;
// Registers per thread: 128 at launch (512 threads), which the first warpgroup keeps
constexpr int kRegsEpilogue = 136, kRegsLoad = 112;
static_assert(128 * 128 + 256 * kRegsEpilogue + 128 * kRegsLoad <= 65536 && kThreads == 384 && kLayerThreads == 512, "register file");
constexpr int kRingDepth = 4;
constexpr int kSoon = 32;                                                 // looks at a barrier before its wait counts as one
constexpr int kOwed = 4;                                                  // finished tiles an epilogue warp counts at once
constexpr int kGatherTasks = 16384;                                       // least number of (token, columns) tasks of the gather role
constexpr uint32_t kOffTmem = 496, kOffRingFull = 320, kOffRingEmpty = 352, kOffItems = 384;
constexpr uint32_t kRingConsumers = 2 * (kEpiWarps + kLoadWarps) + 2;
static_assert(8 * (2 * kMaxStages + 4) <= (int)kOffRingFull && kOffItems + 16 * kRingDepth <= kOffTmem && kOffTmem + 8 <= 512, "barrier block");
static_assert(kSmemBytesP <= 232448, "shared memory");

// words of the sync block
enum { kSyncItem = 0, kSyncToken = 1, kSyncCopy = 2, kSyncKeep = 3, kSyncFirsts = 4, kSyncRows = 5, kSyncWords = 8 };

constexpr int kWideTiles = 74 * 4;                                        // least number of wide tiles of a GEMM (local_layer_plan)

constexpr int column_blocks(int n, int cols) { return (n + cols - 1) / cols; }

__global__ void __launch_bounds__(kRouteThreads) local_route_count_kernel(const RouteArgs a) {
    extern __shared__ int sh[];
    const int E = a.p.E, K = a.p.K, tid = threadIdx.x;
    int* hist = sh;
    int* last = sh + E;
    for (int i = tid; i < 2 * E + 1; i += kRouteThreads) sh[i] = 0;
    __syncthreads();
    const int t = blockIdx.x * kRouteThreads + tid;
    if (t < a.p.T) {
        int m = -1;
        for (int k0 = 0; k0 < K; k0 += 8) {
            int e[8];
            load_experts(a.topk_idx, a.is64, t, K, E, k0, true, e);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (e[j] >= 0) atomicAdd(&hist[e[j]], 1);
                m = max(m, e[j]);
            }
        }
        atomicAdd(&last[m + 1], 1);
    }
    __syncthreads();
    int* ch = a.ws + a.p.chunk_hist + (long)blockIdx.x * E;
    int* cl = a.ws + a.p.chunk_last + (long)blockIdx.x * (E + 1);
    for (int e = tid; e < E; e += kRouteThreads) ch[e] = hist[e];
    for (int e = tid; e <= E; e += kRouteThreads) cl[e] = last[e];
    clear_counters(a);
}

template <bool DIRECT>
__global__ void __launch_bounds__(kRouteThreads) local_route_assign_kernel(const RouteArgs a) {
    extern __shared__ int sh[];
    __shared__ int bound[4];
    if (DIRECT) clear_counters(a);
    route_assign<DIRECT>(a, sh, bound, blockIdx.x, gridDim.x);
}

// -------------------------------------------------------------------------------------------------
// The layer kernel
// -------------------------------------------------------------------------------------------------
struct Phase {
    alignas(64) CUtensorMap map_a;
    alignas(64) CUtensorMap map_b;
    alignas(64) CUtensorMap map_a32;     // the two GEMMs: 32 rows of A
    int nk, b_group_rows, cols, num_n_blocks, n_total, m_total;      // num_n_blocks: of the two GEMMs
};

struct LayerArgsP {
    Phase ph[4];
    alignas(64) CUtensorMap st_act;      // stores: [out_rows, I], [out_rows, 2I] (backward: boxes of 32 columns), [out_rows, H] and
    alignas(64) CUtensorMap st_aux;      // [E, rows, cols] of the weight gradients, in boxes of 32 rows x 64 columns
    alignas(64) CUtensorMap st_y;
    alignas(64) CUtensorMap st_dwd;
    alignas(64) CUtensorMap st_dwg;
    int T, K, H, I, E;
    int stages, stage_bytes, keep, clean, halves;
    const uint8_t* x;                    // [T, H]: forward x, backward grad_out
    const __nv_bfloat16* y;
    __nv_bfloat16* saved_x;              // [T, H]: written by forward (may be null), read by backward
    uint8_t* slot_rows;                  // without loading warps: x in slot order
    uint8_t* slot_x;                     // the same, backward: saved_x in slot order
    __nv_bfloat16* out;
    __nv_bfloat16* preact;               // forward (with keep): written, backward: read; preact_at()
    float* droute_part;
    int n_parts;
    float* dw_topk;
    const int* meta;
    const int* slot_tk;
    const float* slot_w;
    const int* token_order;              // tokens by their last expert
    const int* order_slot;               // [T, K] slots of the tokens in that order
    const int4* work;
    int max_work;
    int* sync;
    int* done1;                          // per unit: epilogue warps that finished a tile of the first GEMM
    int* done2;                          // per 128-row block: the same for the second GEMM
    int* arrived;                        // without loading warps, per 128-row block: rows of slot_rows in place
    unsigned long long* stats;
    int* status;
    int unless_few;                      // the call is local_few.cu's, whose kernel ran before, if the routing says so
};

__device__ __forceinline__ int4 ld_cg_v4_ordered(const void* p) {
    int4 v;
    // volatile keeps it behind the acquire loads that precede it; no memory clobber, so that many can be in flight
    asm volatile("ld.global.cg.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src_smem, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src_smem), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void ld_shared_v4(uint32_t addr, uint32_t (&v)[4]) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
// Warp-wide row copy with 16 loads in flight per lane (8 KB per warp): two warps per SM have to keep HBM busy.
__device__ __forceinline__ void copy_row_deep(int4* dst, const int4* src, int nvec, int lane) {
    for (int b = 0; b < nvec; b += 512) {
        int4 v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = ld_nc_v4(src + min(b + 32 * i + lane, nvec - 1));
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (b + 32 * i + lane < nvec) dst[b + 32 * i + lane] = v[i];
    }
}

template <int R>
__device__ __forceinline__ void registers_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void registers_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

struct Item {
    int kind, n0, halves, group, k0, nk, tail, m0, unit, need, real;      // columns n0 .. n0 + 256 * halves; `real` of the `need` rows are not padding; tail: 16-row slices of the last step
    bool half;          // a unit of one 128-row block, 64 of whose rows each CTA has
    int wait;           // rows of the block that have to be there
    int m_in_group;     // weight gradients: first row of dW inside the expert
};

// rows that a CTA of the pair has of an item of the two GEMMs; `real`: without those that are padding (backward, in the last block of an expert)
__device__ __forceinline__ int unit_rows(const int4& it, uint32_t rank, bool half, bool real) {
    const int two = (it.x >> 4) & 1, pad = real ? (it.x >> 24) & 63 : 0;
    if (half) return max(0, min(BM / 2, ((it.z >> 16) & 0xff) - pad - (int)rank * (BM / 2)));
    return ((it.z >> (rank == 0 ? 16 : 24)) & 0xff) - ((int)rank == two ? pad : 0);
}

__device__ __forceinline__ void decode_item(const LayerArgsP& L, const int4& it, uint32_t rank, Item& q) {
    q.kind = it.x & 15;
    q.group = (it.x >> 8) & 0xffff;
    const Phase& P = L.ph[q.kind];
    q.n0 = (it.z & 0xffff) * P.cols;
    q.halves = (P.cols > BN && q.n0 + BN < P.n_total) ? 2 : 1;
    q.half = false;
    if (q.kind <= kWorkGemm2) {
        q.unit = it.y;
        q.half = L.halves != 0 && ((it.x >> 4) & 1) == 0;
        q.wait = (it.z >> (rank == 0 || q.half ? 16 : 24)) & 0xff;
        q.need = unit_rows(it, rank, q.half, false);
        q.real = unit_rows(it, rank, q.half, true);
        q.m0 = it.w * BM + (int)rank * (q.half ? BM / 2 : BM);
        q.k0 = 0;
        q.nk = P.nk;
        q.tail = BK / UK;
        q.m_in_group = 0;
    } else {
        q.unit = -1;
        q.need = q.real = q.wait = 0;
        q.m_in_group = ((it.z >> 16) * 2 + (int)rank) * BM;
        q.m0 = q.m_in_group;
        q.k0 = it.y;
        q.nk = (it.w + BK / UK - 1) / (BK / UK);
        q.tail = it.w - (q.nk - 1) * (BK / UK);
    }
}

// Rows of A that do not exist are multiplied all the same, into rows of the accumulator that nobody reads, and what earlier items left there draws as much
// power as what counts.  So an item whose rows are fewer than those that may be left has zeros put behind them, in its first steps: as many as there are
// stages, which then stay clean.  Up to 32 rows are left as they are, so that experts of about the same size do not clean all the time.  The producers
// and the loading warps follow, each for itself, how many rows of a CTA's stages may hold something.
// Only where experts have more than 224 rows on average (LayerArgsP::clean): up to there nearly all have one unit, whose second half, if it is there at
// all, mostly takes all rows.  us, without / with, by rows per expert, forward (H=7168 I=2048, 32 experts, top-8): 100 660 / 667, 140 697 / 700, 180 743 /
// 743, 275 1251 / 1200, 525 1669 / 1614, 750 1919 / 1909; steps: 64 1960 / 1968, 140 2278 / 2237, 180 2341 / 2386, 275 3556 / 3458, H=4096 I=1536, 525
// 2192 / 2156, of 2048 rows and more 0 to 0.9 %.
struct Leftover {
    bool on;
    int rows;                                // multiple of 32
    // An item whose A is loaded in boxes, `loaded` rows (0 .. 128, a multiple of 32) in nk steps: up to which row its first steps have to write.  (Of a half
    // unit 64 rows are multiplied.)
    __device__ __forceinline__ int take_boxes(bool half, int loaded, int nk, int stages) {
        const int most = half ? min(rows, BM / 2) : rows;
        const bool need = on && most > loaded + (half ? 0 : 32);
        const int to = need ? most : loaded;
        rows = need && nk >= stages && most == rows ? loaded : max(rows, loaded);
        return to;
    }
    // An item whose A the loading warps bring, 32 rows or all, with zeros behind the `real` ones: how many steps have to write all.
    __device__ __forceinline__ int take_rows(bool half, int real, int nk, int stages) {
        if (real <= 32) {
            if (take_boxes(half, 32, nk, stages) == 32) return 0;
            if (nk >= stages) rows = 32;                     // (all 128 are written)
            return stages;
        }
        rows = nk >= stages ? (real + 31) & ~31 : BM;
        return nk;
    }
};

// Store staging of one epilogue warp: a box of 32 rows x 128 bytes, swizzled as the tensor maps expect.  One box per warp, because the
// 32 KB that a second one would take are worth more as a sixth operand stage; the wait until the store has read the box
// is hidden behind the mainloop of the next tile.
struct Staging {
    uint32_t base;      // 1024-byte aligned
    int lane;
    // 16 bytes at 16-byte column `chunk` of this lane's row
    __device__ __forceinline__ void put(int chunk, uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
        st_shared_v4(base + lane * 128 + ((chunk ^ (lane & 7)) << 4), a, b, c, d);
    }
    // The box as two of 32 rows x 64 bytes (64-byte swizzle) that are used in turn: 32 columns in one, its store in flight while
    // the other is filled.  `turn` counts the stores; a store that is not wanted still closes a group, as `reuse` counts groups.
    __device__ __forceinline__ uint32_t narrow_at(int turn, int row, int chunk) const {
        return base + (turn & 1) * (kBoxBytes / 2) + row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
    }
    __device__ __forceinline__ void put_narrow(int turn, int chunk, uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
        st_shared_v4(narrow_at(turn, lane, chunk), a, b, c, d);
    }
    __device__ __forceinline__ void store_narrow(int turn, bool wanted, const CUtensorMap* map, int c0, int c1) const {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            if (wanted) tma_store_2d(map, base + (turn & 1) * (kBoxBytes / 2), c0, c1);
            tma_store_commit();
        }
    }
    // wait until all but the last N stores of this warp have been read out of shared memory
    template <int N = 0>
    __device__ __forceinline__ void reuse() const {
        if (lane == 0) tma_store_wait_read<N>();
        __syncwarp();
    }
    __device__ __forceinline__ void store(bool wanted, const CUtensorMap* map, int c0, int c1) const {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && wanted) {
            tma_store_2d(map, base, c0, c1);
            tma_store_commit();
        }
    }
    __device__ __forceinline__ void store3(bool wanted, const CUtensorMap* map, int c0, int c1, int c2) const {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && wanted) {
            tma_store_3d(map, base, c0, c1, c2);
            tma_store_commit();
        }
    }
};

// The pre-activation that forward keeps for backward lies in blocks of 32 rows x 8 columns, a block's 16-byte row pieces one after the
// other: an epilogue lane holds one row of the accumulator, so the warp's 32 lanes write, and in backward read, 512 consecutive bytes per
// instruction, straight between registers and memory.  In rows of 2 I columns the forward would need two more boxes and a second read of
// the accumulator per tile, and the backward would have to turn what it reads in shared memory, half a box at a time, between the
// stores of its results.
__device__ __forceinline__ int4* preact_at(const LayerArgsP& L, int row0, int lane, int col) {
    return reinterpret_cast<int4*>(L.preact) + ((long)(row0 >> 5) * (L.I >> 2) + (col >> 3)) * 32 + lane;
}

// First GEMM, forward: accumulator columns (2j, 2j+1) = (gate_j, up_j).  act = silu(g) * u * w, as in gemm_common.cuh.
template <typename R>
__device__ __forceinline__ void epilogue_swiglu(const LayerArgsP& L, const Staging& st, uint32_t taddr, int row0, float w, int n0, R release) {
    const int n_total = 2 * L.I;
    int4* keep = preact_at(L, row0, st.lane, n0);
    st.reuse();
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        uint32_t acc[32];
        tmem_ld_x32(taddr + (uint32_t)(c * 32), acc);
        tmem_ld_wait();
        if (c == 3) release();
        uint32_t o[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float gt = __uint_as_float(acc[4 * p + 2 * e]), up = __uint_as_float(acc[4 * p + 2 * e + 1]);
                v[e] = __fdividef(gt, 1.f + __expf(-gt)) * up * w;
            }
            o[p] = pack_bf16x2(v[0], v[1]);
        }
        st.put(2 * c, o[0], o[1], o[2], o[3]);
        st.put(2 * c + 1, o[4], o[5], o[6], o[7]);
        if (L.keep && n0 + c * 32 < n_total) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const uint32_t* a = acc + 8 * v;
                keep[(4 * c + v) * 32] = make_int4((int)pack_bf16x2(__uint_as_float(a[0]), __uint_as_float(a[1])),
                                                   (int)pack_bf16x2(__uint_as_float(a[2]), __uint_as_float(a[3])),
                                                   (int)pack_bf16x2(__uint_as_float(a[4]), __uint_as_float(a[5])),
                                                   (int)pack_bf16x2(__uint_as_float(a[6]), __uint_as_float(a[7])));
            }
        }
    }
    st.store(n0 < n_total, &L.st_act, n0 >> 1, row0);
}

// First GEMM, backward: accumulator column j = d act_j.  Padding rows give zeros whatever the operands hold there: dGU and
// act x route are operands of the weight gradients, which sum over whole 64-row blocks.  The pre-activation comes 32 columns ahead, the
// first of it before the accumulator is ready.  16 columns are computed before the half box is waited for and written, so that the
// exponentials of 16 columns overlap: a warp is bound by the latency of its instructions (two epilogue warps per scheduler).  A
// 256-column accumulator takes 13.3 to 13.8 thousand cycles, the forward's 3.6 to 3.9, a plain store 1.5 to 2.6 (profiles/).
struct Preact {
    int4 v[8];      // 16-byte pieces of this lane's row: columns 8 i .. 8 i + 7 of 2 I
    __device__ __forceinline__ void request(const LayerArgsP& L, int row0, int col, int half, bool real, int lane) {
        const int4* p = preact_at(L, row0, lane, 2 * col);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * half + i] = real ? ld_nc_v4(p + 32 * (4 * half + i)) : make_int4(0, 0, 0, 0);
    }
};

template <typename R>
__device__ __forceinline__ void epilogue_dswiglu(const LayerArgsP& L, const Staging& st, uint32_t taddr, int row0, bool real, float w, int n0,
                                                 int part, Preact& pre, R release) {
    const long row = row0 + st.lane;
    float droute = 0.f;
    int turn = 0;
    st.reuse();                              // (the last store may be a whole box)
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        const int col = n0 + c * 32;
        const bool in = col < L.I;
        uint32_t acc[32];
        tmem_ld_x32(taddr + (uint32_t)(c * 32), acc);
        tmem_ld_wait();
        if (c == 3) release();
        uint32_t act[16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t dgu[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int v = 4 * h + i;
                const int4 g = pre.v[v];
                const uint32_t pr[4] = {(uint32_t)g.x, (uint32_t)g.y, (uint32_t)g.z, (uint32_t)g.w};
                float av[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 gu = unpack_bf16x2(pr[e]);
                    const float ga = real ? __uint_as_float(acc[4 * v + e]) : 0.f;
                    const float sig = __fdividef(1.f, 1.f + __expf(-gu.x));
                    const float s = gu.x * sig;
                    const float a = s * gu.y;
                    const float gaw = ga * w;
                    const float d_up = s * gaw;
                    const float d_gate = (sig - s * sig + s) * gaw * gu.y;
                    dgu[4 * i + e] = pack_bf16x2(d_gate, d_up);
                    av[e] = a * w;
                    droute += ga * a;
                }
                act[2 * v] = pack_bf16x2(av[0], av[1]);
                act[2 * v + 1] = pack_bf16x2(av[2], av[3]);
            }
            pre.request(L, row0, col + 32, h, real && c < 3 && col + 32 < L.I, st.lane);
            st.reuse<1>();
#pragma unroll
            for (int i = 0; i < 4; ++i) st.put_narrow(turn, i, dgu[4 * i], dgu[4 * i + 1], dgu[4 * i + 2], dgu[4 * i + 3]);
            st.store_narrow(turn++, in, &L.st_aux, 2 * col + 32 * h, row0);
        }
        st.reuse<1>();
#pragma unroll
        for (int i = 0; i < 4; ++i) st.put_narrow(turn, i, act[4 * i], act[4 * i + 1], act[4 * i + 2], act[4 * i + 3]);
        st.store_narrow(turn++, in, &L.st_act, col, row0);
    }
    L.droute_part[row * L.n_parts + part] = droute;
}

// 128 accumulator columns as two boxes; store_box(first column).  The second half is read while the first box is stored, and the
// accumulator is given back before the second box waits for the first: what a wide tile exposes is the time until then.
template <typename R, typename F>
__device__ __forceinline__ void epilogue_plain(const Staging& st, uint32_t taddr, bool zero, R release, F store_box) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t a0[32], a1[32], packed[32];
        tmem_ld_x32(taddr + (uint32_t)(h * 64), a0);
        tmem_ld_x32(taddr + (uint32_t)(h * 64 + 32), a1);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            packed[i] = zero ? 0u : pack_bf16x2(__uint_as_float(a0[2 * i]), __uint_as_float(a0[2 * i + 1]));
            packed[16 + i] = zero ? 0u : pack_bf16x2(__uint_as_float(a1[2 * i]), __uint_as_float(a1[2 * i + 1]));
        }
        if (h == 1) release();
        st.reuse();
#pragma unroll
        for (int c = 0; c < 8; ++c) st.put(c, packed[4 * c], packed[4 * c + 1], packed[4 * c + 2], packed[4 * c + 3]);
        store_box(h * 64);
    }
}

// ROWS: the loading warps bring what is made of token rows.  Without them (where local_layer_plan says so) rows are copied into slot order by
// the other warps first, and TMA loads them from there.
template <bool BWD, bool ROWS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(ROWS ? kLayerThreads : kThreads, 1)
local_layer_kernel(const __grid_constant__ LayerArgsP L) {
    if constexpr (!BWD) {
        if (L.unless_few && L.meta[kMetaFew] != 0) return;
    }
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + kBarOffsetP;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
    auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * kMaxStages + s); };
    auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * kMaxStages + 2 + s); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + kBarOffsetP + kOffTmem);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    auto ring_full = [&](int e) { return bar_base + kOffRingFull + 8u * e; };
    auto ring_empty = [&](int e) { return bar_base + kOffRingEmpty + 8u * e; };

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();

    if (threadIdx.x == 0) {
        *abort_flag = 0u;
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(full_bar(s), ROWS ? 4 : 2);            // of each CTA the producer and a loading warp
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), 2 * kEpiWarps);
        }
        for (int e = 0; e < kRingDepth; ++e) {
            mbar_init(ring_full(e), 1);
            mbar_init(ring_empty(e), ROWS ? kRingConsumers : kRingConsumers - 2 * kLoadWarps);
        }
        fence_mbar_init();
#pragma unroll
        for (int p = 0; p < (BWD ? 4 : 2); ++p) {
            if (!ROWS || (p != kWorkGemm1 && p != kWorkWgradDown)) tma_prefetch_desc(&L.ph[p].map_a);
            if (!ROWS || p != kWorkWgradGateup) tma_prefetch_desc(&L.ph[p].map_b);
        }
    }
    // With few rows per expert most rows of A are never loaded.  Zeros there cost the tensor cores least power; what an earlier kernel left in
    // shared memory would be multiplied for the whole call.  us of a step, back to back, zeros / none: 256 tokens, H=7168 I=2048, 32 experts, top-8
    // 1938 / 1985, I=512 588 / 600, H=4096 I=14336, 8 experts, top-2 1940 / 2011, with 8 rows per expert 1761 / 1770.  Forwards of 17 to 64
    // rows per expert 0 (behind other kernels not measured), steps of 128 rows 0 to 2 %.
    if ((long)L.T * L.K <= 64l * L.E) {
        for (int i = threadIdx.x; i < L.stages * (kAStageBytes / 16); i += (int)blockDim.x) {
            const int st = i / (kAStageBytes / 16);
            *reinterpret_cast<int4*>(smem_gen + st * L.stage_bytes + (i - st * (kAStageBytes / 16)) * 16) = make_int4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
    }
    if (warp == 2) tmem_alloc_2cta(smem_u32((const void*)tmem_slot), kTmemCols);
    tcgen05_fence_before();
    cluster_sync_all();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int target1 = 2 * kEpiWarps * L.ph[0].num_n_blocks;         // epilogue warps that finish a unit's first GEMM,
    const int target2 = kEpiWarps * L.ph[1].num_n_blocks;             // a block's second GEMM

    const int nvec = L.H / 8;
    // ---------------------------------------------------------------------- copy role (without loading warps)
    // Rows into slot order.  All warps but the producer's and the issuer's start with one slot each, so that the first units are in place
    // after the latency of one row; the rest is claimed by the gather warps, eight slots at a time.  A warp has 8 KB of loads in
    // flight: rows of 4096 columns and more one after the other, shorter ones several at once.  (Before, the first pairs of CTAs
    // streamed rows through shared memory and joined the GEMMs afterwards; rows of 1 KB left them waiting for one row at a time:
    // 8531 tokens, H=512, top-8 spent 240 us there.)
    auto copy_slots = [&](const int4* src, int4* dst, int row, uint32_t wanted, int s0, int n) {
        // row: source row of slot s0 + lane, -1 = zeros
        if (nvec >= 512) {
            for (int r = 0; r < n; ++r) {
                if (!((wanted >> r) & 1u)) continue;
                const int sr = __shfl_sync(0xffffffffu, row, r);
                int4* d = dst + (long)(s0 + r) * nvec;
                if (sr >= 0) copy_row_deep(d, src + (long)sr * nvec, nvec, lane);
                else for (int i = lane; i < nvec; i += 32) d[i] = make_int4(0, 0, 0, 0);
            }
            return;
        }
        const int total = n * nvec;
        for (int b = 0; b < total; b += 512) {
            int4 v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int idx = min(b + 32 * i + lane, total - 1), r = idx / nvec;
                const int sr = __shfl_sync(0xffffffffu, row, r);
                v[i] = ld_nc_v4(src + (long)max(sr, 0) * nvec + (idx - r * nvec));
                if (sr < 0) v[i] = make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int idx = b + 32 * i + lane;
                if (idx < total && ((wanted >> (idx / nvec)) & 1u)) dst[(long)s0 * nvec + idx] = v[i];
            }
        }
    };
    auto count_rows = [&](int* counter, int n) {
        __syncwarp();
        if (lane == 0 && n > 0) {
            fence_acq_rel_gpu();
            red_add_gpu(counter, n);
        }
    };
    auto place = [&](int s0, int n) {
        const int tk = lane < n ? L.slot_tk[s0 + lane] : -1;
        const int row = tk >= 0 ? tk / L.K : -1;
        uint32_t wanted = __ballot_sync(0xffffffffu, tk >= 0);
        if constexpr (BWD) {
            // both slot-order tables are operands of the weight gradients, which sum over 64 rows at a time: rows of zeros to the next 64
            wanted = L.slot_tk[s0 & ~63] >= 0 ? (1u << n) - 1u : 0u;
        }
        if (wanted == 0u) return;
        copy_slots(reinterpret_cast<const int4*>(L.x), reinterpret_cast<int4*>(L.slot_rows), row, wanted, s0, n);
        count_rows(L.arrived + (s0 >> 7), __popc(wanted));
    };
    auto place_x = [&](int s0, int n) {
        const int tk = lane < n ? L.slot_tk[s0 + lane] : -1;
        if (L.slot_tk[s0 & ~63] < 0) return;
        copy_slots(reinterpret_cast<const int4*>(L.saved_x), reinterpret_cast<int4*>(L.slot_x), tk >= 0 ? tk / L.K : -1, (1u << n) - 1u, s0, n);
        count_rows(L.sync + kSyncRows, n);
    };
    const int num_slots = L.meta[kMetaSlots];
    // (neighbouring slots go to different SMs: a few rows in one SM would queue behind one another)
    const int first_slots = (int)gridDim.x * kGatherWarps * kFirstRows / kCopyRows * kCopyRows;
    if (!ROWS && warp >= 2) {
        const int s0 = ((warp - 2) * (int)gridDim.x + (int)blockIdx.x) * kFirstRows;
        if (s0 < min(num_slots, first_slots)) place(s0, kFirstRows);
    }
    auto copy_loop = [&]() {
        while (true) {
            int s0 = 0;
            if (lane == 0) s0 = first_slots + atomicAdd(L.sync + kSyncCopy, kCopyRows);
            s0 = __shfl_sync(0xffffffffu, s0, 0);
            if (s0 >= num_slots) break;
            place(s0, kCopyRows);
        }
    };
    auto copy_x_loop = [&]() {
        // backward: x in slot order, which nothing needs before the weight gradients
        while (true) {
            int s0 = 0;
            if (lane == 0) s0 = atomicAdd(L.sync + kSyncKeep, kCopyRows);
            s0 = __shfl_sync(0xffffffffu, s0, 0);
            if (s0 >= num_slots) break;
            place_x(s0, kCopyRows);
        }
    };
    // ---------------------------------------------------------------------- forward: backward's copy of x
    auto keep_x_loop = [&]() {
        // 4 KB of loads in flight per warp
        while (true) {
            int t0 = 0;
            if (lane == 0) t0 = atomicAdd(L.sync + kSyncKeep, kCopyRows);
            t0 = __shfl_sync(0xffffffffu, t0, 0);
            if (t0 >= L.T) break;
            const long first = (long)t0 * nvec, total = (long)min(kCopyRows, L.T - t0) * nvec;
            const int4* src = reinterpret_cast<const int4*>(L.x) + first;
            int4* dst = reinterpret_cast<int4*>(L.saved_x) + first;
            for (long b = lane; b < total; b += 256) {
                int4 v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = ld_nc_v4(src + min(b + 32 * i, total - 1));
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (b + 32 * i < total) dst[b + 32 * i] = v[i];
            }
        }
    };

    // ---------------------------------------------------------------------- gather role
    // Rows [k0, k0 + n) of a token's entries, kVecs pieces of 16 bytes of each per lane, 32 pieces apart: all loads are issued before the
    // first is used (8 kVecs in flight per lane; a load behind a lane-dependent branch would be waited for one at a time, so
    // out-of-range columns are clamped and only their stores are left out).  Backward with loading warps, where the sums run under the weight
    // gradients, one piece: with two the registers do not suffice, and what is spilled then costs 5 %.
    constexpr int kVecs = BWD && ROWS ? 1 : 2;
    auto add_rows = [&](const int (&slots)[8], int n, uint32_t valid, const int (&at)[kVecs], float (&sum)[kVecs][8]) {
        int4 r[kVecs][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j < n) {
                const int4* row = reinterpret_cast<const int4*>(L.y) + (long)slots[j] * nvec;
#pragma unroll
                for (int v = 0; v < kVecs; ++v) r[v][j] = ld_cg_v4_ordered(row + at[v]);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j < n && ((valid >> j) & 1u)) {
#pragma unroll
                for (int v = 0; v < kVecs; ++v) {
                    const uint32_t p[4] = {(uint32_t)r[v][j].x, (uint32_t)r[v][j].y, (uint32_t)r[v][j].z, (uint32_t)r[v][j].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = unpack_bf16x2(p[i]);
                        sum[v][2 * i] += f.x;
                        sum[v][2 * i + 1] += f.y;
                    }
                }
            }
        }
    };
    auto gather_loop = [&]() {
        // A task is (token, part of its columns).  Most tokens become ready in the last few percent of the kernel, so the tail
        // is as long as the last tasks: about eleven for each of the 1480 warps that take part by then, down to 512 columns.
        // The order of a sum (k ascending) does not depend on it.
        const int K = L.K;
        const int steps = (nvec + 32 * kVecs - 1) / (32 * kVecs);
        const int parts = max(1, min(steps, kGatherTasks / max(L.T, 1)));
        const int part_steps = (steps + parts - 1) / parts;
        const int tasks = L.T * parts;
        uint64_t waited = 0;
        bool stamped = false;
        const bool stamps = L.stats != nullptr && lane == 0;
        // claimed one task ahead, with the token's slots, so that a task starts with the test of its counters
        int next_i = tasks, next_t = 0, next_slot = -1;
        // Few tasks are dealt out to all warps that gather in the end: they become ready together, and an atomic per task would be
        // half of what is left to do by then.
        const int warps = (int)gridDim.x * kGatherWarps;
        const bool dealt = !BWD && tasks <= 4 * warps;           // (backward they run under the weight gradients)
        next_i = dealt ? (int)blockIdx.x * kGatherWarps + (warp - 2) - warps : 0;
        auto claim = [&]() {
            if (dealt) {
                next_i += warps;
            } else {
                if (lane == 0) next_i = atomicAdd(L.sync + kSyncToken, 1);
                next_i = __shfl_sync(0xffffffffu, next_i, 0);
            }
            if (next_i < tasks) {
                next_t = L.token_order[next_i / parts];
                next_slot = lane < K ? L.order_slot[(long)(next_i / parts) * K + lane] : -1;
            }
        };
        if (L.T > 0) claim();
        else next_i = tasks;
        while (next_i < tasks) {
            const int part = next_i % parts, t = next_t, slot = next_slot;
            claim();
            const uint32_t valid = __ballot_sync(0xffffffffu, slot >= 0);
            if (!wait_counts_warp(L.done2 + (slot >= 0 ? slot >> 7 : 0), slot >= 0, target2, L.status, 660, waited)) return;      // reported: unwind
            __syncwarp();                                                     // every lane reads behind the other lanes' acquires
            if (stamps && !stamped) {
                stamped = true;
                atomicMax(L.stats + kStatKindFirst + kWorkReduce, ~globaltimer_ns());
            }
            if constexpr (BWD) {
                if (part == 0 && lane < K && slot < 0) L.dw_topk[(long)t * K + lane] = 0.f;
            }
            int4* dst = reinterpret_cast<int4*>(L.out + (long)t * L.H);
            const int step1 = min(steps, (part + 1) * part_steps);
            for (int step = part * part_steps; step < step1; ++step) {
                int at[kVecs];
                float sum[kVecs][8];
#pragma unroll
                for (int v = 0; v < kVecs; ++v) {
                    at[v] = min((step * kVecs + v) * 32 + lane, nvec - 1);
#pragma unroll
                    for (int i = 0; i < 8; ++i) sum[v][i] = 0.f;
                }
                for (int k0 = 0; k0 < K; k0 += 8) {
                    int sl[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) sl[j] = max(0, __shfl_sync(0xffffffffu, slot, (k0 + j) & 31));
                    add_rows(sl, min(K - k0, 8), valid >> k0, at, sum);
                }
#pragma unroll
                for (int v = 0; v < kVecs; ++v)
                    if ((step * kVecs + v) * 32 + lane < nvec)
                        dst[at[v]] = make_int4((int)pack_bf16x2(sum[v][0], sum[v][1]), (int)pack_bf16x2(sum[v][2], sum[v][3]),
                                               (int)pack_bf16x2(sum[v][4], sum[v][5]), (int)pack_bf16x2(sum[v][6], sum[v][7]));
            }
        }
        if (stamps) {
            atomicMax(L.stats + kStatKindLast + kWorkReduce, globaltimer_ns());
            if (waited) atomicAdd(L.stats + kStatWaitLanded, waited);
        }
    };

    // ---------------------------------------------------------------------- worker roles
    {
        const int total_items = min(L.meta[kMetaWork + (BWD ? 1 : 0)], L.max_work);
        const uint32_t ring_addr = bar_base + kOffItems;
        volatile int* ring = reinterpret_cast<volatile int*>(smem_gen + kBarOffsetP + kOffItems);
        // consumer side of the item ring (see layer.cu: the second CTA's entries arrive through the async proxy)
        auto next_item = [&](int& ss, uint32_t& sph, int site, int4& it) -> bool {
            if (!mbar_wait(ring_full(ss), sph, abort_flag, L.status, site)) return false;
            it = make_int4(ring[4 * ss], ring[4 * ss + 1], ring[4 * ss + 2], ring[4 * ss + 3]);
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) mbar_arrive(ring_empty(ss));
                else mbar_arrive_cluster(mapa_shared(ring_empty(ss), 0));
            }
            if (++ss == kRingDepth) { ss = 0; sph ^= 1u; }
            return true;
        };

        // rows of A that TMA loads for an item of which `need` are wanted, in boxes of 32 or of all
        auto rows_loaded = [](int need) { return need > 64 ? BM : (need + 31) & ~31; };
        // -------------------------------------------------------------- token rows
        // Operands that are made of token rows come straight from the caller's [T, H] tensor, row by row of the slot table: A of the first GEMM
        // (128 rows x 64 columns of K per step), A of dW_down and B of dW_gateup (64 rows of K x 128 or more columns).  Four warps of each CTA
        // copy them, eight lanes to 128 bytes, in the layout that TMA gives the other operands.  Before, other warps copied every
        // row into slot order first, and TMA loaded it from there: K times the tensor written and read once more (0.94 GB of each per
        // copy and three copies in a step of 8192 tokens, H=7168, top-8).  TMA's own row gather moves 512 bytes in 70 cycles, a third of what
        // a mainloop needs.  Forward + backward, ms: 16384 tokens, H=7168 I=512, top-8 9.55 -> 8.77 (backward's first GEMM no longer waits
        // for rows: 2283 -> 1280 cycles per step); 4096, H=2048 I=2048, top-8 2.342 -> 2.299; 8192, H=7168 I=2048 14.93 -> 14.92;
        // forward of 3001 tokens 1.897 -> 1.871, of 32 tokens 0.582 -> 0.592.  (With TMA loads of as many consecutive rows instead the
        // large forward would take 3 % less: what these copies cost.)
        //
        // A warp takes every fourth step: it waits for the stage, copies, and hands the step over when its copies have landed, which it sees to
        // behind the copies of its next step if that one's stage is free, so that copies into all stages are under way at a time.
        // All four warps on every step, two steps under way, were 4 % slower; an address computed per column block instead of per
        // row made dW_gateup 25 % slower; registers for fewer addresses (56 instead of 112 per thread, some spilled) cost 5 %.
        auto load_rows = [&]() {
            const int sub = lane >> 3, chunk = lane & 7;
            const uint32_t pair_full = mapa_shared(full_bar(0), 0);
            const uint32_t at[2] = {(uint32_t)(sub * 128 + ((chunk ^ sub) << 4)), (uint32_t)(sub * 128 + ((chunk ^ (sub + 4)) << 4))};      // rows 8i + sub, 8i + 4 + sub
            const uint64_t inverse = ~0ull / (uint32_t)L.K;   // entry / K = (entry + 1) * floor((2^64 - 1) / K) / 2^64, exact for 32-bit entries
            auto token = [&](int tk) { return tk < 0 ? -1 : (int)__umul64hi((uint64_t)(uint32_t)tk + 1u, inverse); };
            const long pitch = L.H * 2l;
            int step = warp - 12, stage = step, ss = 0;      // this warp's next step, counted from the start of the item; its stage
            uint32_t phase = 0, sph = 0;
            int under_way = -1;                              // stage of the step before, if its copies are not yet seen through
            Leftover left{L.clean != 0, BM};
            // The arrive is all that orders the rows before the products that the first CTA issues: no byte count covers them.
            auto hand_over = [&](int s) {
                fence_proxy_async_smem();
                __syncwarp();
                if (lane != 0) return;
                if (rank == 0) mbar_arrive(full_bar(s));
                else mbar_arrive_cluster_release_smem(pair_full + 8u * s);
            };
            auto settle = [&]() {
                if (under_way < 0) return;
                cp_async_wait<0>();
                hand_over(under_way);
                under_way = -1;
            };
            while (true) {
                int4 it;
                if (!__all_sync(0xffffffffu, mbar_test_wait(ring_full(ss), sph))) settle();
                if (!next_item(ss, sph, 654, it) || it.x < 0) break;
                Item q;
                decode_item(L, it, rank, q);
                int row[4] = {-1, -1, -1, -1};               // first GEMM: tokens of rows lane + 32 i; gradients: entries of K rows lane + 32 i of this step
                const bool down = q.kind == kWorkWgradDown;
                int all_rows = 0;                            // first GEMM: steps whose 128 rows are all written
                if (q.kind == kWorkGemm1) {
                    all_rows = left.take_rows(q.half, q.real, q.nk, L.stages);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int r = lane + 32 * i;
                        if (r >= q.real) continue;
                        row[i] = token(L.slot_tk[q.m0 + r]);
                        // a table that says less than the list: a row that never arrives
                        if (row[i] < 0) report_status(L.status, kStatusFlagTimeout, 600, q.m0 + r);
                    }
                } else if (q.kind == kWorkGemm2) {
                    left.take_boxes(q.half, rows_loaded(q.need), q.nk, L.stages);
                } else if (BWD) {
                    left.rows = BM;
#pragma unroll
                    for (int i = 0; i < 2; ++i) row[i] = step < q.nk ? L.slot_tk[q.k0 + step * BK + lane + 32 * i] : -1;
                }
                bool ok = true;
                for (; step < q.nk; step += kLoadWarps) {
                    // (never behind a wait: the stage may be waiting for the step before)
                    if (q.kind == kWorkGemm2 || !__all_sync(0xffffffffu, mbar_test_wait(empty_bar(stage), phase ^ 1u))) settle();
                    if (!(ok = mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, L.status, 611))) break;
                    const uint32_t dst = smem_base + (uint32_t)(stage * L.stage_bytes);
                    if (q.kind == kWorkGemm1) {
                        const uint8_t* src = L.x + step * 128 + 16 * chunk;
                        // (unrolled, with no branch between them, the loads follow each other; a loop that ends with the rows is a third slower)
                        auto copy = [&](auto quads) {
#pragma unroll
                            for (int j = 0; j < decltype(quads)::value; ++j) {
                                const int t = __shfl_sync(0xffffffffu, row[j >> 3], (4 * j + sub) & 31);
                                cp_async_16_or_zeros(dst + j * 512 + at[j & 1], src + max(t, 0) * pitch, t >= 0);
                            }
                        };
                        if (step < all_rows) copy(std::integral_constant<int, 32>());
                        else copy(std::integral_constant<int, 8>());
                    } else if (BWD && q.kind != kWorkGemm2) {
                        const uint8_t* src = (down ? L.x : reinterpret_cast<const uint8_t*>(L.saved_x)) + 16 * chunk;
                        const int tok[2] = {token(row[0]), token(row[1])};
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            row[i] = step + kLoadWarps < q.nk ? L.slot_tk[q.k0 + (step + kLoadWarps) * BK + lane + 32 * i] : -1;
                        // (no branch between the copies: columns past the last are zeros)
                        const int c0 = down ? q.m0 : q.n0 + (int)rank * (BN / 2);
                        auto copy = [&](auto atoms) {
                            constexpr int kAtoms = decltype(atoms)::value;
                            bool in[kAtoms];
                            int at_col[kAtoms];
#pragma unroll
                            for (int a = 0; a < kAtoms; ++a) {
                                const int col = c0 + (a >> 1) * BN + (a & 1) * 64;
                                in[a] = col < L.H;
                                at_col[a] = in[a] ? col * 2 : 0;
                            }
                            const int slices = step == q.nk - 1 ? q.tail : BK / UK;
#pragma unroll 1
                            for (int k = 0; k < slices; ++k) {       // 16 rows
                                const int rows = k < 2 ? tok[0] : tok[1];
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const int t = __shfl_sync(0xffffffffu, rows, (16 * k + 4 * j + sub) & 31);
                                    const uint8_t* from = src + max(t, 0) * pitch;
                                    const uint32_t to = dst + (down ? 0 : kAStageBytes) + (4 * k + j) * 512 + at[j & 1];
#pragma unroll
                                    for (int a = 0; a < kAtoms; ++a) cp_async_16_or_zeros(to + a * kAtomBytes, from + at_col[a], in[a] && t >= 0);
                                }
                            }
                        };
                        if (down || q.halves == 1) copy(std::integral_constant<int, 2>());
                        else copy(std::integral_constant<int, 4>());
                    }
                    if (q.kind == kWorkGemm2) {
                        // no rows; the warp takes part all the same, so that it is never a whole turn through the stages behind or ahead of the
                        // others, which the parity of a phase would not show
                        hand_over(stage);
                    } else {
                        cp_async_commit();
                        if (under_way >= 0) {
                            cp_async_wait<1>();
                            hand_over(under_way);
                        }
                        under_way = stage;
                    }
                    stage += kLoadWarps;
                    if (stage >= L.stages) { stage -= L.stages; phase ^= 1u; }
                }
                if (!ok) break;
                step -= q.nk;
            }
            settle();
        };

        if (ROWS && warp >= 12) {
            registers_dec<kRegsLoad>();
            load_rows();
        } else if (warp < 4) {
        if (warp == 0) {
            // -------------------------------------------------------------- item fetch (first CTA) + TMA producer
            if (elect_one()) {
                const int stages = L.stages;
                const uint32_t stage_bytes = (uint32_t)L.stage_bytes, pair_full = mapa_shared(full_bar(0), 0);
                Leftover left[2] = {{L.clean != 0, BM}, {L.clean != 0, BM}};         // of both CTAs: the first one's producer counts the bytes of both
                int stage = 0;
                uint32_t phase = 0;
                bool ok = true;
                int ss = 0;
                uint32_t sph = 0;
                // Both producers look at the NEXT item while the loads of the current one are in flight: they fetch it and test what
                // its operands wait for, so that between two items there is normally nothing to wait for.
                int claim = (rank == 0) ? atomicAdd(L.sync + kSyncItem, 1) : 0;
                unsigned long long w_arrive = 0, w_unit = 0, w_wgrad = 0;
                bool wgrad_ready = false, wgrad_fenced = false;
                int4 cur = make_int4(-1, 0, 0, 0), nxt = cur;
                bool have = false, nxt_ready = false;
                // 1: got an item, 0: none yet (non-blocking form, second CTA), -1: a wait ran out
                auto get_item = [&](int4& it, bool blocking) -> int {
                    if (rank == 0) {
                        it = (claim < total_items) ? L.work[claim] : make_int4(-1, 0, 0, 0);
                        if (it.x >= 0) claim = atomicAdd(L.sync + kSyncItem, 1);      // needed when the next item is fetched
                        if (!mbar_wait(ring_empty(ss), sph ^ 1u, abort_flag, L.status, 650)) return -1;
                        ring[4 * ss] = it.x; ring[4 * ss + 1] = it.y; ring[4 * ss + 2] = it.z; ring[4 * ss + 3] = it.w;
                        mbar_arrive(ring_full(ss));
                        const uint32_t remote_bar = mapa_shared(ring_full(ss), 1);
                        mbar_arrive_expect_tx_cluster(remote_bar, 16u);
                        st_async_v4_cluster(mapa_shared(ring_addr + 16u * ss, 1), it, remote_bar);
                    } else {
                        if (blocking) {
                            if (!mbar_wait(ring_full(ss), sph, abort_flag, L.status, 651)) return -1;
                        } else if (!mbar_test_wait(ring_full(ss), sph)) {
                            return 0;
                        }
                        it = make_int4(ring[4 * ss], ring[4 * ss + 1], ring[4 * ss + 2], ring[4 * ss + 3]);
                        mbar_arrive_cluster(mapa_shared(ring_empty(ss), 0));
                    }
                    if (++ss == kRingDepth) { ss = 0; sph ^= 1u; }
                    return 1;
                };
                auto counted = [&](const int* flag, int target, bool block, int site, unsigned long long& waited) -> int {
                    if (ld_acquire_gpu(flag) >= target) return 1;
                    if (!block) return 0;
                    const uint64_t t0 = globaltimer_ns();
                    const bool got = wait_count_gpu(flag, target, L.status, site, 64);
                    waited += globaltimer_ns() - t0;
                    return got ? 1 : -1;
                };
                // what the operands of an item wait for; `block`: wait (bounded) instead of only looking
                auto operands_ready = [&](const Item& q, bool block) -> int {
                    if (q.kind == kWorkGemm1) return (ROWS || q.need == 0) ? 1 : counted(L.arrived + q.m0 / BM, q.wait, block, 600, w_arrive);
                    if (q.kind == kWorkGemm2) return counted(L.done1 + q.unit, target1, block, 601, w_unit);
                    // the weight gradients sit behind all first GEMMs in the list: one check per pair is enough (two loads per expert and pair
                    // would cost as much as the smallest of these items)
                    if (wgrad_ready) return 1;
                    int r = counted(L.sync + kSyncFirsts, L.meta[kMetaUnits] * target1, block, 602, w_wgrad);
                    if (!ROWS && r == 1) r = counted(L.sync + kSyncRows, L.meta[kMetaRows], block, 603, w_wgrad);
                    wgrad_ready = r == 1;
                    return r;
                };
                auto look_ahead = [&]() -> bool {            // false: a wait ran out
                    const int r = get_item(nxt, false);
                    if (r < 0) return false;
                    if (r == 0) return true;
                    have = true;
                    nxt_ready = false;
                    if (nxt.x >= 0) {
                        Item qn;
                        decode_item(L, nxt, rank, qn);
                        nxt_ready = operands_ready(qn, false) == 1;
                    }
                    return true;
                };
                while (ok) {
                    bool cur_ready = false;
                    if (have) {
                        cur = nxt;
                        cur_ready = nxt_ready;
                        have = false;
                    } else if (get_item(cur, true) < 0) {
                        ok = false;
                        break;
                    }
                    if (cur.x < 0) break;
                    Item q;
                    decode_item(L, cur, rank, q);
                    const Phase& P = L.ph[q.kind];
                    const bool gemm = q.kind <= kWorkGemm2;
                    const int n0 = q.n0 + (int)rank * (BN / 2);
                    // The two GEMMs, rows of A that a CTA loads: none that nothing is summed from, up to 64 in boxes of 32; behind them zeros in the
                    // first steps, where something else may be left.  What is made of token rows may come from
                    // the loading warps: A of the first GEMM and of dW_down, B of dW_gateup.
                    const int a_rows = rows_loaded(q.need), needs[2] = {unit_rows(cur, 0, q.half, false), unit_rows(cur, 1, q.half, false)};
                    const bool rows_a = ROWS && (q.kind == kWorkGemm1 || q.kind == kWorkWgradDown), rows_b = ROWS && q.kind == kWorkWgradGateup;
                    const int a_pair = rows_a ? 0 : (gemm ? rows_loaded(needs[0]) + rows_loaded(needs[1]) : 2 * BM);
                    uint32_t tx = (uint32_t)(a_pair * (BK * 2) + (rows_b ? 0 : 2 * q.halves * kBHalfBytesP));
                    int zeros_to = 0;                                          // up to which row the first steps write zeros, in this CTA,
                    uint32_t tx_zeros = 0;                                     // and their bytes in both
                    if (L.clean) {
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            if (!gemm) {
                                left[r].rows = BM;
                            } else if (rows_a) {                               // (as the loading warps do it)
                                left[r].take_rows(q.half, unit_rows(cur, r, q.half, true), q.nk, stages);
                            } else {
                                const int loaded = rows_loaded(needs[r]), to = left[r].take_boxes(q.half, loaded, q.nk, stages);
                                tx_zeros += (uint32_t)((to - loaded) * (BK * 2));
                                if (r == (int)rank) zeros_to = to;
                            }
                        }
                    }
                    tx += tx_zeros;                                            // (taken off again behind those steps)
                    const int look_kb = min(stages - 1, q.nk - 1);     // all stages are in flight: a pause of this thread costs nothing
                    auto take_stage = [&](int st, uint32_t ph) {
                        if (!mbar_wait(empty_bar(st), ph ^ 1u, abort_flag, L.status, 610)) return false;
                        if (rank == 0) mbar_arrive_expect_tx(full_bar(st), tx);
                        else mbar_arrive_cluster(pair_full + 8u * st);
                        return true;
                    };
                    const CUtensorMap* map_b = &P.map_b;
                    const int b_row = q.group * P.b_group_rows;
                    auto load_b = [&](int st, int k) {
                        if (rows_b) return;
                        const uint32_t dst = smem_base + (uint32_t)st * stage_bytes + kAStageBytes, bar = pair_full + 8u * st;
                        for (int h = 0; h < q.halves; ++h) {
                            if (!BWD) tma_load_2d_2cta(dst + h * kBHalfBytesP, map_b, bar, k, b_row + n0 + h * BN);
                            else tma_load_3d_2cta(dst + h * kBHalfBytesP, map_b, bar, 0, b_row + k, (n0 + h * BN) >> 6);
                        }
                    };
                    // What a GEMM waits for is its rows; the weights of its first steps come meanwhile.
                    int early = 0;
                    if (!cur_ready) {
                        if (gemm) {
                            int st = stage;
                            uint32_t ph = phase;
                            for (; early < min(stages, q.nk); ++early) {
                                if (!(ok = take_stage(st, ph))) break;
                                load_b(st, early * BK);
                                if (++st == stages) { st = 0; ph ^= 1u; }
                            }
                        }
                        if (!ok) break;
                        // A wait that runs out has been reported.  This item is carried through all the same, on whatever its operands
                        // hold: loads and stores under way end in order, as do the other roles, and no copy outlives its block.  The pair
                        // takes no further item when the first CTA sees it, and no CTA waits for long once the report is there.
                        if (operands_ready(q, true) != 1 && rank == 0) claim = total_items;
                    }
                    // stores of other SMs -> async-proxy reads; the weight gradients acquire once, so they need the fence once
                    if (gemm || !wgrad_fenced) fence_proxy_async_all();
                    if (!gemm) wgrad_fenced = true;
                    int kb = 0;
                    auto load_steps = [&](int end, auto&& load_a) {
                        for (; kb < end; ++kb) {
                            if (kb >= early && !take_stage(stage, phase)) return false;
                            load_a(smem_base + (uint32_t)stage * stage_bytes, pair_full + 8u * stage, kb * BK);
                            if (kb >= early) load_b(stage, q.k0 + kb * BK);
                            if (++stage == stages) { stage = 0; phase ^= 1u; }
                            // (the second CTA keeps looking until the first one has published the item)
                            if (kb >= look_kb && !have && (kb == look_kb || rank != 0) && !look_ahead()) return false;
                        }
                        return true;
                    };
                    if (rows_a) {
                        ok = load_steps(q.nk, [](uint32_t, uint32_t, int) {});
                    } else if (gemm) {
                        const CUtensorMap* map_a = a_rows == BM ? &P.map_a : &P.map_a32;
                        auto load_a = [&](uint32_t dst, uint32_t bar, int k) {
                            if (a_rows != 0) tma_load_2d_2cta(dst, map_a, bar, k, q.m0);
                            if (a_rows == 64) tma_load_2d_2cta(dst + 32 * BK * 2, map_a, bar, k, q.m0 + 32);
                        };
                        if (tx_zeros != 0) {
                            // (rows past the last one of the map are zeros)
                            ok = load_steps(min(stages, q.nk), [&](uint32_t dst, uint32_t bar, int k) {
                                load_a(dst, bar, k);
                                for (int r = a_rows; r < zeros_to; r += 32) tma_load_2d_2cta(dst + r * BK * 2, &P.map_a32, bar, k, P.m_total);
                            });
                            tx -= tx_zeros;
                        }
                        ok = ok && load_steps(q.nk, load_a);
                    } else if constexpr (BWD) {
                        const CUtensorMap* map_a = &P.map_a;
                        ok = load_steps(q.nk, [&](uint32_t dst, uint32_t bar, int k) { tma_load_3d_2cta(dst, map_a, bar, 0, q.k0 + k, q.m0 >> 6); });
                    }
                }
                if (!ok) {
                    // A wait inside the pair ran out: no barrier says when the copies under way have landed (those of both CTAs count on the
                    // first one's, which may never complete).  They take microseconds; no block of the pair ends before this one.
                    for (const uint64_t t0 = globaltimer_ns(); globaltimer_ns() - t0 < 10000000ull;) __nanosleep(1000);
                }
                if (L.stats != nullptr) {
                    if (w_arrive) atomicAdd(L.stats + kStatWaitArrival, w_arrive);
                    if (w_unit) atomicAdd(L.stats + kStatWaitFirstGemm, w_unit);
                    if (w_wgrad) atomicAdd(L.stats + kStatWaitWgrad, w_wgrad);
                }
            }
        } else if (warp == 1 && rank == 0) {
            // -------------------------------------------------------------- UMMA issuer
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int ss = 0;
            uint32_t sph = 0;
            int acc = 0;                                     // accumulators (256 columns) used so far
            while (ok) {
                int4 it;
                if (!next_item(ss, sph, 652, it) || it.x < 0) break;
                Item q;
                decode_item(L, it, rank, q);
                const int slot0 = acc & 1, slot1 = slot0 ^ 1;
                const uint32_t parity0 = ((acc >> 1) & 1) ^ 1u, parity1 = (((acc + 1) >> 1) & 1) ^ 1u;
                acc += q.halves;
                // ROWS_M rows of A, A_MN: K runs along its rows.  (An instance of the loop for each: the instruction descriptor is a constant in it.)
                auto mainloop = [&](auto rows_m, auto a_mn_) -> bool {
                    constexpr bool a_mn = decltype(a_mn_)::value;
                    constexpr uint32_t idesc = make_idesc_bf16(decltype(rows_m)::value, BN, a_mn, BWD);
                    // Operand descriptors of stage 0; a stage or a step of K further on is an addition to their address field.
                    const uint64_t a_base = make_smem_desc_sw128(smem_base, a_mn ? kAtomBytes : 0, 1024);
                    const uint64_t b_base = make_smem_desc_sw128(smem_base + kAStageBytes, BWD ? kAtomBytes : 0, 1024);
                    constexpr uint32_t a_step = (a_mn ? UK * 128 : UK * 2) >> 4, b_step = (BWD ? UK * 128 : UK * 2) >> 4;
                    // 64 columns of K of one half of the tile
                    auto multiply = [&](int s, int h, int slot, int kb) {
                        const uint32_t off = (uint32_t)(s * L.stage_bytes) >> 4;
                        const uint64_t a_desc = a_base + off, b_desc = b_base + off + (uint32_t)(h * (kBHalfBytesP >> 4));
                        const uint32_t d_tmem = tmem_base + (uint32_t)(slot * BN);
                        const int slices = BWD && kb == q.nk - 1 ? q.tail : BK / UK;
#pragma unroll
                        for (int k = 0; k < BK / UK; ++k)
                            if (k < slices) umma_bf16_ss_2cta(d_tmem, a_desc + k * a_step, b_desc + k * b_step, idesc, (kb | k) != 0 ? 1u : 0u);
                    };
                    // (the second CTA's loading warps hand over rows that lie there)
                    auto wait_full = [&](int s, uint32_t ph) {
                        return ROWS ? mbar_wait_cluster_acquire_smem(full_bar(s), ph, abort_flag, L.status, 621) : mbar_wait(full_bar(s), ph, abort_flag, L.status, 621);
                    };
                    if (!mbar_wait(tempty_bar(slot0), parity0, abort_flag, L.status, 620)) return false;
                    tcgen05_fence_after();
                    int kb = 0;
                    if (q.halves == 2) {
                        // The second accumulator is still being read out when a wide tile starts: the first half runs ahead over the stages
                        // that are there, the second half follows and frees them.
                        const int lead = min(q.nk, L.stages);
                        int s = stage;
                        uint32_t ph = phase;
                        for (int i = 0; i < lead; ++i) {
                            if (!wait_full(s, ph)) return false;
                            tcgen05_fence_after();
                            if (elect_one()) {
                                multiply(s, 0, slot0, i);
                                if (i == q.nk - 1) umma_commit_2cta(tfull_bar(slot0), 3u);
                            }
                            __syncwarp();
                            if (++s == L.stages) { s = 0; ph ^= 1u; }
                        }
                        if (!mbar_wait(tempty_bar(slot1), parity1, abort_flag, L.status, 622)) return false;
                        tcgen05_fence_after();
                        for (; kb < lead; ++kb) {
                            if (elect_one()) {
                                multiply(stage, 1, slot1, kb);
                                umma_commit_2cta(empty_bar(stage), 3u);
                                if (kb == q.nk - 1) umma_commit_2cta(tfull_bar(slot1), 3u);
                            }
                            __syncwarp();
                            if (++stage == L.stages) { stage = 0; phase ^= 1u; }
                        }
                    }
                    for (; kb < q.nk; ++kb) {
                        if (!wait_full(stage, phase)) return false;
                        tcgen05_fence_after();
                        if (elect_one()) {
                            const bool last = kb == q.nk - 1;
                            multiply(stage, 0, slot0, kb);
                            if (q.halves == 2) {
                                if (last) umma_commit_2cta(tfull_bar(slot0), 3u);
                                multiply(stage, 1, slot1, kb);
                            }
                            umma_commit_2cta(empty_bar(stage), 3u);
                            if (last) umma_commit_2cta(tfull_bar(q.halves == 2 ? slot1 : slot0), 3u);
                        }
                        __syncwarp();
                        if (++stage == L.stages) { stage = 0; phase ^= 1u; }
                    }
                    return true;
                };
                using Rows = std::integral_constant<uint32_t, 2 * BM>;
                using HalfRows = std::integral_constant<uint32_t, BM>;
                if (BWD && q.kind >= kWorkWgradDown) ok = mainloop(Rows(), std::integral_constant<bool, BWD>());
                else if (q.half) ok = mainloop(HalfRows(), std::false_type());
                else ok = mainloop(Rows(), std::false_type());
                if (ok && q.nk == 0) {                       // an expert without rows: the epilogue stores zeros
                    if (elect_one()) {
                        umma_commit_2cta(tfull_bar(slot0), 3u);
                        if (q.halves == 2) umma_commit_2cta(tfull_bar(slot1), 3u);
                    }
                    __syncwarp();
                }
            }
        } else if (warp >= 2) {
            if constexpr (!ROWS) copy_loop();
            if constexpr (BWD && !ROWS) copy_x_loop();
            if (!BWD && L.saved_x != nullptr) keep_x_loop();
            gather_loop();
        }
        } else {
            // -------------------------------------------------------------- epilogue, then gather
            if constexpr (ROWS) registers_inc<kRegsEpilogue>();
            const int qd = warp & 3;
            const int hh = (warp - 4) >> 2;
            const Staging st{smem_base + kPipeBytesP + (uint32_t)(warp - 4) * kBoxBytes, lane};
            bool ok = true;
            int ss = 0;
            uint32_t sph = 0;
            int acc = 0;
            // Tiles whose stores are not yet counted as complete (bit 31: first GEMM).  They are counted in one go when this warp would
            // have to wait for its next item or accumulator (for more than a moment: counting waits for the stores), or when the
            // list is full: narrow tiles (K of a few hundred) follow each other faster than a store, a fence and an atomic complete.  Never
            // behind such a wait: the next item may be one that waits for this count.
            uint32_t owed[kOwed];
            int n_owed = 0;
            auto flush = [&]() {
                if (n_owed == 0) return;
                __syncwarp();
                if (lane == 0) {
                    tma_store_wait<0>();
                    fence_proxy_async_all();
                    fence_acq_rel_gpu();
                    int firsts = 0;
#pragma unroll
                    for (int i = 0; i < kOwed; ++i) {
                        if (i >= n_owed) break;
                        const int at = (int)(owed[i] & 0x7fffffffu);
                        const bool first = owed[i] >> 31;
                        red_add_gpu((first ? L.done1 : L.done2) + at, 1);      // (ordered by the fence)
                        firsts += first;
                    }
                    if (BWD && firsts != 0) red_add_gpu(L.sync + kSyncFirsts, firsts);
                }
                n_owed = 0;
            };
            auto soon = [&](uint32_t bar, uint32_t parity) {
                for (int i = 0; i < kSoon; ++i)
                    if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
                return false;
            };
            while (ok) {
                int4 it;
                if (n_owed != 0 && !soon(ring_full(ss), sph)) flush();
                if (!next_item(ss, sph, 653, it) || it.x < 0) break;
                const bool stamps = L.stats != nullptr && warp == 4 && lane == 0 && rank == 0;
                Item q;
                decode_item(L, it, rank, q);
                if (stamps) atomicMax(L.stats + kStatKindFirst + q.kind, ~globaltimer_ns());
                if (q.kind > kWorkGemm2) flush();  // (the weight gradients may never wait, and the sums run under them)
                // The accumulator of a half unit: its 64 rows are twice in tensor memory, lanes 0 to 63 with the first 128 columns of the tile and
                // lanes 64 to 127 with the others, so that one of the two warps of a quarter has nothing to do.
                const int row_in = (q.half ? qd & 1 : qd) * 32, col_in = (q.half ? qd >> 1 : hh) * (BN / 2), tmem_col = q.half ? 0 : hh * (BN / 2);
                const int row0 = q.m0 + row_in;
                // rows of a block beyond those that are used are neither computed on nor stored
                const bool live = q.kind > kWorkGemm2 || (row_in < q.need && !(q.half && hh != 0));
                bool real = false;                 // backward, first GEMM: this lane's row is not padding
                if constexpr (BWD) real = q.kind == kWorkGemm1 && live && row_in + lane < q.real;
                for (int h = 0; h < q.halves; ++h) {
                    const int slot = acc & 1;
                    const uint32_t parity = (acc >> 1) & 1;
                    ++acc;
                    const int n0 = q.n0 + h * BN + col_in;
                    const float w = (q.kind == kWorkGemm1 && live) ? L.slot_w[row0 + lane] : 0.f;       // (padding: 0)
                    Preact pre;
                    if constexpr (BWD) {
                        if (q.kind == kWorkGemm1) {
                            pre.request(L, row0, n0, 0, real && n0 < L.I, lane);
                            pre.request(L, row0, n0, 1, real && n0 < L.I, lane);
                        }
                    }
                    if (n_owed != 0 && (n_owed == kOwed || !soon(tfull_bar(slot), parity))) flush();
                    if (!mbar_wait(tfull_bar(slot), parity, abort_flag, L.status, 630)) { ok = false; break; }
                    tcgen05_fence_after();
                    const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + (uint32_t)(slot * BN + tmem_col);
                    // this warp has read its part of the accumulator: the issuer may overwrite it
                    auto release = [&]() {
                        tcgen05_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(mapa_shared(tempty_bar(slot), 0));
                    };
                    if (!live) {
                        release();
                    } else if (q.kind == kWorkGemm1) {
                        if constexpr (BWD) epilogue_dswiglu(L, st, taddr, row0, real, w, n0, n0 / (BN / 2), pre, release);
                        else epilogue_swiglu(L, st, taddr, row0, w, n0, release);
                    } else if (q.kind == kWorkGemm2) {
                        epilogue_plain(st, taddr, false, release, [&](int c) {
                            st.store(n0 + c < L.H, &L.st_y, n0 + c, row0);
                        });
                        if constexpr (BWD) {
                            if (n0 == 0) {
                                // this row's d(route weight): the sum of the first GEMM's partials
                                const long row = row0 + lane;
                                const int tk = L.slot_tk[row];
                                if (tk >= 0) {
                                    float v = 0.f;
                                    for (int p = 0; p < L.n_parts; ++p) v += __ldcg(L.droute_part + row * L.n_parts + p);
                                    L.dw_topk[tk] = v;
                                }
                            }
                        }
                    } else {
                        if constexpr (BWD) {
                            const Phase& P = L.ph[q.kind];
                            const CUtensorMap* map = q.kind == kWorkWgradDown ? &L.st_dwd : &L.st_dwg;
                            const int m = q.m_in_group + qd * 32;
                            epilogue_plain(st, taddr, q.nk == 0, release, [&](int c) {
                                st.store3(m < P.m_total && n0 + c < P.n_total, map, n0 + c, m, q.group);
                            });
                        }
                    }
                }
                if (!ok) break;
                if (stamps) atomicMax(L.stats + kStatKindLast + q.kind, globaltimer_ns());
                // (of a half unit both CTAs count for the one block)
                if (q.kind == kWorkGemm1 || (q.kind == kWorkGemm2 && (q.half ? hh == 0 : rank == 0 || ((it.x >> 4) & 1) != 0))) {
                    const uint32_t entry = q.kind == kWorkGemm1 ? (0x80000000u | (uint32_t)q.unit) : (uint32_t)(q.m0 / BM);
#pragma unroll
                    for (int i = 0; i < kOwed; ++i)
                        if (i == n_owed) owed[i] = entry;
                    ++n_owed;
                }
            }
            flush();
            if (lane == 0) tma_store_wait<0>();
            __syncwarp();
            if (ok) gather_loop();            // the list is done: help with the sums
        }
    }

    tcgen05_fence_before();
    cluster_sync_all();
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc_2cta(tmem_base, kTmemCols);
    }
}

// [rows, cols] bf16, boxes of 32 rows x 32 columns, 64-byte swizzle
cudaError_t make_map_narrow(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols) {
    EncodeTiledFn fn = get_encode_fn();
    if (fn == nullptr) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return cudaErrorInvalidValue;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * 2};
    cuuint32_t box[2] = {32, 32};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// [rows, cols] bf16 (cols a multiple of 64) as an operand whose rows are steps of K: boxes of 64 rows x 128 columns, laid down as two
// swizzled atoms of 64 columns, in one copy
cudaError_t make_map_mn(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols) {
    EncodeTiledFn fn = get_encode_fn();
    if (fn == nullptr) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return cudaErrorInvalidValue;
    cuuint64_t dims[3] = {64, rows, cols / 64};
    cuuint64_t strides[2] = {cols * 2, 128};
    cuuint32_t box[3] = {64, BK, 2};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// [groups, rows, cols] bf16, boxes of 32 rows x 64 columns of one group; rows and columns outside a group are not written
cudaError_t make_store_map3(CUtensorMap* map, const void* base, uint64_t groups, uint64_t rows, uint64_t cols) {
    EncodeTiledFn fn = get_encode_fn();
    if (fn == nullptr) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return cudaErrorInvalidValue;
    cuuint64_t dims[3] = {cols, rows, groups};
    cuuint64_t strides[2] = {cols * 2, rows * cols * 2};
    cuuint32_t box[3] = {64, 32, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <bool BWD, bool ROWS>
cudaError_t launch(const LayerArgsP& L, int num_sms, cudaStream_t stream) {
    auto kern = local_layer_kernel<BWD, ROWS>;
    static bool configured[64] = {};
    if (cudaError_t e = ensure_smem_limit(kern, kSmemBytesP, configured); e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_sms & ~1);
    cfg.blockDim = dim3(ROWS ? kLayerThreads : kThreads);
    cfg.dynamicSmemBytes = kSmemBytesP;
    cfg.stream = stream;
    // every pair waits for tiles of other pairs, and without loading warps for rows that warps of all blocks copy: all have to be resident
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, L);
}

}  // namespace

LocalLayerPlan local_layer_plan(int T, int K, int E, int H, int I, int keep) {
    LocalLayerPlan p{};
    p.T = T; p.K = K; p.E = E; p.H = H; p.I = I; p.keep = keep;
    p.chunks = (T + kRouteThreads - 1) / kRouteThreads;
    const long entries = (long)T * K, segs = entries < E ? entries : E;
    p.blocks_cap = (int)((entries + 127 * segs) / 128);
    p.slots_cap = p.blocks_cap * 128;
    p.units_cap = (int)((p.blocks_cap + segs) / 2);
    const int rows = (int)(entries / (segs > 0 ? segs : 1));
    // Few rows per expert, forward only: weights as the M operand (local_few.cu), 64 rows of an expert at a time, from 41 on average 128.  us, general
    // kernel / local_few.cu, by rows per expert (even routing; in brackets units of 64 and of 128 rows, measured at another time):
    //   H=7168 I=2048, 32 experts, top-8   20 489 / 425   32 507 / 438 (463, 475)   48 523 / 484 (496, 506)   64 534 / 515 (651, 539)   80 545 / 543
    //   H=2048 I=512, 64, top-4            32 103 / 98    48 107 / 108 (106, 107)   51 110 / 113
    //   H=4096 I=1536, 16, top-2           24 129 / 119   48 139 / 139              64 144 / 147   80 147 / 154
    //   H=5120 I=3072, 8, top-2            32 166 / 132   64 178 / 156
    // What an item of the second GEMM stores grows with the rows, what it reads with I (H=4096 I=256, 32 experts, top-2, 37 rows 89 / 85, 62 rows 94 / 102): hence
    // the lines at I / 10 rows up to 40 and at I / 32 up to 64.  Calls of up to 128 tokens are so small that latencies decide: up to 80 rows (H=2048
    // I=256, 8 experts, top-4, 50 rows 39 / 29, H=1024 I=3072, 4, top-2, 32 rows 51 / 37, H=7168 I=768, 16, top-8, 64 rows 139 / 131).  With I >= 4096 it
    // stays at 16 rows: the rows of act that a tile reads are long there (H=1024 I=14336, 4 experts, 48 rows 138 / 131, 64 rows 139 / 149).
    // An expert of more rows than a unit takes its weights again for every unit.  The host cannot see one, but that it matters takes tokens and a
    // large layer: if all T tokens chose the same K experts, K * (T / 64 - 1) units would read 6 H I bytes each.  Up to 128 tokens the kernel chooses units of 64 or 128
    // rows by the routing (wide_units), and with up to 16 rows on average 96 MB are not much: there it is ahead on any routing or close to it.  us, general kernel /
    // local_few.cu: 512 tokens on two experts, H=2048 I=512, 84 MB 49 / 41; H=7168, 128 tokens on two experts, I=2048 87 / 76, I=3072 93 / 96 (the only one of 120 spreads
    // of 80 to 128 tokens, with one more, that was slower by more than 3 %: on eight, I=768 102 / 109, I=1024 117 / 118).  Beyond, the routing decides on
    // the GPU: both kernels are launched, and one returns at once, for 5 us (256 tokens, H=4096 I=768, 64 experts, top-4 268 / 215; all on two experts,
    // H=7168 I=2048 95 / 98).  Units beyond an expert's first may be 1 / few_again of the experts with rows: with 48 rows on average, hottest expert three
    // times the mean, H=7168 I=2048 524 / 512, with 64 543 / 560.
    const bool sixteen = entries <= 16l * E;
    p.few_unit = entries <= 40l * E ? 64 : 128;
    p.few_again = sixteen ? 1 : p.few_unit == 64 ? 3 : 8;
    const long again = (long)K * ((T + 63) / 64 - 1) * 6 * H * I, area = (long)I * E;
    const bool few = sixteen || (I < 4096 && (T <= 128 ? entries <= 80l * E : (entries <= 40l * E && 10 * entries <= area) || (entries <= 64l * E && 32 * entries <= area)));
    p.few = keep || T <= 0 || !few ? 0 : T <= 128 || (sixteen && again <= 96l << 20) ? 1 : 2;
    p.routes = p.few == 1 && entries <= kDirectEntries;
    // Token rows through the loading warps, or copied into slot order first.  The loading warps load a row again for every tile of the other
    // operand, with more energy per byte than TMA; a copy is written and read once.  us of a step, backward by loaders / by copies, by rows per
    // expert:
    //   H=7168 I=2048, 32 experts, top-8   16 1867 / 1662   128 2309 / 2080   256 3141 / 3001   512 4720 / 4683   1024 7861 / 7822
    //   H=7168 I=512, 32, top-8            16 554 / 494     128 689 / 650     256 919 / 916     512 1416 / 1476
    //   H=4096 I=3072, 16, top-2           32 902 / 808     128 1060 / 943    512 2151 / 2086   1024 3386 / 3315
    //   H=4096 I=4096, 16, top-2           32 1172 / 1048   128 1394 / 1248   512 2846 / 2670
    //   H=2048 I=768, 32, top-4            32 279 / 241     128 327 / 306     512 649 / 675
    //   H=4096 I=14336, 8, top-2           128 2385 / 2120  1024 8002 / 7722
    // A forward, by loaders / by copies:
    //   H=7168 I=2048                      17 563 / 561     64 612 / 611      256 994 / 1019    512 1471 / 1507
    //   H=7168 I=512                       17 175 / 177     64 196 / 203      256 308 / 346
    //   H=4096 I=3072                      20 254 / 254     64 279 / 275      256 435 / 434     512 683 / 684
    //   H=4096 I=4096                      20 332 / 333     64 363 / 360      256 571 / 564     512 883 / 884
    //   H=4096 I=14336                     20 583 / 579     128 671 / 655     1024 2614 / 2583
    // Units of a single 128-row block as products of 128 rows, 64 from each CTA, which take half the time of those of 256 (64 and 128 cycles for 256 columns and
    // 16 of K, measured), or with zeros for a second block.  us, zeros / half, by rows per expert: forward (H=7168 I=2048, 32 experts, top-8) 90 670 / 589, 125
    // 736 / 680, 275 1209 / 1129, 325 1187 / 1222, 525 1645 / 1754, 750 1973 / 2026, H=4096 I=1536, 16, top-2 312 307 / 289; steps: 16 1829 / 1715, 64 1972 /
    // 1834, 275 3466 / 3367, 2048 14940 / 15192, H=4096 I=14336, 8, top-2 375 3762 / 3925, H=2048 I=768, 16, top-4 325 284 / 277, H=2048 I=2048, 16, top-8 2048
    // 2277 / 2262, H=2048 I=3072, 16, top-6 3072 5169 / 5136.  Where an expert has whole units besides, a half one runs ahead of them through the weights that
    // they share, and on a long K what it has fetched is gone from L2 before they come: with H=7168 they gain up to 300 rows only.  The other line, H=2048 I=3072, is
    // where the first measurements ended, on the safe side: what lies beyond gains 1 to 9 % more up to about 1000 rows and -1 to 2 % at 1800 (forward, 312 / 550 / 800 rows:
    // H=2048 I=4096 376 / 341, 517 / 491, 678 / 650; H=3072 I=3072 421 / 399, 587 / 559, 739 / 716; H=4096 I=3072 563 / 519, 759 / 748, 944 / 943).
    // The average decides, whatever the routing: with 275 rows on average that all go to 8, 16 or unevenly (Zipf, 1.0) to 32 of 32 experts, H=7168 I=2048, forwards
    // take 780 / 755, 938 / 896, 1047 / 998, steps 2646 / 2623, 2932 / 2838, 3195 / 3107; by every expert's own rows instead it would be 774, 941, 1016 and 2626, 2943, 3130.
    p.halves = entries <= 300l * E || (H <= 2048 && I <= 3072);
    const bool large_i = I >= 4096;
    p.copies[0] = large_i && p.few != 1;          // (local_few.cu gathers rows from x itself)
    p.copies[1] = keep && (large_i || 2 * rows < I);
    // Columns per tile of every GEMM [direction][kind].  The wide tile needs columns for it, enough tiles that every CTA pair gets
    // several, and a mainloop that is long against what it cannot hide: with both accumulators in one tile, the next tile
    // starts when the first half has been read out (in cycles: 2 thousand for a plain store, 3.6 for SwiGLU, 13.5 for its backward), where
    // two 256-column tiles overlap completely.  What the narrow tile lacks is operand bandwidth.  us, wide / narrow (8192 tokens, 16
    // experts, top-8; a forward, or a step in which only this GEMM of the backward changes):
    //   forward's first, by H     512 399 / 455    1024 726 / 791    1536 1070 / 1137   2048 1393 / 1476   4096 2756 / 2992
    //   forward's second, by I    256 728 / 780     512 941 / 1014   1024 1542 / 1646   2048 2823 / 2945
    //   backward's first, by H   1024 2573 / 2512  1536 3489 / 3401  2048 4472 / 4419   3072 6426 / 6373   4096 8257 / 8284
    //   backward's second, by 2I  512 2063 / 2077  1024 2777 / 2873  2048 4405 / 4588   4096 8361 / 8506
    //   weight gradients, by rows per expert   512 1368 / 1346   1024 2303 / 2363   2048 4302 / 4360   4096 8370 / 8368
    // The lines of the forward are on the safe side (wide tiles gain down to H = 512 and I = 256), backward's first is within 1.2 % either way.
    // Number of wide tiles, H=4096 I=2048, 8 experts, top-4, forward: 128 263 / 241, 192 352 / 346, 256 431 / 439, 384 592 / 608.  The number
    // is counted against the whole chip also where total_sms asks for less.
    const int mu_wd = (H + 2 * BM - 1) / (2 * BM), mu_wg = (2 * I + 2 * BM - 1) / (2 * BM);
    auto columns = [&](int n, long row_units, int k, int min_k) {
        return n >= 2 * BN && k >= min_k && row_units * column_blocks(n, 2 * BN) >= kWideTiles ? 2 * BN : BN;
    };
    const long units = entries / (2 * BM);
    p.cols[0][0] = columns(2 * I, units, H, 2048);
    p.cols[0][1] = columns(H, units, I, 1024);
    p.cols[1][0] = columns(I, units, H, 2048);
    p.cols[1][1] = columns(H, units, 2 * I, 1024);
    p.cols[1][2] = columns(I, (long)E * mu_wd, rows, 1024);
    p.cols[1][3] = columns(H, (long)E * mu_wg, rows, 1024);
    p.work_cap[0] = p.few == 1 ? 0 : p.units_cap * (column_blocks(2 * I, p.cols[0][0]) + column_blocks(H, p.cols[0][1]));
    p.work_cap[1] = keep ? p.units_cap * (column_blocks(I, p.cols[1][0]) + column_blocks(H, p.cols[1][1])) +
                               E * (mu_wd * column_blocks(I, p.cols[1][2]) + mu_wg * column_blocks(H, p.cols[1][3]))
                         : 0;
    long at = 0;
    auto take = [&](long n) {
        const long o = at;
        at += (n + 3) / 4 * 4;
        return o;
    };
    const int dirs = keep ? 2 : 1;
    for (int d = 0; d < dirs; ++d) {
        p.stats[d] = take(2 * kLayerStatWords);
        p.sync[d] = take(kSyncWords);
        p.done1[d] = take(p.few ? 2 * p.blocks_cap : p.units_cap);
        p.arrived[d] = take(p.copies[d] ? p.blocks_cap : 0);
        p.done2[d] = take(p.few ? 2 * p.blocks_cap : p.blocks_cap);
    }
    p.zero_words = at;
    p.meta = take(kMetaWords);
    p.counts = take(E);
    p.slot_tk = take(p.slots_cap);
    p.slot_w = take(p.slots_cap);
    p.token_order = take(T);
    p.order_slot = take(entries);
    p.chunk_hist = take((long)p.chunks * E);
    p.chunk_last = take((long)p.chunks * (E + 1));
    for (int d = 0; d < dirs; ++d) p.work[d] = take(4l * p.work_cap[d]);
    p.words = at;
    return p;
}

RouteArgs local_route_args(const LocalLayerParams& q) {
    const LocalLayerPlan& p = q.plan;
    RouteArgs a{};
    a.p = p;
    a.ws = q.ws; a.topk_idx = q.topk_idx; a.is64 = q.idx_is64; a.topk_w = q.topk_w;
    a.nb1[0] = column_blocks(2 * p.I, p.cols[0][0]); a.nb2[0] = column_blocks(p.H, p.cols[0][1]);
    a.nb1[1] = column_blocks(p.I, p.cols[1][0]); a.nb2[1] = column_blocks(p.H, p.cols[1][1]);
    a.mu_wd = (p.H + 2 * BM - 1) / (2 * BM); a.nb_wd = column_blocks(p.I, p.cols[1][2]);
    a.mu_wg = (2 * p.I + 2 * BM - 1) / (2 * BM); a.nb_wg = column_blocks(p.H, p.cols[1][3]);
    a.group_units = q.group_units;
    for (int d = 0; d < 2; ++d) {
        const long full1 = (long)q.group_units * a.nb1[d];       // tiles of a batch's first GEMM
        const long lag_items = std::max<long>((full1 * q.lag_percent + 99) / 100, q.min_lag_items);
        const long lag = std::max<long>(1, (lag_items + full1 - 1) / full1);
        a.lag[d] = (int)lag;
        a.head[d] = (int)std::min(full1, std::max<long>(0, lag_items - (lag - 1) * full1));
    }
    while ((p.E >> a.id_bits) != 0) ++a.id_bits;
    return a;
}

cudaError_t local_layer_route(const LocalLayerParams& q, cudaStream_t stream) {
    const LocalLayerPlan& p = q.plan;
    if (p.E < 1 || p.E > kLocalMaxExperts || p.K < 1 || p.K > 32 || q.group_units <= 0 || q.lag_percent < 0 || q.lag_percent > 100)
        return cudaErrorInvalidValue;
    const RouteArgs a = local_route_args(q);
    // blocks for the lists (tens of thousands of items for a large layer), a third of them for each with keep
    const int grid = p.chunks + (p.few == 1 ? kRouteTableBlocks : p.keep ? 96 : 64);
    const size_t smem = route_words(p.E) * sizeof(int);
    if ((long)p.T * p.K <= kDirectEntries) {
        local_route_assign_kernel<true><<<grid, kRouteThreads, smem, stream>>>(a);
        return cudaGetLastError();
    }
    count_launch();                                       // (callers count one launch)
    local_route_count_kernel<<<p.chunks, kRouteThreads, (2 * p.E + 1) * sizeof(int), stream>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    local_route_assign_kernel<false><<<grid, kRouteThreads, smem, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t local_layer_launch(const LocalLayerParams& q, cudaStream_t stream) {
    const LocalLayerPlan& p = q.plan;
    if (p.few) {
        const cudaError_t e = local_few_launch(q, stream);
        if (p.few == 1 || e != cudaSuccess) return e;
        count_launch();                                   // (callers count one launch)
    }
    const int H = p.H, I = p.I, E = p.E, dir = q.bwd ? 1 : 0;
    if (H % BK != 0 || I % BK != 0 || q.out_rows % BM != 0 || q.out_rows < BM || q.out_rows < p.slots_cap || p.K < 1 || p.K > 32 || (q.bwd && !p.keep))
        return cudaErrorInvalidValue;
    if (reinterpret_cast<uintptr_t>(q.x) % 16 != 0 || reinterpret_cast<uintptr_t>(q.saved_x) % 16 != 0) return cudaErrorInvalidValue;
    const uint64_t R = (uint64_t)q.out_rows;
    LayerArgsP L{};
    cudaError_t e;
    // The tensor-map encoder wants a current context; a thread that has not used the device yet (an autograd worker whose
    // allocations were all served from the cache) has none until the runtime binds it.
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess || (e = cudaSetDevice(dev)) != cudaSuccess) return e;
    Phase& g1 = L.ph[kWorkGemm1];
    Phase& g2 = L.ph[kWorkGemm2];
    g1.nk = H / BK;
    g1.cols = p.cols[dir][0];
    g2.n_total = H; g2.cols = p.cols[dir][1]; g2.num_n_blocks = column_blocks(H, g2.cols);
    const bool copies = p.copies[dir] != 0;
    if (copies && ((e = make_map(&g1.map_a, q.slot_rows, R, H, BK, BM)) != cudaSuccess || (e = make_map(&g1.map_a32, q.slot_rows, R, H, BK, 32)) != cudaSuccess)) return e;
    if (q.bwd && (e = make_map_narrow(&L.st_aux, q.aux, R, 2 * I)) != cudaSuccess) return e;
    if ((e = q.bwd ? make_map_narrow(&L.st_act, q.act, R, I) : make_map(&L.st_act, q.act, R, I, 64, 32)) != cudaSuccess) return e;
    if ((e = make_map(&L.st_y, q.y, R, H, 64, 32)) != cudaSuccess) return e;
    if (!q.bwd) {
        // gate_up: A = token rows, B = W_gateup [E*2I, H] K-major;  down: A = act, B = W_down [E*H, I] K-major
        if ((e = make_map(&g1.map_b, q.w_gateup, (uint64_t)E * 2 * I, H, BK, BN / 2)) != cudaSuccess) return e;
        if ((e = make_map(&g2.map_a, q.act, R, I, BK, BM)) != cudaSuccess || (e = make_map(&g2.map_a32, q.act, R, I, BK, 32)) != cudaSuccess) return e;
        if ((e = make_map(&g2.map_b, q.w_down, (uint64_t)E * H, I, BK, BN / 2)) != cudaSuccess) return e;
        g1.n_total = 2 * I; g1.b_group_rows = 2 * I;
        g2.nk = I / BK; g2.b_group_rows = H;
    } else {
        // grad_act: A = dY, B = W_down MN-major;  dX: A = dGU, B = W_gateup MN-major
        if ((e = make_map_mn(&g1.map_b, q.w_down, (uint64_t)E * H, I)) != cudaSuccess) return e;
        if ((e = make_map(&g2.map_a, q.aux, R, 2 * I, BK, BM)) != cudaSuccess || (e = make_map(&g2.map_a32, q.aux, R, 2 * I, BK, 32)) != cudaSuccess) return e;
        if ((e = make_map_mn(&g2.map_b, q.w_gateup, (uint64_t)E * 2 * I, H)) != cudaSuccess) return e;
        g1.n_total = I; g1.b_group_rows = H;
        g2.nk = 2 * I / BK; g2.b_group_rows = 2 * I;
        // dW_down[e] = dY[seg]^T . act_w[seg]  ([H, I]);  dW_gateup[e] = dGU[seg]^T . X[seg]  ([2I, H])
        Phase& gd = L.ph[kWorkWgradDown];
        Phase& gg = L.ph[kWorkWgradGateup];
        if (copies && (e = make_map_mn(&gd.map_a, q.slot_rows, R, H)) != cudaSuccess) return e;
        if ((e = make_map_mn(&gd.map_b, q.act, R, I)) != cudaSuccess) return e;
        if ((e = make_map_mn(&gg.map_a, q.aux, R, 2 * I)) != cudaSuccess) return e;
        if (copies && (e = make_map_mn(&gg.map_b, q.slot_x, R, H)) != cudaSuccess) return e;
        gd.m_total = H; gd.n_total = I; gd.cols = p.cols[1][2];
        gg.m_total = 2 * I; gg.n_total = H; gg.cols = p.cols[1][3];
        if ((e = make_store_map3(&L.st_dwd, q.dw_down, E, H, I)) != cudaSuccess) return e;
        if ((e = make_store_map3(&L.st_dwg, q.dw_gateup, E, 2 * I, H)) != cudaSuccess) return e;
    }
    g1.num_n_blocks = column_blocks(g1.n_total, g1.cols);
    g1.m_total = g2.m_total = q.out_rows;
    L.T = p.T; L.K = p.K; L.H = H; L.I = I; L.E = E; L.keep = p.keep;
    L.x = static_cast<const uint8_t*>(q.x);
    L.y = static_cast<const __nv_bfloat16*>(q.y);
    L.saved_x = static_cast<__nv_bfloat16*>(q.saved_x);
    L.slot_rows = static_cast<uint8_t*>(q.slot_rows);
    L.slot_x = static_cast<uint8_t*>(q.slot_x);
    L.arrived = q.ws + p.arrived[dir];
    L.out = static_cast<__nv_bfloat16*>(q.out);
    L.preact = static_cast<__nv_bfloat16*>(q.preact);
    L.droute_part = q.droute_part;
    L.n_parts = 2 * ((I + BN - 1) / BN);
    L.dw_topk = q.dw_topk;
    L.meta = q.ws + p.meta;
    L.slot_tk = q.ws + p.slot_tk;
    L.slot_w = reinterpret_cast<const float*>(q.ws + p.slot_w);
    L.token_order = q.ws + p.token_order;
    L.order_slot = q.ws + p.order_slot;
    L.work = reinterpret_cast<const int4*>(q.ws + p.work[dir]);
    L.max_work = p.work_cap[dir];
    L.sync = q.ws + p.sync[dir];
    L.done1 = q.ws + p.done1[dir];
    L.done2 = q.ws + p.done2[dir];
    L.stats = reinterpret_cast<unsigned long long*>(q.ws + p.stats[dir]);
    L.status = q.status;
    L.unless_few = p.few == 2;
    const int sms = default_sms(q.num_sms) & ~1;
    if (sms < 4) return cudaErrorInvalidConfiguration;
    bool wide = false;
    for (int k = 0; k < (q.bwd ? 4 : 2); ++k) wide |= L.ph[k].cols > BN;
    L.stages = wide ? 4 : 6;
    L.clean = (long)p.T * p.K > 224l * E;
    L.halves = p.halves;
    L.stage_bytes = wide ? kWideStageBytes : kNarrowStageBytes;
    if (q.bwd) return copies ? launch<true, false>(L, sms, stream) : launch<true, true>(L, sms, stream);
    return copies ? launch<false, false>(L, sms, stream) : launch<false, true>(L, sms, stream);
}

}  // namespace tmoe
