// The layer's forward on one rank when experts have few rows (local_layer_plan decides), as in decoding: the time is that of reading the
// weights once.  The weights are the M operand here, 128 rows of a tile, and an expert's tokens the N operand, 16 to 64 or 128 columns.  With the
// roles of local_layer.cu eight tokens were multiplied as 256 rows; under the power cap, which such a call reaches too, the tensor
// cores' share is bandwidth lost.  Forward of 32 tokens, H=7168 I=2048, 32 experts, top-8: 585 -> 430 us, 6.6 TB/s, which is what a plain
// copy reaches; of 64 tokens 588 -> 437; with I=512 179 -> 132 and 185 -> 134; of 128 and 256 tokens (32 and 64 rows per expert) 507 -> 438 and
// 534 -> 515: every step brings a unit's rows from L2 next to the weights, half as many bytes again at 64 rows, which is what the time grows by.
//
// One persistent block per SM, no clusters.  Items: first the tiles of the first GEMM (128 rows of W_gateup of an expert x a unit of up to
// 64 or 128 of its tokens), then those of the second, dealt out in turn: they nearly cost the same.  Units of one expert are neighbours, so that
// they share the tile of weights in L2.
//   warp 0     loads: weights by TMA boxes, the second GEMM's rows by boxes of 16
//   warps 2, 3 load the first GEMM's token rows, every other step each, by cp.async
//   warp 1     issues tcgen05.mma, 128 x N x 16, into one of four accumulators
//   warps 4-7  epilogue: a lane holds one row of weights, so gate and up of a token sit in neighbouring lanes
//   warps 2-7  at the end of their items: sums of the tokens' expert rows, in the order of their entries
// Nine stages of 24 KB keep 144 KB of weights per SM on their way; with units of 128 rows, six of 32 KB keep 96 KB, which costs 2 to 4 % where experts
// have few rows (32 tokens as above 430 / 449) and saves reading weights again where many have more than 64 (256 tokens 651 / 539).  wide_units chooses.
//
// Where the host can tell that this kernel takes the call (LocalLayerPlan::routes) it makes the routing tables too, in front of a barrier of the whole grid:
// a kernel of their own costs 5 us, and a boundary between two kernels of a stream up to 2 us more.  us of a forward, routing kernel / here / here with the
// first weights on their way meanwhile: one token, H=2048 I=768, 16 experts, top-4 28.7 / 26.7 / 26.7, 30, H=1024 I=512, 8, top-2 24.6 / 22.6 / 22.6,
// 64, H=7168 I=512, 32, top-8 138 / 136 / 133, 400, H=1024 I=256, 64, top-2 37.0 / 35.7 / 34.9.
#include "local_layer.h"

#include <cooperative_groups.h>

#include "gemm_common.cuh"
#include "layer.h"
#include "local_route.cuh"

namespace tmoe {

using namespace detail;

namespace {

constexpr int kFewAccs = 4;
constexpr int kFewThreads = 256;
constexpr int kFewEpiWarps = 4;
constexpr int kFewSumWarps = 6;
constexpr long kFewReadAgain = 64l << 20;                                 // wide_units

// Shared memory: the operand stages, barriers, [experts + 1] first unit, [experts] rows, [experts] first slot
template <int UNIT>
struct Few {
    static constexpr int kStageBytes = kAStageBytes + UNIT * BK * 2;      // 24 KB, 32 KB
    static constexpr int kStages = UNIT == 64 ? 9 : 6;
    static_assert(UNIT % 64 == 0 && 128 % UNIT == 0 && kFewAccs * UNIT <= 512, "units");
};
constexpr int kFewMostStages = Few<64>::kStages;
constexpr int kFewBarOffset = kFewMostStages * Few<64>::kStageBytes;
constexpr int kFewUnitsOffset = kFewBarOffset + 256;
constexpr int kFewSmemBytes = kFewUnitsOffset + (3 * kLocalMaxExperts + 1) * 4 + 1024;
static_assert(Few<128>::kStages * Few<128>::kStageBytes <= kFewBarOffset, "stages");
static_assert(8 * (2 * kFewMostStages + 2 * kFewAccs) <= 240 && kFewSmemBytes <= 232448, "shared memory");
// The routing works in the last stages, before they are loaded.
constexpr int kFewRouteOffset = 7 * Few<64>::kStageBytes;
static_assert(kFewRouteOffset + route_words(kLocalMaxExperts) * 4 <= kFewBarOffset && kFewThreads == kRouteThreads, "routing");

struct FewArgs {
    alignas(64) CUtensorMap map_wg, map_wd, map_act;
    const uint8_t* x;
    int T, K, H, I, E;
    __nv_bfloat16* act;
    __nv_bfloat16* y;
    __nv_bfloat16* out;
    const int* counts;
    const int* slot_tk;
    const float* slot_w;
    const int* token_order;
    const int* order_slot;
    int* done1;                          // per 64 slots: epilogue warps that finished a tile of the first GEMM
    int* done2;                          // the same for the second
    unsigned long long* stats;
    int* status;
    int* ran_unit;                       // for whoever asks: rows of a unit
    const int* wanted;                   // the routing's word for this kernel; null: it takes the call
};

struct FewItem {
    int second, expert, tile, slot0, rows, n;      // n: columns of the accumulator that are computed
};

// What both kernels have in shared memory
struct FewShared {
    uint32_t base, bars;
    uint8_t* gen;
    volatile uint32_t* words;                // [0] address in tensor memory, [1] abort flag, [2] rows of a unit
    int *units, *counts, *seg;

    __device__ __forceinline__ FewShared(uint8_t* raw, int E) {
        base = (smem_u32(raw) + 1023u) & ~1023u;
        gen = raw + (base - smem_u32(raw));
        bars = base + kFewBarOffset;
        words = reinterpret_cast<volatile uint32_t*>(gen + kFewBarOffset + 240);
        units = reinterpret_cast<int*>(gen + kFewUnitsOffset);
        counts = units + E + 1;
        seg = counts + E;
    }
    __device__ __forceinline__ uint32_t full_bar(int s) const { return bars + 8u * s; }
    __device__ __forceinline__ uint32_t empty_bar(int s) const { return bars + 8u * (kFewMostStages + s); }
    __device__ __forceinline__ uint32_t tfull_bar(int a) const { return bars + 8u * (2 * kFewMostStages + a); }
    __device__ __forceinline__ uint32_t tempty_bar(int a) const { return bars + 8u * (2 * kFewMostStages + kFewAccs + a); }

    __device__ __forceinline__ void init(const FewArgs& L) const {
        words[1] = 0u;
        for (int s = 0; s < kFewMostStages; ++s) {
            mbar_init(full_bar(s), 1 + 32);                  // the producer, and every lane of a loading warp
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < kFewAccs; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), kFewEpiWarps);
        }
        fence_mbar_init();
        tma_prefetch_desc(&L.map_wg);
        tma_prefetch_desc(&L.map_wd);
        tma_prefetch_desc(&L.map_act);
    }
    // One warp: units of 64 or 128 rows and slots of every expert, from its rows
    __device__ __forceinline__ void lay_out(const int* rows, int E, int unit, int lane) const {
        const int log_unit = unit == 64 ? 6 : 7;
        int run = 0, run_s = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane, c = e < E ? rows[e] : 0, own = (c + unit - 1) >> log_unit, own_s = (c + 127) & ~127;
            int v = own, s = own_s;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o), us = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) {
                    v += u;
                    s += us;
                }
            }
            if (e < E) {
                units[e] = run + v - own;
                counts[e] = c;
                seg[e] = run_s + s - own_s;
            }
            run += __shfl_sync(0xffffffffu, v, 31);
            run_s += __shfl_sync(0xffffffffu, s, 31);
        }
        if (lane == 0) units[E] = run;
    }
};

// The layer, once the units are known.  ROUTES: the tables are being written; counts_only: not by this block.  (The body of the kernels, for each size of a unit.)
template <int UNIT, bool ROUTES>
__device__ __forceinline__ void few_layer(const FewArgs& L, const FewShared& sh, uint32_t tmem_base, bool counts_only) {
    constexpr int kUnit = UNIT, kFewStages = Few<UNIT>::kStages, kFewStageBytes = Few<UNIT>::kStageBytes;
    const uint32_t smem_base = sh.base;
    auto full_bar = [&](int s) { return sh.full_bar(s); };
    auto empty_bar = [&](int s) { return sh.empty_bar(s); };
    auto tfull_bar = [&](int a) { return sh.tfull_bar(a); };
    auto tempty_bar = [&](int a) { return sh.tempty_bar(a); };
    volatile uint32_t* abort_flag = sh.words + 1;
    const int *units = sh.units, *counts = sh.counts, *seg = sh.seg;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, E = L.E;

    const int n1 = 2 * L.I / BM, n2 = (L.H + BM - 1) / BM, U = units[E], items = U * (n1 + n2);
    auto decode = [&](int i) {
        FewItem q;
        q.second = i >= U * n1;
        const int n = q.second ? n2 : n1, j = q.second ? i - U * n1 : i;
        int lo = 0, hi = E;                          // the expert: units[lo] * n <= j < units[lo + 1] * n
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (units[mid] * n <= j) lo = mid;
            else hi = mid;
        }
        const int of_expert = units[lo + 1] - units[lo], r = j - units[lo] * n;
        q.expert = lo;
        q.tile = r / of_expert;
        const int row0 = (r - q.tile * of_expert) * kUnit;
        q.slot0 = seg[lo] + row0;
        q.rows = min(kUnit, counts[lo] - row0);
        q.n = (q.rows + 15) & ~15;
        return q;
    };
    const int nk1 = L.H / BK, nk2 = L.I / BK;
    int primed = 0;                                              // steps of this block's first item whose weights are on their way
    if constexpr (ROUTES) {
        // Blocks that do not write the tables have the weights of their first item on their way while they wait for them.
        fence_proxy_async_smem();                                // what the routing wrote is written over by copies
        if (counts_only && (int)blockIdx.x < U * n1) {
            primed = min(nk1, kFewRouteOffset / kFewStageBytes);
            if (warp == 0 && lane == 0) {
                const FewItem q = decode(blockIdx.x);
                for (int s = 0; s < primed; ++s) {
                    mbar_arrive_expect_tx(full_bar(s), kAStageBytes);
                    tma_load_2d(smem_base + s * kFewStageBytes, &L.map_wg, full_bar(s), s * BK, q.expert * 2 * L.I + q.tile * BM);
                }
            }
            __syncwarp();
        }
        cooperative_groups::this_grid().sync();
    }

    if (warp == 0) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        uint64_t waited = 0;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const FewItem q = decode(i);
            const int nk = q.second ? nk2 : nk1, boxes = q.n / 16;
            const int w_row = q.second ? q.expert * L.H + q.tile * BM : q.expert * 2 * L.I + q.tile * BM;
            const CUtensorMap* map_w = q.second ? &L.map_wd : &L.map_wg;
            const uint32_t tx = (uint32_t)(kAStageBytes + (q.second ? boxes * 16 * BK * 2 : 0));
            auto weights = [&](int s, uint32_t ph, int kb) {
                if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, L.status, 680)) return false;
                if (lane == 0) {
                    if (q.second) mbar_arrive_n(full_bar(s), 32);            // for the loading warp
                    mbar_arrive_expect_tx(full_bar(s), tx);
                    tma_load_2d(smem_base + s * kFewStageBytes, map_w, full_bar(s), kb * BK, w_row);
                }
                __syncwarp();
                return true;
            };
            // the weights of a second GEMM's first steps come while its rows are waited for
            int early = i == (int)blockIdx.x ? primed : 0;
            if (q.second) {
                const int* flag = L.done1 + q.slot0 / kUnit;
                int ready = lane == 0 ? ld_acquire_gpu(flag) >= kFewEpiWarps * n1 : 0;
                ready = __shfl_sync(0xffffffffu, ready, 0);
                if (!ready) {
                    int s = stage;
                    uint32_t ph = phase;
                    for (; early < min(kFewStages, nk); ++early) {
                        if (!(ok = weights(s, ph, early))) break;
                        if (++s == kFewStages) { s = 0; ph ^= 1u; }
                    }
                    if (!ok) break;
                    // (a wait that runs out is reported, and the item carried through on whatever its rows hold)
                    if (lane == 0) {
                        const uint64_t t0 = globaltimer_ns();
                        wait_count_gpu(flag, kFewEpiWarps * n1, L.status, 681, 64);
                        waited += globaltimer_ns() - t0;
                    }
                }
                __syncwarp();
                fence_proxy_async_all();                         // stores of other SMs -> async-proxy reads
            }
            for (int kb = 0; kb < nk; ++kb) {
                if (kb >= early && !(ok = weights(stage, phase, kb))) break;
                const uint32_t dst = smem_base + stage * kFewStageBytes + kAStageBytes;
                if (q.second && lane < boxes) tma_load_2d(dst + lane * 16 * BK * 2, &L.map_act, full_bar(stage), kb * BK, q.slot0 + 16 * lane);
                if (++stage == kFewStages) { stage = 0; phase ^= 1u; }
            }
        }
        if (waited != 0) atomicAdd(L.stats + kStatWaitFirstGemm, (unsigned long long)waited);
        if (!ok)                                                 // (no barrier says when the copies under way have landed: microseconds)
            for (const uint64_t t0 = globaltimer_ns(); globaltimer_ns() - t0 < 10000000ull;) __nanosleep(1000);
    } else if (warp == 1) {
        int stage = 0, acc = 0;
        uint32_t phase = 0, acc_phase = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const FewItem q = decode(i);
            const int nk = q.second ? nk2 : nk1;
            const uint32_t idesc = make_idesc_bf16(BM, q.n, false, false);
            if (!(ok = mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag, L.status, 682))) break;
            tcgen05_fence_after();
            for (int kb = 0; kb < nk; ++kb) {
                if (!(ok = mbar_wait(full_bar(stage), phase, abort_flag, L.status, 683))) break;
                tcgen05_fence_after();
                if (elect_one()) {
                    if (!q.second) fence_proxy_async_smem();     // rows that the loading warps' copies wrote -> async-proxy reads
                    const uint32_t at = smem_base + stage * kFewStageBytes;
                    const uint64_t a = make_smem_desc_sw128(at, 0, 1024), b = make_smem_desc_sw128(at + kAStageBytes, 0, 1024);
#pragma unroll
                    for (int k = 0; k < BK / UK; ++k)
                        umma_bf16_ss(tmem_base + acc * kUnit, a + k * (UK * 2 >> 4), b + k * (UK * 2 >> 4), idesc, (kb | k) != 0 ? 1u : 0u);
                    umma_commit(empty_bar(stage));
                    if (kb == nk - 1) umma_commit(tfull_bar(acc));
                }
                __syncwarp();
                if (++stage == kFewStages) { stage = 0; phase ^= 1u; }
            }
            if (++acc == kFewAccs) { acc = 0; acc_phase ^= 1u; }
        }
    } else if (warp < 4) {
        // Token rows.  Eight lanes copy 128 bytes of a row, in the layout that TMA gives the weights; a warp's arrive follows its copies by itself.
        // (Handed over behind the copies of the next step, as in local_layer.cu, fewer would be under way: us, so / here, 32 tokens, H=7168 I=2048,
        // 32 experts, top-8 449 / 433; where items have few steps it is the other way round, 21 tokens, H=512 I=4096, 16 experts 66 / 69.)
        // The second GEMM's items are all behind the first's; there the producer arrives for it.
        // TMA's row gather takes 70 cycles for four rows, 1120 for a unit of 64, where a step's weights take 720: with experts of unequal
        // load the few SMs that had the tiles of a large one came last.  us, general kernel / row gather / this: 64 tokens, H=7168 I=512, 32
        // experts, top-8, hottest expert 20 rows 179 / 149 / 137, 63 rows 179 / 195 / 137, all on 8 experts 90 / 122 / 70.
        const int sub = lane >> 3, chunk = lane & 7;
        const uint32_t at[2] = {(uint32_t)(sub * 128 + ((chunk ^ sub) << 4)), (uint32_t)(sub * 128 + ((chunk ^ (sub + 4)) << 4))};      // rows 8j + sub, 8j + 4 + sub
        int step = warp - 2, stage = step;                       // this warp's next step, counted from the start of the item; its stage
        uint32_t phase = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < U * n1 && ok; i += gridDim.x) {
            const FewItem q = decode(i);
            const int quads = (q.rows + 3) / 4;
            // of rows 4 j + sub, which this lane copies pieces of; past the last row that one again, whose copies nobody reads (of all SMs the same row would be
            // one hot line of L2).  Asking the other lanes in every step instead, with units of 128 rows the loading warps are what the step waits for: 128 tokens on the
            // same eight experts, H=7168 I=768, first GEMM 60 / 53 us.
            int token[kUnit / 4];
#pragma unroll
            for (int c = 0; c < kUnit / 32; ++c) {
                const int t = L.slot_tk[q.slot0 + min(lane + 32 * c, q.rows - 1)] / L.K;
#pragma unroll
                for (int j = 0; j < 8; ++j) token[8 * c + j] = __shfl_sync(0xffffffffu, t, 4 * j + sub);
            }
            for (; step < nk1; step += 2) {
                if (!(ok = mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, L.status, 686))) break;
                const uint32_t dst = smem_base + stage * kFewStageBytes + kAStageBytes;
                const uint8_t* src = L.x + step * (BK * 2) + 16 * chunk;
                auto copy = [&](int j) {
                    cp_async_16(dst + j * 512 + at[j & 1], src + (long)token[j] * (L.H * 2l));
                };
                if (quads <= 4) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < quads) copy(j);
                } else {
                    // 16 rows with no branch between the copies, so that they follow each other (the last example 85 -> 70 us)
#pragma unroll
                    for (int g = 0; g < kUnit / 16; ++g) {
                        if (4 * g >= quads) break;
#pragma unroll
                        for (int j = 0; j < 4; ++j) copy(4 * g + j);
                    }
                }
                cp_async_arrive(full_bar(stage));
                stage += 2;
                if (stage >= kFewStages) { stage -= kFewStages; phase ^= 1u; }
            }
            step -= nk1;
        }
        cp_async_wait_all();
    } else {
        const int quarter = warp & 3;
        int acc = 0;
        uint32_t acc_phase = 0;
        const bool stamps = warp == 4 && lane == 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x) {
            const FewItem q = decode(i);
            // (the clock is read for the first and the last item of a kind only)
            const bool ends = i + (int)gridDim.x >= (q.second ? items : U * n1);
            if (stamps && i - (int)gridDim.x < (q.second ? U * n1 : 0))
                atomicMax(L.stats + kStatKindFirst + (q.second ? kWorkGemm2 : kWorkGemm1), ~globaltimer_ns());
            float w[kUnit / 32];
#pragma unroll
            for (int c = 0; c < kUnit / 32; ++c) w[c] = !q.second && lane + 32 * c < q.rows ? L.slot_w[q.slot0 + lane + 32 * c] : 0.f;
            if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag, L.status, 684)) break;
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * kUnit);
#pragma unroll
            for (int c = 0; c < kUnit / 32; ++c) {
                if (c * 32 >= q.rows) break;
                uint32_t v[32];
                tmem_ld_x32(taddr + c * 32, v);
                tmem_ld_wait();
                if (q.second) {
                    const int h = q.tile * BM + quarter * 32 + lane;
                    __nv_bfloat16* y = L.y + (long)(q.slot0 + c * 32) * L.H + h;
#pragma unroll
                    for (int r = 0; r < 32; ++r)
                        if (c * 32 + r < q.rows && h < L.H) y[(long)r * L.H] = __float2bfloat16_rn(__uint_as_float(v[r]));
                } else {
                    // lanes 2j and 2j + 1 hold gate and up of column j: of two tokens each lane takes one
                    const int odd = lane & 1;
                    __nv_bfloat16* act = L.act + (long)(q.slot0 + c * 32 + odd) * L.I + q.tile * (BM / 2) + quarter * 16 + (lane >> 1);
#pragma unroll
                    for (int r = 0; r < 32; r += 2) {
                        const float mine = __uint_as_float(odd ? v[r + 1] : v[r]);
                        const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? v[r] : v[r + 1]), 1);
                        const float route = __shfl_sync(0xffffffffu, w[c], r + odd);
                        const float gt = odd ? other : mine, up = odd ? mine : other;
                        const float a = __fdividef(gt, 1.f + __expf(-gt)) * up * route;
                        if (c * 32 + r + odd < q.rows) act[(long)r * L.I] = __float2bfloat16_rn(a);
                    }
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(tempty_bar(acc));
                fence_acq_rel_gpu();
                red_add_gpu((q.second ? L.done2 : L.done1) + q.slot0 / kUnit, 1);
            }
            if (stamps && ends) atomicMax(L.stats + kStatKindLast + (q.second ? kWorkGemm2 : kWorkGemm1), globaltimer_ns());
            if (++acc == kFewAccs) { acc = 0; acc_phase ^= 1u; }
        }
    }
    __syncwarp();

    if (warp >= 2) {
        // sums: (token, 256 columns) per task.  The loading warps wait for the epilogue: looking at counters during the second GEMM would slow it down
        // (64 tokens, H=7168 I=512, 32 experts, top-8 137 -> 150 us).
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kFewSumWarps) : "memory");
        const int nvec = L.H / 8, parts = (nvec + 31) / 32, tasks = L.T * parts, K = L.K;
        const bool stamps = warp == 2 && lane == 0;              // (one warp's clock: atomics of all of them would be a microsecond of a small call)
        uint64_t waited = 0, counted = 0;
        for (int task = (warp - 2) * (int)gridDim.x + (int)blockIdx.x; task < tasks; task += kFewSumWarps * (int)gridDim.x) {
            const int place = task / parts, col = (task - place * parts) * 32 + lane, at = min(col, nvec - 1);
            const int t = L.token_order[place], slot = lane < K ? L.order_slot[(long)place * K + lane] : -1;
            const uint32_t valid = __ballot_sync(0xffffffffu, slot >= 0);
            if (!wait_counts_warp(L.done2 + max(slot, 0) / kUnit, slot >= 0, kFewEpiWarps * n2, L.status, 685, waited)) break;      // reported: unwind
            __syncwarp();                                        // every lane reads behind the other lanes' acquires
            float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int k0 = 0; k0 < K; k0 += 8) {
                int4 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int s = max(0, __shfl_sync(0xffffffffu, slot, (k0 + j) & 31));
                    // (volatile keeps the load behind the acquire loads above)
                    if (k0 + j < K)
                        asm volatile("ld.global.cg.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v[j].x), "=r"(v[j].y), "=r"(v[j].z), "=r"(v[j].w)
                                     : "l"(reinterpret_cast<const int4*>(L.y) + (long)s * nvec + at));
                }
                if (stamps && k0 == 0) {                         // while the loads are under way: reading the clock takes long, and this may be the end
                    const uint64_t now = globaltimer_ns();
                    atomicMax(L.stats + kStatKindFirst + kWorkReduce, ~now);
                    atomicMax(L.stats + kStatKindLast + kWorkReduce, now);
                    if (waited != counted) atomicAdd(L.stats + kStatWaitLanded, (unsigned long long)(waited - counted));
                    counted = waited;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (k0 + j >= K || !((valid >> (k0 + j)) & 1u)) continue;
                    const uint32_t p[4] = {(uint32_t)v[j].x, (uint32_t)v[j].y, (uint32_t)v[j].z, (uint32_t)v[j].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = unpack_bf16x2(p[i]);
                        sum[2 * i] += f.x;
                        sum[2 * i + 1] += f.y;
                    }
                }
            }
            if (col < nvec)
                reinterpret_cast<int4*>(L.out + (long)t * L.H)[col] = make_int4((int)pack_bf16x2(sum[0], sum[1]), (int)pack_bf16x2(sum[2], sum[3]),
                                                                                (int)pack_bf16x2(sum[4], sum[5]), (int)pack_bf16x2(sum[6], sum[7]));
        }
    }
}

// All units of UNIT rows, tables by a routing kernel
template <int UNIT>
__global__ void __launch_bounds__(kFewThreads, 1) local_few_kernel(const __grid_constant__ FewArgs L) {
    if (L.wanted != nullptr && *L.wanted == 0) return;
    extern __shared__ uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const FewShared sh(smem_raw, L.E);
    if (threadIdx.x == 0) sh.init(L);
    if (warp == 2) tmem_alloc(smem_u32((const void*)sh.words), kFewAccs * UNIT);
    if (warp == 1) sh.lay_out(L.counts, L.E, UNIT, lane);
    if (threadIdx.x == 0 && blockIdx.x == 0) *L.ran_unit = UNIT;
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = sh.words[0];
    few_layer<UNIT, false>(L, sh, tmem_base, false);
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, kFewAccs * UNIT);
    }
}

// Whether units of 128 rows take less time than those of 64, by one warp from the entries per expert.  With 64 an expert of more rows has its weights multiplied
// again, from L2; with 128 there are fewer tiles, which may not fill the blocks, and a step of K takes longer: 0.62 + 1.1 rows / 128 of one with 64 rows at most (a
// first GEMM of one turn, H=7168 I=768, 64 / 80 / 96 / 112 / 128 rows 37 / 43 / 44 / 51 / 53 us).  Compared are the steps of a block: whole turns of its tiles through the grid and
// as they would be dealt out evenly, half and half, as a last turn runs next to the second GEMM.  us of a forward, H=7168, general kernel / 64 / 128, tokens all
// on as many experts as they have entries:
//   128, I=512, top-8   95 / 82 / 97     I=768, 8   101 / 109 / 105     I=768, 4   84 / 74 / 84      I=2048, 8   200 / 222 / 177     I=2048, 4   113 / 114 / 112
//    96, I=768, top-8   97 / 107 / 91    80, I=3072, 8  275 / 318 / 219                  128 on ten of 32, top-8, I=768 111 / 119 / 104, I=2048 227 / 270 / 206
//   128 evenly on eight, top-4, I=1024 106 / 100 / 89, I=3072 262 / 232 / 211; on sixteen, top-8, I=2048 334 / 338 / 284
// Below 64 MB the weights that are read again cost less than the larger unit's steps (H=2048 I=512, 128 on ten of 32, top-8, 60 MB 52 / 43 / 50).
__device__ __forceinline__ bool wide_units(const FewArgs& L, const int* totals, int lane) {
    uint32_t all = 0, most = 0, narrow = 0, wide = 0;
    for (int e = lane; e < L.E; e += 32) {
        const uint32_t n = (uint32_t)totals[e];
        all += n;
        most = max(most, n);
        narrow += (n + 63) / 64;
        wide += (n + 127) / 128;
    }
    narrow = __reduce_add_sync(0xffffffffu, narrow);
    wide = __reduce_add_sync(0xffffffffu, wide);
    all = __reduce_add_sync(0xffffffffu, all);
    most = __reduce_max_sync(0xffffffffu, most);
    const float blocks = (float)gridDim.x, rows = 0.5f * (min(most, 128u) + (float)all / wide);
    auto steps = [&](uint32_t units) {
        auto turns = [&](int tiles) {
            const float n = (float)(units * tiles) / blocks;
            return 0.5f * (ceilf(n) + fmaxf(n, 1.f));
        };
        return turns(2 * L.I / BM) * (L.H / BK) + turns((L.H + BM - 1) / BM) * (L.I / BK);
    };
    return (narrow - wide) * 6l * L.H * L.I > kFewReadAgain && steps(wide) * (0.62f + 1.1f * rows / 128.f) < steps(narrow);
}

// Routing in the same launch: a few blocks write the tables, the others only count.  All know the units then.
__global__ void __launch_bounds__(kFewThreads, 1) local_few_routes_kernel(const __grid_constant__ FewArgs L, const __grid_constant__ RouteArgs R) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ int bound[4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, E = L.E;
    const FewShared sh(smem_raw, E);
    if (threadIdx.x == 0) sh.init(L);
    if (warp == 2) tmem_alloc(smem_u32((const void*)sh.words), 512);
    int* route = reinterpret_cast<int*>(sh.gen + kFewRouteOffset);
    int* totals = route + route_totals(E);
    clear_counters(R);
    const int blocks = R.p.chunks + kRouteTableBlocks;
    const bool counts_only = (int)blockIdx.x >= blocks;
    if (counts_only) {
        for (int i = threadIdx.x; i < 2 * E + 1; i += kFewThreads) totals[i] = 0;
        __syncthreads();
        count_entries(R, totals, nullptr, 0);
    }
    for (int b = blockIdx.x; b < blocks; b += gridDim.x) {
        __syncthreads();
        route_assign<true>(R, route, bound, b, blocks);
    }
    __syncthreads();
    if (warp == 1) {
        const bool wide = wide_units(L, totals, lane);
        sh.lay_out(totals, E, wide ? 128 : 64, lane);
        if (lane == 0) {
            sh.words[2] = wide ? 128u : 64u;
            if (blockIdx.x == 0) *L.ran_unit = wide ? 128 : 64;
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = sh.words[0];
    if (sh.words[2] == 64u) few_layer<64, true>(L, sh, tmem_base, counts_only);
    else few_layer<128, true>(L, sh, tmem_base, counts_only);
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <typename... Args>
cudaError_t launch(void (*kernel)(Args...), bool (&configured)[64], int num_sms, cudaStream_t stream, const Args&... args) {
    if (cudaError_t e = ensure_smem_limit(kernel, kFewSmemBytes, configured); e != cudaSuccess) return e;
    const int sms = default_sms(num_sms) & ~1;
    if (sms < 4) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms);
    cfg.blockDim = dim3(kFewThreads);
    cfg.dynamicSmemBytes = kFewSmemBytes;
    cfg.stream = stream;
    // blocks wait for tiles of other blocks: all of them have to be resident
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

cudaError_t local_few_launch(const LocalLayerParams& q, cudaStream_t stream) {
    const LocalLayerPlan& p = q.plan;
    const int H = p.H, I = p.I, E = p.E;
    if (q.group_units <= 0 || q.lag_percent < 0 || q.lag_percent > 100) return cudaErrorInvalidValue;
    if (!p.few || q.bwd || H % BK != 0 || I % BK != 0 || q.out_rows < p.slots_cap || p.K < 1 || p.K > 32 || E < 1 || E > kLocalMaxExperts)
        return cudaErrorInvalidValue;
    if (reinterpret_cast<uintptr_t>(q.x) % 16 != 0) return cudaErrorInvalidValue;
    int dev = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess || (e = cudaSetDevice(dev)) != cudaSuccess) return e;      // (the tensor-map encoder wants a current context)
    FewArgs L{};
    if ((e = make_map(&L.map_wg, q.w_gateup, (uint64_t)E * 2 * I, H, BK, BM)) != cudaSuccess) return e;
    if ((e = make_map(&L.map_wd, q.w_down, (uint64_t)E * H, I, BK, BM)) != cudaSuccess) return e;
    if ((e = make_map(&L.map_act, q.act, q.out_rows, I, BK, 16)) != cudaSuccess) return e;
    L.T = p.T; L.K = p.K; L.H = H; L.I = I; L.E = E;
    L.x = static_cast<const uint8_t*>(q.x);
    L.act = static_cast<__nv_bfloat16*>(q.act);
    L.y = static_cast<__nv_bfloat16*>(q.y);
    L.out = static_cast<__nv_bfloat16*>(q.out);
    L.counts = q.ws + p.counts;
    L.slot_tk = q.ws + p.slot_tk;
    L.slot_w = reinterpret_cast<const float*>(q.ws + p.slot_w);
    L.token_order = q.ws + p.token_order;
    L.order_slot = q.ws + p.order_slot;
    L.done1 = q.ws + p.done1[0];
    L.done2 = q.ws + p.done2[0];
    L.stats = reinterpret_cast<unsigned long long*>(q.ws + p.stats[0]);
    L.status = q.status;
    L.ran_unit = q.ws + p.meta + kMetaFewUnit;
    L.wanted = p.few == 2 ? q.ws + p.meta + kMetaFew : nullptr;
    static bool configured[3][64] = {};
    if (p.routes) return launch(local_few_routes_kernel, configured[0], q.num_sms, stream, L, local_route_args(q));
    return p.few_unit == 64 ? launch(local_few_kernel<64>, configured[1], q.num_sms, stream, L)
                            : launch(local_few_kernel<128>, configured[2], q.num_sms, stream, L);
}

}  // namespace tmoe
