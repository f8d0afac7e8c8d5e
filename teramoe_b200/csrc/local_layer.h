// The MoE layer on one rank (local_layer.cu): routing preparation in one launch or two (by the number of entries), then ONE cooperative persistent kernel per
// direction; a forward with few rows per expert has its own (local_few.cu), which with up to 4096 entries prepares the routing itself.  Every sum has the terms and the order that it has in the kernel
// for several ranks (layer.h), so both give the same bits; what differs is where batches of the work list end, slices of K that are
// all padding, and everything that only a second rank needs (peer tables, completion flags, landing rows).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tmoe {

constexpr int kLocalMaxExperts = 512;    // the routing kernels keep 23 words per expert in shared memory

// words of the meta block
enum { kMetaUnits = 0, kMetaSlots = 1, kMetaWork = 2, kMetaRows = 4, kMetaFew = 5, kMetaFewUnit = 6, kMetaWords = 8 };

// Word offsets of the tables of one call inside its int32 workspace.  Capacities follow from the sizes alone (T * K entries in
// at most min(E, T * K) segments padded to 128 rows), so the host never has to read the layout back.
struct LocalLayerPlan {
    int T, K, E, H, I, keep;             // keep: tables of the backward pass too
    int copies[2];                       // per direction: token rows are copied into slot order, not loaded by the slot table
    int few;                             // a forward with few rows per expert: 1 local_few.cu, 2 local_few.cu if the routing says so (kMetaFew)
    int few_unit;                        // rows of an expert that it multiplies at a time: 64 or 128; with `routes` it chooses itself
    int few_again;                       // with few = 2: most units beyond an expert's first, as a share of the experts with rows: 1 / few_again
    int routes;                          // local_few.cu makes the routing tables itself: there is no routing kernel
    int halves;                          // units of one 128-row block are multiplied as 128 rows
    int chunks;                          // blocks of the routing kernels
    int slots_cap, blocks_cap, units_cap;
    int work_cap[2];                     // items of the forward / backward list
    int cols[2][4];                      // columns per tile: [direction][first GEMM, second GEMM, dW_down, dW_gateup]
    // zero-filled by local_layer_route, or with `routes` by local_few.cu
    long stats[2], sync[2], done1[2], done2[2], arrived[2], zero_words;
    // written by the same
    long meta, counts, slot_tk, slot_w, token_order, order_slot, chunk_hist, chunk_last, work[2], words;
};
LocalLayerPlan local_layer_plan(int T, int K, int E, int H, int I, int keep);

struct LocalLayerParams {
    LocalLayerPlan plan;
    int* ws;                             // plan.words int32
    const void* topk_idx;
    int idx_is64;
    const float* topk_w;                 // forward
    // schedule
    int group_units, lag_percent, min_lag_items, num_sms;
    int bwd;
    const void* x;                       // [T, H] forward x, backward grad_out
    const void* w_gateup;
    const void* w_down;
    void* y;                             // [out_rows, H] second GEMM's output in slot order
    int out_rows;                        // rows of the slot-order tensors: max(slots_cap, 128)
    void* act;                           // forward act, backward act x route [out_rows, I]
    void* aux;                           // backward dGU [out_rows, 2I]
    void* saved_x;                       // [T, H] copy of x: written by forward (may be null), read by backward
    void* out;                           // [T, H]
    void* preact;                        // written by forward (with keep), read by backward: 2I * out_rows values in 32 x 8 blocks
    void* slot_rows;                     // with plan.copies: rows of x in slot order [out_rows, H], backward also of saved_x
    void* slot_x;
    // backward
    float* droute_part;                  // [out_rows, 2 * ceil(I / 256)]
    float* dw_topk;                      // [T, K]
    void* dw_gateup;
    void* dw_down;
    int* status;
};

// Routing tables and both work lists (p: plan, ws, topk_*, schedule).  Not called with plan.routes.
cudaError_t local_layer_route(const LocalLayerParams& p, cudaStream_t stream);
cudaError_t local_layer_launch(const LocalLayerParams& p, cudaStream_t stream);
// The forward of plans with `few` (local_few.cu); local_layer_launch calls it.
cudaError_t local_few_launch(const LocalLayerParams& p, cudaStream_t stream);

}  // namespace tmoe
