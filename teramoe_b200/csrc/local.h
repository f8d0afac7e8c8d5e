// Un-fused exchange on one rank (local.cu): the same calls as over NVLink, with nothing to send.  Rows are re-ordered straight
// from the caller's tensors into the result tensors; there is no symmetric arena, no barrier and no staging copy.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tmoe {

constexpr int kLocalChunk = 128;         // tokens that local_route numbers the rows of together
constexpr int kLocalMaxParts = 2;        // payloads that travel together (FP8 rows and their scales)

struct LocalPart {
    const void* src;
    void* dst;
    uint32_t row_bytes;                  // any size; 16-byte multiples on 16-byte aligned tensors are copied 16 bytes at a time
};

// Routing summary of topk_idx [T,K].
//   totals     [E + 2]: entries per expert, tokens with at least one valid entry, (scratch)
//   row_local  [T] position of the token among its chunk's tokens that have a valid entry, -1 for tokens without
//   chunk_base [ceil(T / kLocalChunk)] row of the chunk's first such token
//   in_rank    optional bool [T]; host_out optional host-visible [E + 1]: number of rows, entries per expert,
//              each with host_seq in its upper half
cudaError_t local_route(const void* topk_idx, int is64, int T, int K, int E, int* totals, int* row_local, int* chunk_base, uint8_t* in_rank,
                        unsigned long long* host_out, int host_seq, cudaStream_t stream);

// Rows of the tokens that have a valid entry, in token order, with their expert ids (-1 where invalid) and weights (0 there);
// send_row[t] = row of token t or -1.  worst_rows > 0: rows from the received count to worst_rows read as "nothing".
cudaError_t local_dispatch(const LocalPart* parts, int num_parts, const void* topk_idx, int is64, const float* topk_w, int T, int K, int E,
                           const int* totals, const int* row_local, const int* chunk_base, int* send_row, void* recv_idx, float* recv_w,
                           int worst_rows, cudaStream_t stream);

// to_rows: dst row send_row[t] <- src row t; otherwise dst row t <- src row send_row[t] (zeros where that is -1), and with
// `weights` [rows, K]: weights_out[t, k] = weights[send_row[t], k] for valid entries, else 0.  A row past `rows` (those of the tensors
// that send_row points into) is left alone, or reads as none.
cudaError_t local_move(const LocalPart* parts, int num_parts, const int* send_row, int T, long rows, int to_rows, const void* topk_idx, int is64, int K,
                       int E, const float* weights, float* weights_out, cudaStream_t stream);

}  // namespace tmoe
