// The flat form of a sampling step: instead of a few fat persistent CTAs that each own a row (or a
// large piece of one) from the first load to the last draw, the step is a short sequence of kernels
//
//   k_flat_prep    one CTA per row   what a row needs before it can be streamed: the filter bound of
//                                    a top-k row (an order statistic of its first 4096 logits), zeroed
//                                    counters
//   k_flat_stream_chunks
//                  one small CTA per piece of a row (stg_flat_chunks.cu).  Greedy rows keep a running
//                  arg-max key (64-bit atomicMax), top-k rows append every logit above the row's bound
//                  to the row's candidate list (staged in shared memory, one global atomicAdd per CTA)
//   k_flat_finish  one CTA per row   candidates only: the exact top-N selection, penalties, softmax
//                                    over k, min-p, top-p and the draw of SampleTopK
//                                    (src/OpenTail.Stingray.Engine/Sampler.cs:216-357); built for 1024,
//                                    512 and 256 threads (one, two, four CTAs per SM)
//   k_row          one cluster of CTAs per full-vocabulary row (stg_row.cuh), beside the kernels above
//   k_greedy_step  a step whose rows are all plain arg-max rows: the HBM pass with prep and finish
//                  folded in, one launch (stg_flat_greedy.cu)
//
// so that the HBM pass runs on all SMs whatever the mix of rows - thousands of 256-thread CTAs that
// the hardware scheduler balances - and everything serial touches a few hundred candidates per row.
//
// The bound of a top-k row is optimistic, and checked: k_flat_finish accepts the candidate list only
// when it holds between N = top_k + history length and its capacity entries - they are then exactly
// the logits above the bound, hence a superset of the N best.  Otherwise (the first 4096 logits were
// not representative: ties, masks, sorted rows) the finishing CTA streams the row again itself with
// the exact selection of stg_select.cuh.  No CTA of these kernels waits on another.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "stg_pdl.cuh"
#include "stg_types.h"

namespace stg {

constexpr int kFlatThreads = 256;                  // threads of a k_flat_stream_chunks CTA
constexpr int kFlatPiece = 16384;                  // elements of a row one such CTA reads
constexpr int kFlatSample = 4096;                  // leading elements of a row the bound is guessed from
constexpr int kFlatSlack = 8192;                   // candidate capacity of a top-k row beyond N (the bound scatters: up to ~3x the expected count was seen)
constexpr int kFlatStage = 1024;                   // candidates a k_flat_stream_chunks CTA collects in shared memory

// per-row state of the flat step (device memory, 32 bytes)
struct FlatRow {
    unsigned long long key;  // greedy: running (value, lowest index) arg-max key; 0: nothing finite yet
    float tau;               // top-k: every logit > tau is a candidate
    int32_t cnt;             // top-k: candidates appended (may exceed the capacity: the excess was dropped)
    int32_t cap;             // top-k: capacity of the row's candidate list
    int32_t ticket;          // all-greedy step (stg_flat_greedy.cu): pieces of the row that have arrived; 0 between steps
    int32_t pad[2];
};
static_assert(sizeof(FlatRow) == 32, "FlatRow layout");

// The kernels of the step are launched behind one another (stg_pdl.cuh).  One fp32 row with top-k 18.4 -> 16.7 us a
// step, 512 rows of 256,000 140.1 -> 135.5 us.
cudaError_t launch_flat_prep(const SampleArgs &a, FlatRow *fr, cudaStream_t stream);
// the HBM pass over rows of the top-k path and plain arg-max rows only (stg_flat_chunks.cu)
cudaError_t launch_flat_stream_chunks(const SampleArgs &a, FlatRow *fr, cudaStream_t stream);
// a step of plain arg-max rows only, in one launch (stg_flat_greedy.cu); needs every row's key and ticket at zero
cudaError_t launch_greedy_step(const SampleArgs &a, FlatRow *fr, cudaStream_t stream);
// the small-CTA finishes (512 threads, two CTAs per SM; 256 threads, four per SM; a.finish_cap entries per buffer)
cudaError_t launch_flat_finish_half(const SampleArgs &a, FlatRow *fr, cudaStream_t stream);
cudaError_t launch_flat_finish_quarter(const SampleArgs &a, FlatRow *fr, cudaStream_t stream);
// one CTA of 1024 threads per row of a.items
cudaError_t launch_flat_finish(const SampleArgs &a, FlatRow *fr, size_t smem, cudaStream_t stream);

}  // namespace stg
