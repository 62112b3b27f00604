// Full-vocabulary rows (Sampler.Sample's slow path, src/OpenTail.Stingray.Engine/Sampler.cs:41-95;
// BuildFilteredDistribution, :118-163; GreedyWithHistoryPenalties, :421-437) as ONE kernel: a cluster of
// CTAs owns a row from its first load to its draw.  See stg_row.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "stg_types.h"

namespace stg {

constexpr int kRowThreads = 512;     // threads of a CTA of the cluster
constexpr int kRowMaxCluster = 16;   // CTAs of a cluster at most (above 8 is an opt-in of the kernel)

// device workspace of the full-vocabulary rows of a step, indexed by RowPlan::flat_full
struct RowWs {
    float *e;            // [n, e_stride] exp values (L2-resident between the phases), rows padded to whole tiles of 256
    int32_t *ids;        // [n, e_stride] tokens of a row that was closed up to what its mask allows
    int64_t e_stride;
    int32_t *redo;       // [n] 1: the row kernel of the first design has to redo the row
};

// rows of a.items[0 .. a.n_items): every one a full-vocabulary row or a greedy row with penalties.
// want_argmax: descriptor mode (a.mode == 2) needs the arg-max of the raw row as well.
cudaError_t launch_row_clusters(const SampleArgs &a, const RowWs &ws, bool want_argmax, cudaStream_t stream);

// speculative verification behind the descriptor passes: accept chain and draw of every sequence (at most 32 draft
// tokens); fallback[s] becomes 1 where k_spec_finish has to redo sequence s
struct SpecArgs;
cudaError_t launch_spec_rows(const SpecArgs &a, const RowWs &ws, int32_t *fallback, cudaStream_t stream);

}  // namespace stg
