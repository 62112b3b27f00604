// Kernels of the flat form of a sampling step (see stg_flat.cuh): prep and the per-row finish of the top-k path.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "stg_flat.cuh"
#include "stg_flat_finish.cuh"
#include "stg_flat_prep.cuh"
#include "stg_launch.h"
#include "stg_select.cuh"
#include "stg_types.h"

namespace stg {

// ---- k_flat_prep --------------------------------------------------------------------------------------
// One 1024-thread CTA per row (flat_prep_row, stg_flat_prep.cuh).
template <bool BF16, bool CAP>
__global__ void __launch_bounds__(kThreads) k_flat_prep(const __grid_constant__ SampleArgs a, FlatRow *fr)
{
    __shared__ uint32_t red[32];
    __shared__ uint32_t list[kPrepList + 2];
    pdl_release();
    const int row = blockIdx.x;
    const RowPlan rp = a.plans[row];
    if (rp.n_chunks == 0) return;  // not a row of the flat step
    flat_prep_row<BF16>(a, fr, row, rp, CAP ? a.softcap : 0.f, red, list);
}

// ---- k_flat_finish ------------------------------------------------------------------------------------
// The rows of a.items, one per CTA.
template <bool BF16>
__global__ void __launch_bounds__(kThreads, 1) k_flat_finish(const __grid_constant__ SampleArgs a, FlatRow *fr)
{
    extern __shared__ __align__(16) unsigned char arena[];
    __shared__ SelCtl ctl;
    __shared__ FlatShared fs;
    flat_finish_row<BF16>(a, fr, a.items[blockIdx.x].row, blockIdx.x, a.cap, arena, ctl, fs);
    __syncthreads();  // all warps leave together, as in the smaller forms (stg_flat_finish_small.inc)
}

cudaError_t launch_flat_prep(const SampleArgs &a, FlatRow *fr, cudaStream_t stream)
{
    const bool cap = a.softcap != 0.f;
    if (a.dtype == 1) { if (cap) k_flat_prep<true, true><<<a.rows, kThreads, 0, stream>>>(a, fr); else k_flat_prep<true, false><<<a.rows, kThreads, 0, stream>>>(a, fr); }
    else { if (cap) k_flat_prep<false, true><<<a.rows, kThreads, 0, stream>>>(a, fr); else k_flat_prep<false, false><<<a.rows, kThreads, 0, stream>>>(a, fr); }
    return cudaGetLastError();
}

cudaError_t launch_flat_finish(const SampleArgs &a, FlatRow *fr, size_t smem, cudaStream_t stream)
{
    void (*fn)(const SampleArgs, FlatRow *) = a.dtype == 1 ? k_flat_finish<true> : k_flat_finish<false>;
    cudaError_t e = ensure_dynamic_smem((const void *)fn, smem);
    if (e != cudaSuccess) return e;
    return launch_behind(fn, dim3((unsigned)a.n_items), kThreads, smem, stream, a, fr);
}

}  // namespace stg
