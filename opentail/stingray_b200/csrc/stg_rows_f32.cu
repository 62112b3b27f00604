// The row kernel (full-vocabulary pipeline, one row per CTA) for f32 logits.
#include "stg_kernels_impl.cuh"

namespace stg {

cudaError_t launch_rows_f32(const SampleArgs &a, int grid, cudaStream_t stream)
{
    void (*fn)(const SampleArgs) = k_sample_rows<false>;
    cudaError_t e = ensure_dynamic_smem((const void *)fn, kRowArenaBytes);
    if (e != cudaSuccess) return e;
    // as the second chance it is set up while the clusters of k_row run out (24 mixed rows of 50,257: 81.4 -> 78.7 us)
    if (a.redo_flags != nullptr) return launch_behind(fn, dim3((unsigned)grid), kThreads, kRowArenaBytes, stream, a);
    fn<<<grid, kThreads, kRowArenaBytes, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace stg
