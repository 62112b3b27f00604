// The HBM pass of the flat step over the rows of the top-k path and plain arg-max rows.  40 registers and no second
// register set for prefetched loads: the warps that fit besides cover the load latency - measured on the
// arg-max form of this loop (stg_flat_greedy.cu), that is worth more than the prefetch.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "stg_flat.cuh"
#include "stg_flat_load.cuh"
#include "stg_launch.h"
#include "stg_select.cuh"
#include "stg_types.h"

#ifndef STG_CHUNKS_MB
#define STG_CHUNKS_MB 5
#endif

namespace stg {

// grid (pieces of STEPS * 4096 elements, rows of a.items); 256 threads; in round s thread t reads elements
// 256 E (U s + u) + E t .. + E - 1 (u < U) of the piece as U independent 16-byte loads (E 4 of fp32, 8 of bf16:
// a loop's step of 96 bf16 rows of 151,936 went from 86.9 to 84.6 us with those instead of 8-byte loads).
// STEPS is 4 where that gives every SM two CTAs to hold, else 1: a lone row of 151,936 is ten pieces of 16,384,
// each four dependent rounds of loads long, or 38 of 4096.
template <bool BF16, bool CAP, int STEPS>
__global__ void __launch_bounds__(kFlatThreads, STG_CHUNKS_MB) k_flat_stream_chunks(const __grid_constant__ SampleArgs a, FlatRow *fr)
{
    const int row = __ldg(&a.items[blockIdx.y].row), tid = threadIdx.x, lane = tid & 31;
    const RowPlan *rpp = a.plans + row;
    const int begin = blockIdx.x * (STEPS * 4096);
    const int end = min(a.vocab, begin + STEPS * 4096);
    const int esz = BF16 ? 2 : 4;
    const LogitRow rowp{(const char *)a.logits + (int64_t)row * a.row_stride * esz, CAP ? a.softcap : 0.f};
    const bool mine = __ldg(&rpp->n_chunks) != 0 && begin < end;
    // While the rows' bounds are still being found: the pieces of the CTAs that are resident by then, into L2.
    if (mine && blockIdx.y * gridDim.x + blockIdx.x < (unsigned)a.sm_count * STG_CHUNKS_MB)
        for (int i = begin + tid * (128 / esz); i < end; i += kFlatThreads * (128 / esz))
            asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)rowp.p + (int64_t)i * esz));
    pdl_release();
    pdl_wait();
    if (!mine) return;  // not a row of this pass
    const uint32_t *mrow = (__ldg(&rpp->use_mask) && a.mask) ? a.mask + (int64_t)row * a.mask_stride : nullptr;
    typedef FlatShare<BF16, STEPS> S;
    const int i0 = begin + tid * S::E;

    if (__ldg(&rpp->path) == kPathGreedy) {
        __shared__ unsigned long long red[kFlatThreads / 32];
        float best = -CUDART_INF_F;
        int best_i = -1;
#pragma unroll 1
        for (int s = 0; s < S::R; s++) {
            float cur[S::U][S::E];
#pragma unroll
            for (int u = 0; u < S::U; u++) flat_load<BF16>(rowp, mrow, i0 + (s * S::U + u) * S::kStride, end, cur[u]);
#pragma unroll
            for (int u = 0; u < S::U; u++)
#pragma unroll
                for (int e = 0; e < S::E; e++)
                    if (cur[u][e] > best) { best = cur[u][e]; best_i = i0 + (s * S::U + u) * S::kStride + e; }
        }
        // a thread visits ascending indices, so it holds its lowest index of the value; the key
        // order (value, then lower index) settles ties between threads, pieces and CTAs
        unsigned long long k = best_i >= 0 ? make_key(best, best_i) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xFFFFFFFFu, k, o);
            k = t > k ? t : k;
        }
        if (lane == 0) red[tid >> 5] = k;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kFlatThreads / 32; w++) k = red[w] > k ? red[w] : k;
            if (k != 0ull) atomicMax(&fr[row].key, k);
        }
        return;
    }

    // top-k path: every element above the row's bound becomes a candidate.  The CTA collects its
    // candidates in shared memory and hands them to the row's list with a single global atomicAdd at
    // the end; should a piece hold more than the staging area takes, the excess goes to the list
    // directly.
    __shared__ unsigned long long stage[kFlatStage];
    __shared__ int stage_cnt, list_first;
    if (tid == 0) stage_cnt = 0;
    __syncthreads();
    const float tau = fr[row].tau;
    const int cap = fr[row].cap;
    unsigned long long *cand = a.cand + __ldg(&rpp->cand_off);
    int *cnt_p = &fr[row].cnt;
    // The sweep itself only notes which of the thread's elements pass (one bit each): keeping the
    // key construction and the appends out of the loop keeps it as tight as the arg-max loop.  The
    // few that pass (a fraction of a percent) are read again afterwards, from L2.
    unsigned long long passed = 0ull;
#pragma unroll 1
    for (int s = 0; s < S::R; s++) {
        float cur[S::U][S::E];
#pragma unroll
        for (int u = 0; u < S::U; u++) flat_load<BF16>(rowp, mrow, i0 + (s * S::U + u) * S::kStride, end, cur[u]);
        unsigned pass = 0u;
#pragma unroll
        for (int u = 0; u < S::U; u++)
#pragma unroll
            for (int e = 0; e < S::E; e++) pass |= (cur[u][e] > tau) ? (1u << (u * S::E + e)) : 0u;  // out of range and masked read -inf
        passed |= (unsigned long long)pass << (S::U * S::E * s);
    }
    static_assert(STEPS * 16 <= 64, "one bit per element of a thread");
    while (passed != 0ull) {
        const int b = __ffsll((long long)passed) - 1;
        passed &= passed - 1ull;
        const int idx = i0 + b / S::E * S::kStride + b % S::E;  // bit E (U s + u) + e
        const unsigned long long key = make_key(load_one<BF16>(rowp, idx), idx);
        const int slot = atomicAdd(&stage_cnt, 1);
        if (slot < kFlatStage) {
            stage[slot] = key;
        } else {
            const int g = atomicAdd(cnt_p, 1);
            if (g < cap) cand[g] = key;
        }
    }
    __syncthreads();
    const int staged = min(stage_cnt, kFlatStage);
    if (staged > 0) {
        if (tid == 0) list_first = atomicAdd(cnt_p, staged);
        __syncthreads();
        const int g0 = list_first;
        for (int t = tid; t < staged; t += kFlatThreads)
            if (g0 + t < cap) cand[g0 + t] = stage[t];
    }
}

cudaError_t launch_flat_stream_chunks(const SampleArgs &a, FlatRow *fr, cudaStream_t stream)
{
    const int pieces = (a.vocab + kFlatPiece - 1) / kFlatPiece;
    const bool few = (long long)pieces * a.n_items < 2 * a.sm_count;
    const dim3 grid((unsigned)(few ? (a.vocab + 4095) / 4096 : pieces), (unsigned)a.n_items);
    const bool cap = a.softcap != 0.f;
    void (*fn)(const SampleArgs, FlatRow *);
    if (a.dtype == 1) fn = few ? (cap ? k_flat_stream_chunks<true, true, 1> : k_flat_stream_chunks<true, false, 1>)
                               : (cap ? k_flat_stream_chunks<true, true, 4> : k_flat_stream_chunks<true, false, 4>);
    else fn = few ? (cap ? k_flat_stream_chunks<false, true, 1> : k_flat_stream_chunks<false, false, 1>)
                  : (cap ? k_flat_stream_chunks<false, true, 4> : k_flat_stream_chunks<false, false, 4>);
    return launch_behind(fn, grid, kFlatThreads, 0, stream, a, fr);
}

}  // namespace stg
