// The loads of the flat step's streaming kernels (stg_flat_chunks.cu, stg_flat_greedy.cu): 16 bytes each, four logits
// of fp32 or eight of bf16.
#pragma once
#include <math_constants.h>

#include "stg_flat.cuh"
#include "stg_select.cuh"

namespace stg {

// How a thread reads its share of a piece of STEPS * 4096 elements (256 threads): R rounds of U loads of E elements.
template <bool BF16, int STEPS>
struct FlatShare {
    static constexpr int E = BF16 ? 8 : 4;
    static constexpr int U = STEPS * 16 / E < 4 ? STEPS * 16 / E : 4;
    static constexpr int R = STEPS * 16 / (E * U);
    static constexpr int kStride = kFlatThreads * E;  // from one load of a thread to the next
};

// elements i .. i + E - 1 of the row; masked ones and those at or beyond `end` read as -infinity
template <bool BF16>
__device__ __forceinline__ void flat_load(const LogitRow rowp, const uint32_t *mrow, int i, int end, float *v)
{
    constexpr int E = BF16 ? 8 : 4;
    if (i + E - 1 < end) {
        if constexpr (BF16) {
            if (((uintptr_t)rowp.p & 15) == 0) {
                const uint4 t = __ldcs((const uint4 *)((const uint16_t *)rowp.p + i));
                v[0] = bf16_lo(t.x); v[1] = bf16_hi(t.x); v[2] = bf16_lo(t.y); v[3] = bf16_hi(t.y);
                v[4] = bf16_lo(t.z); v[5] = bf16_hi(t.z); v[6] = bf16_lo(t.w); v[7] = bf16_hi(t.w);
                if (rowp.cap != 0.f) {
#pragma unroll
                    for (int e = 0; e < E; e++) v[e] = soft_cap(v[e], rowp.cap);
                }
            } else {  // rows of a stride that is no multiple of eight
                load_vec4<true, true>(rowp, i, v);
                load_vec4<true, true>(rowp, i + 4, v + 4);
            }
        } else {
            load_vec4<false, true>(rowp, i, v);
        }
    } else {
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = (i + e < end) ? load_one<BF16>(rowp, i + e) : -CUDART_INF_F;
    }
    if (mrow != nullptr && i < end) {
        const uint32_t bits = __ldg(mrow + (i >> 5)) >> (i & 31);
#pragma unroll
        for (int e = 0; e < E; e++)
            if (!((bits >> e) & 1u)) v[e] = -CUDART_INF_F;
    }
}

}  // namespace stg
