// One cluster of CTAs per full-vocabulary row.
//
// What the reference does to such a row is a chain of sums that are sequential in fp32, a sort and a
// draw, each step needing the one before it for the whole row.  As a chain of kernels it was bound by the
// chain: a dozen launches, each as long as its slowest row.  Here the CTAs of a hardware cluster keep the
// row to themselves, every pass over its V elements is cut between them, the passes are separated by
// cluster barriers (a few hundred nanoseconds), and what one CTA has to see of the others' work (tile
// summaries, histograms, candidates) is pushed into its shared memory:
//
//   P0  history / bias overrides of the CTA's own tokens -> hash table
//   P1  maximum, and per tile an estimate of its sum of exp values that needs none (the only pass that goes to HBM)
//   P2  e = exp(x - max) -> scratch (L2); on the way the guesses, compositions and runs of stg_walk.cuh and the
//       histogram of the exp values
//   P3  rank 0's first warp walks to the exact sum; the other CTAs' histograms go to rank 0
//   P4  rank 0 bounds the nucleus.  Narrow (the usual case for a peaked row: up to kNarrow candidates):
//       the candidates go to rank 0, are sorted, cut, sorted by token and drawn from there.
//   P5  wide: per histogram bin the integer increment of all its elements (no order needed inside a
//       bin), except in the bins where the order counts - the sum changes binade, meets top_p, or meets
//       an exact rounding tie - whose elements are handed to rank 0 and sorted
//   P6  the sorted-order sum bin by bin -> top-p threshold
//   P7  Normalize's sum; compositions of the final probabilities; the walk to the uniform
//
// Bound: the latency of the phases one after the other; a lone row of 32,000 spends 1 to 6 us in each (table 2.4,
// maximum 3.5, guesses 0.9, exp values 5.5, walk 4.8, plan 4.8; narrow another 8, wide 31).  As passes of their own - exp
// values, compositions, histogram, each reading them again - the first four took as long for a lone row, but 64 rows of
// 151,936 took 172 us instead of 159, and 288 + 256 descriptors of a verification step 455 instead of 375.  Where many rows run,
// warps wait for instructions as much as for data: hence one tile to a turn of a loop (for_tiles), rare cases out of line, and
// additions by predicate instead of branch (add_if: the increments of 64 rows 25 -> 19 us).  The row is read from HBM
// once and from L2 in every later pass as long as the rows in flight fit there (64 rows of 151,936 do: 40 MB read for 39);
// 288 rows, one CTA each and 1.2 MB with their exp values, do not, and their passes run at 4.7 TB/s.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdlib.h>

#include "stg_launch.h"
#include "stg_row.cuh"
#include "stg_rowdist.cuh"
#include "stg_pdl.cuh"
#include "stg_spec_prov.cuh"
#include "stg_walk.cuh"

namespace cg = cooperative_groups;

namespace stg {

namespace {

constexpr int kRT = kRowThreads;
constexpr int kRW = kRT / 32;
constexpr int kNarrow = 2048;        // candidates rank 0 handles on its own
constexpr int kRowList = 5120;       // elements of the bins whose order counts (every bin padded to a multiple of 8) at most
constexpr int kFlagged = 512;        // bins whose order counts at most
constexpr unsigned char kBinOrder = 255;  // bin_e: the bin's order counts; 0: below the nucleus
static_assert(kBins == 8 * kRT, "the bin scans give 8 bins to a thread");

// dynamic shared memory: the override table of P0..P2, the histogram and the candidate lists.  The table of `slots` entries
// is int key[], u32 cnt[] (occurrences 12 bits, in the window 12, bias 1), float val[] and 65536 folded bits; one of up to
// kSmallTable slots (512 history and bias entries) lies where the lists will be, so that the histogram can be filled
// while it is in use, a larger one lies over the histogram too.
constexpr int kSmallTable = 1024;
constexpr int kTabEnd = kMaxOvSlots * 12 + 8192;
constexpr int kOffBinMass = 0;                                  // u32[kBins]
constexpr int kOffBinD = kBins * 4;                             // u32[kBins]
constexpr int kOffBinE = 2 * kBins * 4;                         // u8[kBins]
constexpr int kOffList = 2 * kBins * 4 + kBins;                 // u32[kRowList] | u64[kNarrow]
constexpr int kListEnd = kOffList + kRowList * 4;
static_assert(kSmallTable * 12 + 8192 <= kRowList * 4, "a small table fits the list");
constexpr int kOffWalk = (kListEnd > kTabEnd ? kListEnd : kTabEnd);
constexpr int kRowSmem = kOffWalk + (int)sizeof(WalkArea);
static_assert(kNarrow * 8 <= kRowList * 4, "the narrow list borrows the wide one");

struct RowSh {
    u64 maxkey[kRowMaxCluster], rawkey[kRowMaxCluster];
    float cmax[kRowMaxCluster];
    double tot[2][kRowMaxCluster];
    double part[kRowMaxCluster];
    int cnt[kRowMaxCluster];
    double red_d[kRW];
    float red_f[kRW];
    u64 red_k[kRW];
    int red_i[kRW], red_i2[kRW];
    float tile_sum[kMaxSubTiles];
    unsigned char guess[kMaxSubTiles], kind[kMaxSubTiles];
    // pushed by rank 0
    float sum;
    int narrow, c_lo, stop;
    int hit_keep;            // ties at the threshold: the first `hit_keep` of them by token survive; 0: all
    float tstar;
    int tie_idx;
    RowDist dist;
    int n_cand, list_n;
    // rank 0 only
    int n_flagged, cut_lo, p_all;
    unsigned tie_bits[kBins / 32];   // bins whose order turned out to count
    unsigned new_bits[kBins / 32];   // those of them whose elements are to be handed over
    unsigned short flagged[kFlagged];
    uint32_t flags;
};

// out of line, like everything that few rows or few tiles need (stg_walk.cuh)
__device__ __noinline__ Lane8 soft_cap_8(Lane8 x, float cap)
{
#pragma unroll
    for (int j = 0; j < 8; j++) x.v[j] = soft_cap(x.v[j], cap);
    return x;
}

// ---- the row's adjusted, temperature-scaled logits ---------------------------------------------------
template <bool BF16>
struct RowSrc {
    LogitRow rowp;
    const uint32_t *mrow;
    int vec;              // 8: rows start on a boundary of 8 elements (32-byte loads of fp32), 4: of 4, 1: anywhere
    int n;
    float inv_t;
    bool scale;
    const unsigned char *tab;  // null: no overrides
    int tab_mask;

    // this lane's 8 raw elements at `base` (-inf beyond the row) and their mask bits; nothing is read where no
    // token is allowed
    __device__ __forceinline__ void fetch(int base, float x[8], unsigned &bits) const
    {
        bits = 0xFFu;
        if (mrow != nullptr) {
            bits = base < n ? (__ldg(mrow + (base >> 5)) >> (base & 31)) & 0xFFu : 0u;
            if (base + 8 > n) bits &= (1u << max(n - base, 0)) - 1u;
        }
        if (bits == 0u) return;
        if (base + 8 <= n && vec >= 4) {
            if (BF16) {
                const uint2 *p = (const uint2 *)((const uint16_t *)rowp.p + base);
                uint4 q;
                if (vec == 8) q = __ldg((const uint4 *)p);
                else { const uint2 q0 = __ldg(p), q1 = __ldg(p + 1); q = make_uint4(q0.x, q0.y, q1.x, q1.y); }
                x[0] = bf16_lo(q.x); x[1] = bf16_hi(q.x); x[2] = bf16_lo(q.y); x[3] = bf16_hi(q.y);
                x[4] = bf16_lo(q.z); x[5] = bf16_hi(q.z); x[6] = bf16_lo(q.w); x[7] = bf16_hi(q.w);
            } else {
                const float *p = (const float *)rowp.p + base;
                if (vec == 8) {
                    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]) : "l"(p));
                } else {
                    const float4 q0 = __ldg((const float4 *)p), q1 = __ldg((const float4 *)p + 1);
                    x[0] = q0.x; x[1] = q0.y; x[2] = q0.z; x[3] = q0.w; x[4] = q1.x; x[5] = q1.y; x[6] = q1.z; x[7] = q1.w;
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                x[j] = -CUDART_INF_F;
                if (base + j < n) {
                    if (BF16) x[j] = __uint_as_float((uint32_t)__ldg((const uint16_t *)rowp.p + base + j) << 16);
                    else x[j] = __ldg((const float *)rowp.p + base + j);
                }
            }
        }
    }
    __device__ __forceinline__ void mask(float x[8], unsigned bits, int base) const
    {
        if (bits == 0u) {
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = -CUDART_INF_F;
            return;
        }
        if (rowp.cap != 0.f) {
            const Lane8 y = soft_cap_8(lane8(x), rowp.cap);
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (base + j < n) x[j] = y.v[j];
        }
        if (bits != 0xFFu) {
#pragma unroll
            for (int j = 0; j < 8; j++)
                if (!((bits >> j) & 1u)) x[j] = -CUDART_INF_F;
        }
    }
    __device__ __forceinline__ int find(int id) const
    {
        const int *key = (const int *)tab;
        int h = (int)(((unsigned)id * 2654435761u) >> 7) & tab_mask;
        for (;;) {
            const int k = key[h];
            if (k == id) return h;
            if (k == -1) return -1;
            h = (h + 1) & tab_mask;
        }
    }
    __device__ __forceinline__ void override_(float x[8], int base) const
    {
        if (tab != nullptr) {
            unsigned m = (tab + 12 * (tab_mask + 1))[(base & 0xFFFF) >> 3];
#pragma unroll 1
            while (m) {
                const int j = __ffs(m) - 1;
                m &= m - 1u;
                const int slot = base + j < n ? find(base + j) : -1;
                if (slot >= 0) {
                    const float v = ((const float *)(tab + 8 * (tab_mask + 1)))[slot];
#pragma unroll
                    for (int k = 0; k < 8; k++) x[k] = k == j ? v : x[k];
                }
            }
        }
    }
    __device__ __forceinline__ void adjust(float x[8], int base) const
    {
        override_(x, base);
        rescale(x);
    }
    __device__ __forceinline__ void rescale(float x[8]) const
    {
        if (scale) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {  // two elements to an instruction
                const float2 v = __fmul2_rn(make_float2(x[j], x[j + 1]), make_float2(inv_t, inv_t));
                x[j] = v.x;
                x[j + 1] = v.y;
            }
        }
    }
};

// 8 elements of the row's scratch, which is padded with zeros to whole tiles
__device__ __forceinline__ void load_e(const float *e, int base, float x[8])
{
    asm volatile("ld.global.cg.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]) : "l"(e + base) : "memory");
}
__device__ __forceinline__ void store_e(float *e, int base, const float x[8])
{
    asm volatile("st.global.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7]), "l"(e + base) : "memory");
}
// an fp32 value >= 0 as a double by its bits: conversions run at a fraction of the integer rate.  Zeros and
// subnormals come out as less than 2^-126, which no sum they go into can show.
__device__ __forceinline__ double widen(float p)
{
    const uint32_t b = __float_as_uint(p);
    return __hiloint2double((int)((b >> 3) + (896u << 20)), (int)(b << 29));
}

// adds v to a word of this CTA's shared memory where `on`.  By a predicate: a branch around every one of eight additions
// parts the warp eight times, and costs more than the addition.
__device__ __forceinline__ void add_if(bool on, unsigned *at, unsigned v)
{
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p red.shared.add.u32 [%1], %2;\n}"
                 ::"r"((unsigned)on), "r"((unsigned)__cvta_generic_to_shared(at)), "r"(v) : "memory");
}
__device__ __forceinline__ float exp2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_max_f(float x)
{
    float y;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_sum_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}
// One warp: {maximum, sum of exp(x - maximum)} of a tile's elements (8 per lane, scaled by 1 / T as the exp values will be), to *est,
// and the lane's maximum.  What the tile will weigh against the row's maximum, before that is known: a guess, good to 1e-6
// for what weighs something and 1e-5 for the rest.  Of the logits before they are scaled it is good for nothing where
// 1 / T makes a unit of them large: at T = 1e-6 softmax sums were expected in the wrong binade, and 16 rows with logits
// next to their maximum took 125 us instead of 76.
constexpr float kLog2E = 1.44269504f;
__device__ __forceinline__ float estimate_tile(const float x[8], float2 *est)
{
    float m = x[0];
#pragma unroll
    for (int j = 1; j < 8; j++) m = fmaxf(m, x[j]);
    const float top = warp_max_f(m), ref = top > -CUDART_INF_F ? top : 0.f;
    float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {  // two elements to an instruction
        const float2 v = __fmul2_rn(__fadd2_rn(make_float2(x[j], x[j + 1]), make_float2(-ref, -ref)), make_float2(kLog2E, kLog2E));
        s2 = __fadd2_rn(s2, make_float2(exp2_approx(v.x), exp2_approx(v.y)));
    }
    const float s = warp_sum_f(s2.x + s2.y);
    if ((threadIdx.x & 31) == 0) *est = make_float2(top, s);
    return m;
}

__device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}
__device__ __forceinline__ double warp_scan_d(double v)  // inclusive
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
__device__ __forceinline__ int warp_scan_i(int v)  // inclusive
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
// sum over the block, the same order every time; every thread gets it
__device__ __forceinline__ double block_sum_d(double v, double *red)
{
    v = warp_sum_d(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kRW; w++) t += red[w];
    return t;
}
// two inclusive block scans at once
__device__ __forceinline__ void block_scan_2(int &v, int &w, int *red, int *red2)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_scan_i(v);
    w = warp_scan_i(w);
    __syncthreads();
    if (lane == 31) { red[warp] = v; red2[warp] = w; }
    __syncthreads();
    int b = 0, c = 0;
#pragma unroll
    for (int k = 0; k < kRW; k++)
        if (k < warp) { b += red[k]; c += red2[k]; }
    v += b;
    w += c;
}
__device__ __forceinline__ u64 block_max_k(u64 k, u64 *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const u64 t = __shfl_xor_sync(0xFFFFFFFFu, k, o);
        k = t > k ? t : k;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = k;
    __syncthreads();
    k = 0ull;
#pragma unroll
    for (int w = 0; w < kRW; w++) k = red[w] > k ? red[w] : k;
    return k;
}
__device__ __forceinline__ float block_max_f(float v, float *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < kRW; w++) v = fmaxf(v, red[w]);
    return v;
}

// descending bitonic sort of p2 (a power of two, >= 64) 64-bit keys in shared memory by the block.  Steps
// inside aligned groups of 64 keys need no block barrier: a warp holds two keys per lane.
__device__ __forceinline__ void row_sort_desc(u64 *a, int p2)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto tail = [&](u64 &x, u64 &y, int i, int k, int j0) {
        // x = key i (i = group * 64 + lane), y = key i + 32; steps j0 .. 1 of stage k
        if (j0 >= 32 && (x < y) == ((i & k) == 0)) { const u64 t = x; x = y; y = t; }
        for (int j = min(j0, 16); j > 0; j >>= 1) {
            const u64 ox = __shfl_xor_sync(0xFFFFFFFFu, x, j), oy = __shfl_xor_sync(0xFFFFFFFFu, y, j);
            const bool lower = (lane & j) == 0;
            const bool dx = (i & k) == 0, dy = ((i + 32) & k) == 0;
            x = (lower == dx) ? (x > ox ? x : ox) : (x < ox ? x : ox);
            y = (lower == dy) ? (y > oy ? y : oy) : (y < oy ? y : oy);
        }
    };
    for (int g = warp; g < p2 / 64; g += kRW) {
        const int i = g * 64 + lane;
        u64 x = a[i], y = a[i + 32];
        for (int k = 2; k <= 64; k <<= 1) tail(x, y, i, k, k >> 1);
        a[i] = x;
        a[i + 32] = y;
    }
    __syncthreads();
    for (int k = 128; k <= p2; k <<= 1) {
        for (int j = k >> 1; j >= 64; j >>= 1) {
            for (int t = tid; t < (p2 >> 1); t += kRT) {
                const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1)), l = i | j;
                const u64 x = a[i], y = a[l];
                if ((x < y) == ((i & k) == 0)) { a[i] = y; a[l] = x; }
            }
            __syncthreads();
        }
        for (int g = warp; g < p2 / 64; g += kRW) {
            const int i = g * 64 + lane;
            u64 x = a[i], y = a[i + 32];
            tail(x, y, i, k, 32);
            a[i] = x;
            a[i + 32] = y;
        }
        __syncthreads();
    }
}

// P0: the overrides among the tokens [lo, hi): ApplyHistoryPenalties after the logit bias
// (Sampler.cs:50-56, :367-419).  Every CTA reads the whole history and keeps its own tokens.
template <bool BF16>
__device__ __forceinline__ void build_table(const SampleArgs &a, const RowPlan &rp, const RowSrc<BF16> &src, unsigned char *tab, int slots,
                                            int nh, int nb, int lo, int hi)
{
    const int tid = threadIdx.x, mask = slots - 1;
    int *key = (int *)tab;
    unsigned *cnt = (unsigned *)(key + slots);
    float *val = (float *)(cnt + slots);
    unsigned *map = (unsigned *)(val + slots);
    for (int t = tid; t < slots; t += kRT) { key[t] = -1; cnt[t] = 0u; val[t] = 0.f; }
    for (int t = tid; t < 2048; t += kRT) map[t] = 0u;
    __syncthreads();
    for (int t = tid; t < nh + nb; t += kRT) {
        const bool hist = t < nh;
        const int id = __ldg(hist ? a.hist_ids + rp.hist_off + t : a.bias_ids + rp.bias_off + (t - nh));
        if (id < lo || id >= hi) continue;
        int h = (int)(((unsigned)id * 2654435761u) >> 7) & mask;
        for (;;) {
            const int old = atomicCAS(&key[h], -1, id);
            if (old == -1 || old == id) break;
            h = (h + 1) & mask;
        }
        if (hist) {
            atomicAdd(&cnt[h], 1u + (t >= rp.window_start ? 4096u : 0u));
        } else {
            atomicAdd(&val[h], __ldg(a.bias_vals + rp.bias_off + (t - nh)));
            atomicOr(&cnt[h], 1u << 31);
        }
    }
    __syncthreads();
    for (int h = tid; h < slots; h += kRT) {
        const int id = key[h];
        if (id < 0) continue;
        float x = load_one<BF16>(src.rowp, id);
        if (src.mrow && !mask_bit(src.mrow, id)) x = -CUDART_INF_F;
        const unsigned c = cnt[h];
        if (c >> 31) x = __fadd_rn(x, val[h]);
        const int occ_all = (int)(c & 4095u), occ_w = (int)((c >> 12) & 4095u);
        if (occ_all > 0) {
            if (rp.rep != 1.0f)
                for (int r = 0; r < occ_w; r++) x = x > 0.f ? __fdiv_rn(x, rp.rep) : __fmul_rn(x, rp.rep);
            if (!(rp.pres == 0.f && rp.freq == 0.f)) x = __fsub_rn(x, __fadd_rn(rp.pres, __fmul_rn(rp.freq, (float)occ_all)));
        }
        val[h] = x;
        atomicOr(&map[(id & 0xFFFF) >> 5], 1u << (id & 31));
    }
    __syncthreads();
}

// body(t, x) for a warp's tiles t = first, first + stride, ... below end, whose elements load(t, x) fetches: one tile at a time,
// the next one's elements on the way.  Two tiles to a turn hide as much latency, but their loop is twice as long, and
// the warps wait for its instructions: 64 rows of 151,936 166 -> 161 us with this (and the rare cases out of line) in P2 alone.
template <class Load, class Body>
__device__ __forceinline__ void for_tiles(int first, int end, int stride, const Load &load, const Body &body)
{
    float nx[8];
    if (first < end) load(first, nx);
#pragma unroll 1
    for (int t = first; t < end; t += stride) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = nx[j];
        if (t + stride < end) load(t + stride, nx);
        body(t, x);
    }
}

// The fp64 prefix sums of the CTA's tiles: thread i holds those around its tiles 2 i and 2 i + 1.
struct TilePrefix { double in, mid, out, all; };
// every thread; two block barriers, the first of them ahead of any access to `red`
__device__ __forceinline__ TilePrefix tile_prefix(const float *tile_sum, int nt, double *red)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    const double v = 2 * tid < nt ? (double)tile_sum[2 * tid] : 0.0, w = 2 * tid + 1 < nt ? (double)tile_sum[2 * tid + 1] : 0.0;
    TilePrefix p;
    const double inc = warp_scan_d(v + w);
    if (lane == 31) red[warp] = inc;
    __syncthreads();
    double before = 0.0, all = 0.0;
#pragma unroll
    for (int k = 0; k < kRW; k++) {
        const double r = red[k];
        before += k < warp ? r : 0.0;
        all += r;
    }
    p.in = before + (inc - (v + w));
    p.mid = p.in + v;
    p.out = before + inc;
    p.all = all;
    return p;
}

// guessed binades and kinds of the CTA's tiles [t0, t1): the sum in front of tile t is base + factor times the
// prefix; `end`: the guess for the whole sum, `target` where the walk is to end.  Ends in a block barrier.
__device__ __forceinline__ void guess_tiles(RowSh &sh, const TilePrefix &p, int t0, int t1, double base, double factor, double all, double target)
{
    const int tid = threadIdx.x, g_end = exp_of_double(all);
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int i = 2 * tid + u, t = t0 + i;
        if (t < t1) {
            const double lo = base + (u ? p.mid : p.in) * factor, hi = base + (t + 1 == t1 ? p.all : u ? p.out : p.mid) * factor;
            const int g = exp_of_double(lo);
            int k = walk_kind(t, g, exp_of_double(hi), g_end);
            if (lo < target && target <= hi && t > 0) k = kTileSlot + kWalkCross;
            sh.guess[i] = (unsigned char)g;
            sh.kind[i] = (unsigned char)k;
        }
    }
    __syncthreads();
}

// One warp: the composition of tile t (8 elements per lane in x) under its guess, or what its kind asks for, into rank 0's
// walk area.
__device__ __forceinline__ void compose_tile(const RowSh &sh, WalkArea *wa, WalkArea *dst, const float x[8], int t, int t0)
{
    const int lane = threadIdx.x & 31;
    const int k = sh.kind[t - t0], g = sh.guess[t - t0];
    int a0 = 0, a1 = 0;
    if (k == kTileRun) {
        tile_composite(x, g, a0, a1);
    } else if (k != kTileReplay || t == 0) {
        WalkCross *c = &dst->xs[k >= kTileSlot ? (k - kTileSlot) % (kWalkCross + 1) : k - 1];
        if (t != 0) {
            if (k < kTileSlot) walk_cross(c, lane8(x), g);
            if (lane == 0) c->tile = t;
        }
        float4 *q = (float4 *)((t == 0 ? dst->head : c->x) + lane * 8);
        q[0] = make_float4(x[0], x[1], x[2], x[3]);
        q[1] = make_float4(x[4], x[5], x[6], x[7]);
    }
    if (lane == 0) {
        wa->comp[t] = make_int2(a0, a1);
        if (dst != wa) dst->comp[t] = make_int2(a0, a1);
    }
}

// The runs of the CTA's composed tiles, a group of them per warp (behind a block barrier).  A run ends with its group, so
// that the groups need nothing of each other: one warp over all 594 tiles of a row of 151,936 took as long as the rest.
constexpr int kRunGroup = 64;
__device__ __forceinline__ void runs_of_tiles(const RowSh &sh, const WalkArea *wa, WalkArea *dst, int t0, int t1)
{
    for (int g = t0 + (int)(threadIdx.x >> 5) * kRunGroup; g < t1; g += kRW * kRunGroup)
        walk_runs(dst, wa->comp + g, sh.guess + (g - t0), sh.kind + (g - t0), g, min(t1, g + kRunGroup));
}

// guesses, compositions and runs of the CTA's tiles [t0, t1) over the elements load(t, x) and then map(t, x), whose sums are in
// tile_sum (times `scale` they are what the walk will see) and whose prefix is `p`, into rank 0's walk area.
// `base`: the sum of the tiles before t0, `all` of the row, both unscaled.
template <class Load, class Map>
__device__ __forceinline__ void summarise(RowSh &sh, WalkArea *wa, WalkArea *dst, const Load &load, const Map &map, int t0, int t1,
                                          const TilePrefix &p, double base, double all, double scale, double target)
{
    guess_tiles(sh, p, t0, t1, base * scale, scale, all * scale, target);
    for_tiles(t0 + (int)(threadIdx.x >> 5), t1, kRW, load, [&](int t, float (&x)[8]) {
        map(t, x);
        compose_tile(sh, wa, dst, x, t, t0);
    });
    __syncthreads();
    runs_of_tiles(sh, wa, dst, t0, t1);
}

// a warp's sort of a short list (descending) by counting ranks; lists of one value - the rule for rows that
// were bf16 - are copied
__device__ __forceinline__ void warp_rank_sort(const uint32_t *src, uint32_t *dst, int c)
{
    const int lane = threadIdx.x & 31;
    uint32_t mn = 0xFFFFFFFFu, mx = 0u;
    for (int e = lane; e < c; e += 32) { mn = min(mn, src[e]); mx = max(mx, src[e]); }
    mn = __reduce_min_sync(0xFFFFFFFFu, mn);
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    if (mn == mx) {
        for (int e = lane; e < c; e += 32) dst[e] = mx;
        return;
    }
    for (int e0 = 0; e0 < c; e0 += 128) {
        uint32_t k[4];
        int r[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int e = e0 + u * 32 + lane;
            k[u] = e < c ? src[e] : 0u;
            r[u] = 0;
        }
        for (int j = 0; j < c; j++) {
            const uint32_t o = src[j];
#pragma unroll
            for (int u = 0; u < 4; u++) r[u] += (o > k[u] || (o == k[u] && j < e0 + u * 32 + lane)) ? 1 : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (e0 + u * 32 + lane < c) dst[r[u]] = k[u];
    }
}

// s = fl(s + p[i]) for i = 0 .. c-1 (c a multiple of 8, zeros pad) until s >= target: the hit's index, or -1.
// The same in every lane; load(i, x) fetches elements i .. i + 7.
template <class Load>
__device__ __forceinline__ int serial_sum(const Load &load, int c, float target, float &s, float &before)
{
    if (c <= 0) return -1;
    float x[8], nx[8];
    load(0, nx);
    for (int b = 0; b < c; b += 8) {
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = nx[j];
        load(b + 8 < c ? b + 8 : 0, nx);
        float r = s;
#pragma unroll
        for (int j = 0; j < 8; j++) r = __fadd_rn(r, x[j]);
        if (r >= target) {
            int h = -1;
            float v = s;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (h < 0) {
                    before = v;
                    v = __fadd_rn(v, x[j]);
                    if (v >= target) h = b + j;
                }
            }
            s = v;
            return h;
        }
        s = r;
    }
    return -1;
}

// Histogram bins are ranges of exp values (0 < e <= 1), 128 to a binade, the last one at 1; a probability
// is a non-decreasing function of its exp value, so bins are ranges of probabilities in the same order.
constexpr unsigned kBinBase = 0x3F80u - (kBins - 1);  // upper 16 bits of the values of bin 0
__device__ __forceinline__ int row_bin(uint32_t ebits)
{
    const int b = (int)(ebits >> 16) - (int)kBinBase;
    return min(max(b, 0), kBins - 1);
}
__device__ __forceinline__ uint32_t row_bin_floor(int b) { return (kBinBase + (unsigned)b) << 16; }

// Softmax scale, then a filter that drops everything below a probability.  The filter is a comparison of exp
// values: fl(e * inv) is non-decreasing in e, so the smallest e it lets through says it all.
struct RowProb {
    float inv, e_min;
    __device__ __forceinline__ float operator()(float e) const { return e >= e_min ? __fmul_rn(e, inv) : 0.f; }
};
// the smallest e >= 0 with fl(e * inv) >= thr (thr > 0); false when it was not found near thr / inv
__device__ __forceinline__ bool smallest_e(float thr, float inv, float &e_min)
{
    uint32_t b = __float_as_uint(__fdiv_rn(thr, inv));
    int steps = 0;
    while (b > 0u && __fmul_rn(__uint_as_float(b - 1u), inv) >= thr && ++steps < 64) b--;
    while (!(__fmul_rn(__uint_as_float(b), inv) >= thr) && ++steps < 64) b++;
    e_min = __uint_as_float(b);
    return steps < 64;
}

__device__ __forceinline__ double pow2_double(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// P4 on rank 0: the nucleus bound and the binade of the sorted running sum at every bin from the mass
// histogram (steps (1) to (3) of topp_cut, stg_rowdist.cuh).  An estimate throughout: whatever it gets
// wrong is noticed by the exact sum of P6.
__device__ __forceinline__ void plan_bins(RowSh &sh, unsigned char *dyn, float top_p, double scale_p, bool complete)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned *mass = (unsigned *)(dyn + kOffBinMass);
    unsigned *dd = (unsigned *)(dyn + kOffBinD);
    unsigned char *bin_e = dyn + kOffBinE;
    if (tid == 0) sh.cut_lo = -1;
    // thread t: bins kBins - 1 - 8 t downwards
    const int b0 = kBins - 8 - tid * 8;
    double lm[8], tm = 0.0;
    int lc[8], tc = 0;
    {
        const uint4 q0 = *(const uint4 *)(mass + b0), q1 = *(const uint4 *)(mass + b0 + 4);
        const unsigned m[8] = {q1.w, q1.z, q1.y, q1.x, q0.w, q0.z, q0.y, q0.x};
        const uint4 h0 = *(const uint4 *)(dd + b0), h1 = *(const uint4 *)(dd + b0 + 4);
        const unsigned h[8] = {h1.w, h1.z, h1.y, h1.x, h0.w, h0.z, h0.y, h0.x};
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const unsigned pb = kBinBase + (unsigned)(b0 + 7 - j);  // upper 16 bits of the bin's values
            lc[j] = m[j] ? max(1, (int)((float)m[j] / (4111.5f + 32.f * (float)(pb & 127u)) + 0.5f)) : 0;
            // the mantissas were cut: half a unit each, and what those whose lower bits are known have above or below it
            lm[j] = ((double)m[j] + 0.5 * (double)lc[j] + (double)(int)h[j] * (1.0 / 2048.0)) * pow2_double((int)(pb >> 7) - 139) * scale_p;
            tm += lm[j];
            tc += lc[j];
        }
    }
    double im = warp_scan_d(tm);
    int ic = warp_scan_i(tc);
    if (lane == 31) { sh.red_d[warp] = im; sh.red_i[warp] = ic; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRW; k++)
        if (k < warp) { im += sh.red_d[k]; ic += sh.red_i[k]; }
    const double tp = (double)top_p;
    {
        double am = im - tm;
        int ac = ic - tc, best = -1;
        if (im >= tp && am <= tp * 1.01 + 1e-3) {  // the bin lies in one of a few threads' share
#pragma unroll
            for (int j = 0; j < 8; j++) {
                am += lm[j];
                ac += lc[j];
                if (best < 0 && lc[j]) {
                    const double need = tp * (1.0 + 1.0 / 65536.0) + (double)(16.f * sqrtf((float)ac) * 2.98e-8f) + 1e-7;
                    if (am >= need) best = max(b0 + 7 - j - 1, 0);
                }
            }
        }
        if (best >= 0) atomicMax(&sh.cut_lo, best);
    }
    __syncthreads();
    const int c_lo = max(sh.cut_lo, 0);
    const bool open = sh.cut_lo < 0;  // the mass never reaches top_p: every survivor stays
    // How near top_p a bin's sums have to lie for its elements to be handed over with the first.  Of a top_p near 1 they all do,
    // tens of thousands of them: there the bin in which the exact sum meets top_p is asked for when it is known, which takes
    // another round over the row.  16 rows of 151,936, T = 1.1, with 2^-14 everywhere / (1 - top_p) / 16 / (1 - top_p) / 64: top_p
    // 0.999 127 / 124 / 144 us, 0.9993 138 / 134 / 148, 0.9997 148 / 115 / 140, 0.9998 5,605 (all rows redone) / 199 / 193;
    // T = 0.7: 0.999 117 / 113 / 103, 0.9993 130 / 119 / 128, 0.9997 172 / 138 / 126.
    const double near = fmin(1.0 / 16384.0, (1.0 - tp) / 16.0);
    double before = im - tm;
    int ac = ic - tc;
    uint32_t eb[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int b = b0 + 7 - j;
        // the estimate is good to some 1e-5, and the sum to come drifts by as much
        const double lo = before * (1.0 - 1.0 / 16384.0), hi = (before + lm[j]) * (1.0 + 1.0 / 16384.0);
        const int e_lo = exp_of_double(lo);
        const bool order = lc[j] > 0 && (e_lo != exp_of_double(hi) || (before * (1.0 - near) <= tp && (before + lm[j]) * (1.0 + near) >= tp));
        const uint32_t v = b < c_lo ? 0u : (order ? (uint32_t)kBinOrder : (uint32_t)e_lo);
        eb[(7 - j) >> 2] |= v << (8 * ((7 - j) & 3));
        before += lm[j];
        ac += lc[j];
        if (b == c_lo) sh.n_cand = open && !complete ? INT_MAX : ac;
    }
    *(uint2 *)(bin_e + b0) = make_uint2(eb[0], eb[1]);
    *(uint4 *)(dd + b0) = make_uint4(0u, 0u, 0u, 0u);
    *(uint4 *)(dd + b0 + 4) = make_uint4(0u, 0u, 0u, 0u);
    if (tid < kBins / 32) sh.tie_bits[tid] = 0u;
    if (tid == 0) { sh.list_n = 0; sh.c_lo = c_lo; }
    __syncthreads();
}

// appends make(j) for the bits of `take` to a list in this CTA's shared memory (whole warps call it)
template <class T, class Make>
__device__ __forceinline__ void append(T *list, int cap, int *count, unsigned take, const Make &make)
{
    const int lane = threadIdx.x & 31;
    if (!__any_sync(0xFFFFFFFFu, take != 0u)) return;
    const int inc = warp_scan_i(__popc(take));
    int pos = 0;
    if (lane == 31) pos = atomicAdd(count, inc);
    pos = __shfl_sync(0xFFFFFFFFu, pos, 31) + inc - __popc(take);
#pragma unroll
    for (int j = 0; j < 8; j++)
        if ((take >> j) & 1u) {
            if (pos < cap) list[pos] = make(j);
            pos++;
        }
}

// P6 on rank 0: the sorted-order sum over the bins; sh.list_n elements of the bins whose order counts lie in
// the list.  Returns 0 when the cut is found, 1 when the row has to be redone, 2 when the elements of the bin in
// sh.new_bits have to be handed over as well (the sum meets top_p, or leaves the binade, in a bin that was
// taken without its order).
__device__ __forceinline__ int cut_bins(RowSh &sh, unsigned char *dyn, float top_p, const RowProb &prob)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned *fidx = (unsigned *)(dyn + kOffBinMass);         // bin -> its number among the bins whose order counts
    const unsigned *dd = (const unsigned *)(dyn + kOffBinD);
    const unsigned char *bin_e = dyn + kOffBinE;
    const uint32_t *list = (const uint32_t *)(dyn + kOffList);  // elements, and zeros that pad
    uint32_t *binned = (uint32_t *)(dyn + kOffWalk);          // [kRowList] by bin, padded with zeros to multiples of 8
    uint32_t *sorted = (uint32_t *)(dyn + kOffList);          // [kRowList] the same, every bin sorted (over the list)
    int4 *fd = (int4 *)(binned + kRowList);                   // [kFlagged] {increments above, first element, elements, binade above}
    int *cnt = (int *)(fd + kFlagged);                        // [kFlagged]
    static_assert(sizeof(WalkArea) >= kRowList * 4 + kFlagged * 20, "scratch of the cut");
    const int c_lo = sh.c_lo, n_list = sh.list_n;
    if (n_list > kRowList) return 1;  // the same for every thread
    for (int t = tid; t < kFlagged; t += kRT) cnt[t] = 0;
    if (tid < kBins / 32) sh.new_bits[tid] = 0u;
    int loc = 0, nf = 0;
    const int b0 = kBins - 8 - tid * 8;
    const unsigned ties = (sh.tie_bits[b0 >> 5] >> (b0 & 31)) & 0xFFu;
    unsigned char e8[8];
    *(uint2 *)e8 = *(const uint2 *)(bin_e + b0);
    unsigned d8[8];
    *(uint4 *)d8 = *(const uint4 *)(dd + b0);
    *(uint4 *)(d8 + 4) = *(const uint4 *)(dd + b0 + 4);
#pragma unroll
    for (int j = 7; j >= 0; j--) {
        const bool order = e8[j] == kBinOrder || ((ties >> j) & 1u);
        nf += order ? 1 : 0;
        loc += order || e8[j] == 0 ? 0 : (int)d8[j];
    }
    int f_run = nf, p_run = loc;
    block_scan_2(f_run, p_run, sh.red_i, sh.red_i2);
    if (tid == kRT - 1) { sh.n_flagged = f_run; sh.p_all = p_run; }
    f_run -= nf;
    p_run -= loc;
    __syncthreads();
    const int n_flag = sh.n_flagged;
    if (n_flag > kFlagged) return 1;
#pragma unroll
    for (int j = 7; j >= 0; j--) {
        const int b = b0 + j;
        if (e8[j] == kBinOrder || ((ties >> j) & 1u)) {
            sh.flagged[f_run] = (unsigned short)b;
            fidx[b] = (unsigned)f_run;
            // the binade of the unordered bins right above (they all have one); 0: none
            fd[f_run] = make_int4(p_run, 0, 0, b + 1 < kBins ? bin_e[b + 1] : 0);
            f_run++;
        } else if (e8[j] != 0) {
            p_run += (int)d8[j];
        }
    }
    __syncthreads();
    for (int i = tid; i < n_list; i += kRT)
        if (list[i]) atomicAdd(&cnt[fidx[row_bin(list[i])]], 1);
    __syncthreads();
    {
        static_assert(kFlagged == kRT, "one bin per thread");
        const int c = cnt[tid], padded = tid < n_flag ? (c + 7) & ~7 : 0;
        int incl = padded, none = 0;
        block_scan_2(incl, none, sh.red_i, sh.red_i2);
        if (tid == kRT - 1) sh.n_cand = incl;
        if (tid < n_flag) {
            fd[tid].y = incl - padded;
            fd[tid].z = c;
            cnt[tid] = incl - padded;
        }
    }
    __syncthreads();
    if (sh.n_cand > kRowList) return 1;
    if (tid == 0) sh.list_n = sh.n_cand;
    for (int i = tid; i < n_list; i += kRT) {
        const uint32_t e = list[i];
        if (e) binned[atomicAdd(&cnt[fidx[row_bin(e)]], 1)] = e;
    }
    __syncthreads();
    for (int i = warp; i < n_flag; i += kRW) {
        const int4 f = fd[i];
        warp_rank_sort(binned + f.y, sorted + f.y, f.z);
        if (lane < ((8 - (f.z & 7)) & 7)) sorted[f.y + f.z + lane] = 0u;
    }
    __syncthreads();
    if (warp == 0) {
        float s = 0.f, before = 0.f;
        int done = 0, hit_i = -1, hit = -1, more = -1;
        bool redo = false;
        int4 f = n_flag > 0 ? fd[0] : make_int4(0, 0, 0, 0);
        for (int i = 0; i <= n_flag; i++) {
            if (i == n_flag) f = make_int4(sh.p_all, 0, 0, bin_e[c_lo]);
            const int d = f.x - done;
            if (d) {
                // the unordered bins above this one
                const uint32_t sb = __float_as_uint(s);
                const int ef = (int)(sb >> 23);
                const unsigned at0 = (sb & 0x7FFFFFu) | 0x800000u, S = at0 + (unsigned)d;
                if (ef < 24 || f.w != ef) { redo = true; break; }
                const unsigned lim = (unsigned)min((long long)(1 << 24), target_units(top_p, true, ef));
                if (S >= lim) {
                    // in which bin?
                    unsigned at = at0;
                    int b = i > 0 ? sh.flagged[i - 1] - 1 : kBins - 1;
                    const int b_end = i < n_flag ? sh.flagged[i] : c_lo - 1;
                    for (; b > b_end; b -= 32) {
                        const int bb = b - lane;
                        const unsigned v = (unsigned)warp_scan_i(bb > b_end ? (int)dd[bb] : 0);
                        const unsigned m = __ballot_sync(0xFFFFFFFFu, at + v >= lim);
                        if (m) { b -= __ffs(m) - 1; break; }
                        at += __shfl_sync(0xFFFFFFFFu, v, 31);
                    }
                    if (b > b_end) more = b; else redo = true;
                    break;
                }
                s = __uint_as_float(((uint32_t)ef << 23) | (S & 0x7FFFFFu));
                done = f.x;
            }
            if (i == n_flag) break;
            const uint32_t *q = sorted + f.y;
            const int c = (f.z + 7) & ~7;
            if (i + 1 < n_flag) f = fd[i + 1];
            hit = serial_sum([&](int k, float x[8]) {
                const uint4 a = *(const uint4 *)(q + k), b = *(const uint4 *)(q + k + 4);
                x[0] = prob(__uint_as_float(a.x)); x[1] = prob(__uint_as_float(a.y)); x[2] = prob(__uint_as_float(a.z)); x[3] = prob(__uint_as_float(a.w));
                x[4] = prob(__uint_as_float(b.x)); x[5] = prob(__uint_as_float(b.y)); x[6] = prob(__uint_as_float(b.z)); x[7] = prob(__uint_as_float(b.w));
            }, c, top_p, s, before);
            if (hit >= 0) { hit_i = i; break; }
        }
        if (hit < 0 && more < 0 && c_lo > 0) redo = true;  // the bound was too tight
        int keep = 0, all = 0;
        float tstar = 0.f;
        if (!redo && hit >= 0) {
            const int4 g = fd[hit_i];
            const uint32_t *q = sorted + g.y;
            tstar = prob(__uint_as_float(q[hit]));
            for (int j = lane; j < g.z; j += 32)
                if (prob(__uint_as_float(q[j])) == tstar) { all++; keep += j <= hit ? 1 : 0; }
            all = __reduce_add_sync(0xFFFFFFFFu, all);
            keep = __reduce_add_sync(0xFFFFFFFFu, keep);
            // two exp values next to one another can have one probability: should the bin's edge lie between
            // them, its neighbours' tokens would tie with these
            const int b = sh.flagged[hit_i];
            if (b == 0 || prob(__uint_as_float(row_bin_floor(b) - 1u)) == tstar ||
                (b + 1 < kBins && prob(__uint_as_float(row_bin_floor(b + 1))) == tstar)) redo = true;
        }
        if (lane == 0) {
            sh.stop = redo ? 1 : (more >= 0 ? 2 : 0);
            if (more >= 0) sh.new_bits[more >> 5] |= 1u << (more & 31);  // not tie_bits: another CTA may still be reading those
            sh.tstar = tstar;
            sh.hit_keep = keep < all ? keep : 0;
            if (!redo && hit >= 0 && (s - top_p <= kNearTol || top_p - before <= kNearTol)) sh.flags |= kFlagNearCut;
            if (keep < all) sh.flags |= 1u << 4;
        }
    }
    __syncthreads();
    return sh.stop;
}

// s = fl(s + p) from 0, at most `count` times, until s >= target: the index of the addition that got there, -1 when none
// does.  One thread.  Inside a binade the sum grows by the same number of units with every addition behind the first (where p
// lies half way between two units, the first leaves the sum even, and from even sums the rounding always goes the same
// way), so a binade takes three additions and a division.
__device__ __forceinline__ int equal_sum(float p, int count, float target, float &s, float &before)
{
    s = 0.f;
    before = 0.f;
    for (int i = 0; i < count;) {
        before = s;
        s = __fadd_rn(s, p);
        if (s >= target) return i;
        i++;
        const uint32_t at0 = __float_as_uint(before), at = __float_as_uint(s), next = __float_as_uint(__fadd_rn(s, p));
        if (next == at) return -1;  // it stays there
        if ((at0 ^ at) >> 23 || (at ^ next) >> 23) continue;
        // floats >= 0 are ordered as their bits: as many more as stay below the target and the next binade
        const uint32_t d = next - at, end = min(((at >> 23) + 1u) << 23, __float_as_uint(target));
        const int k = min((int)((end - 1u - at) / d), count - i);
        if (k > 0) {
            s = __uint_as_float(at + (uint32_t)k * d);
            before = __uint_as_float(at + (uint32_t)(k - 1) * d);
            i += k;
        }
    }
    return -1;
}

// A row without a finite logit.  Softmax gives each of its tokens 1 / V (Sampler.cs:452-458): the filters and the draw
// are sums of equal addends, done by the first thread; where the distribution is asked for, every CTA of the cluster
// writes the tokens [lo, hi) of it.  Out of line: it is over in two microseconds, and k_row has no registers to spare.
__device__ __noinline__ void uniform_row(const SampleArgs &a, const RowPlan &rp, RowSh &sh, int row, int rank, int lo, int hi, u64 rk)
{
    const int tid = threadIdx.x, n = a.vocab;
    if (tid == 0) {
        RowDist d;
        d.flags = kDistUniform;
        d.uniform_p = __fdiv_rn(1.0f, (float)n);
        d.max_x = -CUDART_INF_F;
        d.inv_t = rp.temperature != 1.0f ? __fdiv_rn(1.0f, rp.temperature) : 1.0f;
        d.inv1 = 1.f; d.kth = 0.f; d.inv2 = 1.f; d.minp_thr = 0.f; d.tstar = 0.f; d.inv3 = 1.f;
        d.tie_idx_max = INT_MAX;
        d.argmax = rk ? key_idx(rk) : 0;
        d.sum_end = 0.f;
        int kept = n;  // the first `kept` tokens
        float s, before;
        if (rp.min_p > 0.f) {
            d.minp_thr = __fmul_rn(rp.min_p, d.uniform_p);
            d.flags |= kDistMinP;
            if (d.uniform_p < d.minp_thr) kept = 0;
        }
        if (rp.top_p < 1.0f && rp.top_p > 0.f && kept > 0) {
            const int hit = equal_sum(d.uniform_p, n, rp.top_p, s, before);
            d.flags |= kDistTopP;
            if (hit >= 0) {
                kept = hit + 1;
                d.tstar = d.uniform_p;
                if (s - rp.top_p <= kNearTol || rp.top_p - before <= kNearTol) sh.flags |= kFlagNearCut;
                if (kept < n) { sh.flags |= 1u << 4; d.tie_idx_max = hit; }
            }
        }
        const float s3 = (float)((double)kept * (double)d.uniform_p);
        if (s3 > 0.f && s3 != 1.0f) { d.flags |= kDistScale3; d.inv3 = __fdiv_rn(1.0f, s3); }
        sh.dist = d;
        if (rank == 0) {
            if (a.mode == 2) a.dists[row] = d;
            if (a.mode == 1 && a.row_flags) a.row_flags[row] = kPathFull | sh.flags;
            if (a.mode == 0 || a.mode == 3) {
                const float u01 = a.uniforms ? __ldg(a.uniforms + row) : 0.5f;
                const int hit = u01 > 0.f ? equal_sum(eval_p3(d.uniform_p, 0, d), kept, u01, s, before) : 0;
                const int tok = hit >= 0 ? hit : n - 1;
                uint32_t fl = kPathFull | sh.flags | (1u << 6);
                if (hit < 0) fl |= 1u << 5;
                else if (u01 > 0.f && (u01 - before <= kNearTol || s - u01 <= kNearTol)) fl |= kFlagNearBoundary;
                a.tokens[row] = tok;
                if (a.token_probs) a.token_probs[row] = eval_p3(d.uniform_p, tok, d);
                if (a.row_flags) a.row_flags[row] = fl;
                count_row_flags(a.counters, fl);
            }
        }
    }
    if ((a.mode == 1 || a.mode == 3) && a.dist_out) {
        __syncthreads();
        const RowDist d = sh.dist;
        float *o = a.dist_out + (int64_t)row * n;
        for (int i = lo + tid; i < hi; i += kRT) o[i] = eval_p3(d.uniform_p, i, d);
    }
}

// ---- the kernel ----------------------------------------------------------------------------------------
// CLOSE: for batches with masks (the code that closes rows up costs the other batches 3 %)
template <bool BF16, bool CLOSE>
__global__ void __launch_bounds__(kRT, 2) k_row(const __grid_constant__ SampleArgs a, const RowWs ws, const int want_argmax)
{
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ RowSh sh;
    cg::cluster_group cl = cg::this_cluster();
    cl.barrier_arrive();  // waited for before the first push: another CTA's shared memory is there once that CTA runs
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fi = blockIdx.x / C;
    const int row = a.items[fi].row;
    const RowPlan &rp = a.plans[row];
    int n = a.vocab, nsub = (n + kSub - 1) / kSub;
    int per = (nsub + C - 1) / C;
    int t0 = min(rank * per, nsub), t1 = min(t0 + per, nsub);  // this CTA's tiles
    WalkArea *wa = (WalkArea *)(dyn + kOffWalk);
    WalkArea *dst = rank == 0 ? wa : (WalkArea *)cl.map_shared_rank((unsigned char *)wa, 0);
    RowSh *sh0 = rank == 0 ? &sh : cl.map_shared_rank(&sh, 0);
    float *e = ws.e + (size_t)fi * ws.e_stride;
    unsigned long long *tk = a.phase_ticks && rank == 0 ? a.phase_ticks + (int64_t)fi * 32 : nullptr;
    tick(tk, 0);

    const float temperature = rp.temperature;
    const bool greedy = temperature <= 0.f;
    const float top_p = rp.top_p, min_p = rp.min_p;
    const bool want_topp = top_p < 1.0f && top_p > 0.f;
    RowSrc<BF16> src;
    src.rowp = LogitRow{(const char *)a.logits + (int64_t)row * a.row_stride * (BF16 ? 2 : 4), a.softcap};
    src.mrow = (rp.use_mask && a.mask) ? a.mask + (int64_t)row * a.mask_stride : nullptr;
    src.n = n;
    src.scale = !greedy && temperature != 1.0f;
    src.inv_t = src.scale ? __fdiv_rn(1.0f, temperature) : 1.0f;
    {
        const unsigned al = (unsigned)(uintptr_t)src.rowp.p;
        src.vec = BF16 ? ((al & 15u) == 0u ? 8 : (al & 7u) == 0u ? 4 : 1) : ((al & 31u) == 0u ? 8 : (al & 15u) == 0u ? 4 : 1);
    }
    src.tab = nullptr;
    src.tab_mask = 0;
    bool small_table = true;
    if (tid == 0) { sh.flags = 0u; sh.n_cand = 0; sh.list_n = 0; sh.stop = 0; sh.hit_keep = 0; sh.tie_idx = INT_MAX; }
    {
        const int nh = rp.has_penalty ? rp.hist_len : 0, nb = greedy ? 0 : rp.bias_len;
        if (nh + nb > 0) {
            int slots = 64;
            while (slots < 2 * (nh + nb)) slots <<= 1;
            small_table = slots <= kSmallTable;
            unsigned char *tab = dyn + (small_table ? kOffList : 0);
            build_table<BF16>(a, rp, src, tab, slots, nh, nb, t0 * kSub, min(n, t1 * kSub));
            src.tab = tab;
            src.tab_mask = slots - 1;
        }
    }
    unsigned *mass = (unsigned *)(dyn + kOffBinMass);
    unsigned *dd = (unsigned *)(dyn + kOffBinD);
    unsigned char *bin_e = dyn + kOffBinE;
    auto clear_bins = [&]() {
        for (int b = tid; b < kBins / 2; b += kRT) ((uint4 *)mass)[b] = make_uint4(0u, 0u, 0u, 0u);  // mass and dd
    };
    if (want_topp && small_table) clear_bins();
    tick(tk, 1);

    // A row behind a mask that allows at most half of the vocabulary is closed up as it is read: its allowed tokens, in
    // order, are the row from here on (what is masked has probability zero, which no sum sees), and `ids` knows
    // which tokens they were.  64 rows of 262,144 behind masks of 0.1 to 30 %: 191 us as whole rows, 119 closed up.
    int32_t *ids = nullptr;
    int first_id = 0;  // of this CTA's allowed tokens, in the closed-up row
    int *tile_at = (int *)sh.tile_sum;
    const bool counted = CLOSE && src.mrow != nullptr && !greedy && a.mode == 0;  // the same for every thread of the cluster
    if (counted) {
        // a word per lane, four tiles to a load
        for (int g = t0 + 4 * warp; g < t1; g += 4 * kRW) {
            const int t = g + lane / 8, base = g * kSub + lane * 32;
            uint32_t w = 0u;
            if (t < t1 && base < n) {
                w = __ldg(src.mrow + (base >> 5));
                if (base + 32 > n) w &= (1u << (n - base)) - 1u;
            }
            int c = __popc(w);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
            if ((lane & 7) == 0 && t < t1) tile_at[t - t0] = c;
        }
        __syncthreads();
        cl.barrier_wait();
        if (warp == 0) {
            int run = 0;
            for (int b = 0; b < t1 - t0; b += 32) {
                const int c = b + lane < t1 - t0 ? tile_at[b + lane] : 0, inc = warp_scan_i(c);
                if (b + lane < t1 - t0) tile_at[b + lane] = run + inc - c;
                run += __shfl_sync(0xFFFFFFFFu, inc, 31);
            }
            if (lane < C) cl.map_shared_rank(&sh, lane)->cnt[rank] = run;
        }
        cl.sync();
        int total = 0;
        for (int r = 0; r < C; r++) {
            if (r == rank) first_id = total;
            total += sh.cnt[r];
        }
        if (total <= n / 2) {
            ids = ws.ids + (size_t)fi * ws.e_stride;
            n = total;
        }
    }

    // P1: the maximum, and for the tiles' sums of exp values estimates that need no maximum
    float2 *est = (float2 *)wa->comp;
    TilePrefix tp{0.0, 0.0, 0.0, 0.0};
    {
        float best = -CUDART_INF_F, cmax = -CUDART_INF_F;  // cmax: what the CTA's estimates are relative to
        u64 key = 0ull, raw = 0ull;
        if (CLOSE && ids != nullptr) {
            float nx[8];
            unsigned nbits = 0u;
            if (t0 + warp < t1) src.fetch((t0 + warp) * kSub + lane * 8, nx, nbits);
#pragma unroll 1
            for (int t = t0 + warp; t < t1; t += kRW) {  // the next tile's logits on the way, as in for_tiles
                const int base = t * kSub + lane * 8;
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; j++) x[j] = nx[j];
                const unsigned bits = nbits;
                if (t + kRW < t1) src.fetch(base + kRW * kSub, nx, nbits);
                if (!__any_sync(0xFFFFFFFFu, bits != 0u)) continue;
                src.mask(x, bits, base);  // what is not allowed is -infinity
                src.adjust(x, base);
                const int c = __popc(bits);
                const int at = first_id + tile_at[t - t0] + warp_scan_i(c) - c;
                float *ep = e + at;
                int32_t *ip = ids + at;
                if (__reduce_max_sync(0xFFFFFFFFu, (unsigned)c) <= 2u) {  // few: one after the other (64 rows of 262,144 behind masks of 1 % 64 -> 58 us)
                    unsigned left = bits;
#pragma unroll 1
                    while (__any_sync(0xFFFFFFFFu, left != 0u)) {
                        const int j = __ffs(left) - 1;
                        float v = x[0];
#pragma unroll
                        for (int q = 1; q < 8; q++) v = q == j ? x[q] : v;
                        if (left) {
                            best = fmaxf(best, v);
                            *ep++ = v;
                            *ip++ = base + j;
                            left &= left - 1u;
                        }
                    }
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const unsigned on = (bits >> j) & 1u;
                    best = fmaxf(best, on ? x[j] : -CUDART_INF_F);
                    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p st.global.f32 [%1], %2;\n @p st.global.s32 [%3], %4;\n}"
                                 ::"r"(on), "l"(ep), "f"(x[j]), "l"(ip), "r"(base + j) : "memory");  // by a predicate, as in add_if
                    ep += on;
                    ip += on;
                }
            }
            best = block_max_f(best, sh.red_f);
            if (best > -CUDART_INF_F) key = make_key(best, 0);
            nsub = (n + kSub - 1) / kSub;
            per = (nsub + C - 1) / C;
            t0 = min(rank * per, nsub);
            t1 = min(t0 + per, nsub);
        } else if (greedy || want_argmax) {
            // the (value, lowest index) keys: of the adjusted row (a greedy row's token), of the raw one
            float rbest = -CUDART_INF_F;
            int best_i = -1, rbest_i = -1;
            for (int t = t0 + warp; t < t1; t += kRW) {
                const int base = t * kSub + lane * 8;
                float x[8];
                unsigned bits;
                src.fetch(base, x, bits);
                src.mask(x, bits, base);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (x[j] > rbest) { rbest = x[j]; rbest_i = base + j; }
                src.override_(x, base);
                src.rescale(x);
                if (!greedy) cmax = fmaxf(cmax, estimate_tile(x, est + t));
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (x[j] > best) { best = x[j]; best_i = base + j; }
            }
            key = block_max_k(best_i >= 0 ? make_key(best, best_i) : 0ull, sh.red_k);
            __syncthreads();
            raw = block_max_k(rbest_i >= 0 ? make_key(rbest, rbest_i) : 0ull, sh.red_k);
            cmax = block_max_f(cmax, sh.red_f);
        } else {
            for (int t = t0 + warp; t < t1; t += 2 * kRW) {
                float x[2][8];
                unsigned bits[2];
                const int b0 = t * kSub + lane * 8, b1 = b0 + kRW * kSub;
                src.fetch(b0, x[0], bits[0]);
                const bool two = t + kRW < t1;
                if (two) src.fetch(b1, x[1], bits[1]);
                src.mask(x[0], bits[0], b0);
                src.adjust(x[0], b0);
                cmax = fmaxf(cmax, estimate_tile(x[0], est + t));
                if (two) {
                    src.mask(x[1], bits[1], b1);
                    src.adjust(x[1], b1);
                    cmax = fmaxf(cmax, estimate_tile(x[1], est + t + kRW));
                }
            }
            best = cmax = block_max_f(cmax, sh.red_f);
            if (best > -CUDART_INF_F) key = make_key(best, 0);
        }
        if (!greedy && !(CLOSE && ids != nullptr)) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int i = 2 * tid + u;
                if (t0 + i < t1) {
                    const float2 v = est[t0 + i];
                    sh.tile_sum[i] = v.x > -CUDART_INF_F ? v.y * exp2_approx((v.x - cmax) * kLog2E) : v.y;  // of nothing but -infinity 0
                }
            }
            tp = tile_prefix(sh.tile_sum, t1 - t0, sh.red_d);
        }
        if (!counted) cl.barrier_wait();
        if (tid < C) {
            RowSh *o = cl.map_shared_rank(&sh, tid);
            o->maxkey[rank] = key;
            o->rawkey[rank] = raw;
            o->cmax[rank] = cmax;
            o->tot[0][rank] = tp.all;
        }
        cl.sync();
    }
    u64 mk = 0ull, rk = 0ull;
    for (int r = 0; r < C; r++) {
        mk = sh.maxkey[r] > mk ? sh.maxkey[r] : mk;
        rk = sh.rawkey[r] > rk ? sh.rawkey[r] : rk;
    }
    tick(tk, 2);
    if (greedy) {
        const int tok = mk ? key_idx(mk) : 0;
        if (a.mode == 2) {
            if (rank == 0 && tid == 0) {
                RowDist d;
                memset(&d, 0, sizeof(d));
                d.flags = kDistOneHot;
                d.tie_idx_max = tok;
                d.argmax = tok;
                d.inv_t = 1.f; d.inv1 = 1.f; d.inv2 = 1.f; d.inv3 = 1.f;
                a.dists[row] = d;
                ws.redo[fi] = 0;
            }
            return;
        }
        if ((a.mode == 1 || a.mode == 3) && a.dist_out) {
            float *o = a.dist_out + (int64_t)row * n;
            for (int i = t0 * kSub + tid; i < min(n, t1 * kSub); i += kRT) o[i] = i == tok ? 1.f : 0.f;
        }
        if (rank == 0 && tid == 0) {
            if (a.tokens) a.tokens[row] = tok;
            if (a.token_probs) a.token_probs[row] = 1.f;
            if (a.row_flags) a.row_flags[row] = (uint32_t)rp.path | (mk ? 0u : (1u << 6));
            ws.redo[fi] = 0;
        }
        return;
    }
    if (a.row_drill == 1) {
        if (rank == 0 && tid == 0) ws.redo[fi] = 1;
        return;
    }
    if (mk == 0ull) {  // nothing finite; [t0, t1) may be tiles of the closed-up row, but that is of no distribution
        if (rank == 0 && tid == 0) ws.redo[fi] = 0;
        uniform_row(a, rp, sh, row, rank, t0 * kSub, min(n, t1 * kSub), rk);
        return;
    }
    const float mx = key_val(mk);

    double base = 0.0, all = 0.0;
    float own = 1.f;  // what the CTA's estimates are to be multiplied by
    if (CLOSE && ids != nullptr) {
        // the closed-up row's tiles, now that the maximum is known
        for (int t = t0 + warp; t < t1; t += kRW) {
            const int b = t * kSub + lane * 8;
            float x[8], acc = 0.f;
            load_e(e, b, x);
#pragma unroll
            for (int j = 0; j < 8; j++) acc += b + j < n ? exp2_approx((x[j] - mx) * kLog2E) : 0.f;
            acc = warp_sum_f(acc);
            if (lane == 0) sh.tile_sum[t - t0] = acc;
        }
        tp = tile_prefix(sh.tile_sum, t1 - t0, sh.red_d);
        if (tid < C) cl.map_shared_rank(&sh, tid)->tot[1][rank] = tp.all;
        cl.sync();
        for (int r = 0; r < C; r++) {
            if (r == rank) base = all;
            all += sh.tot[1][r];
        }
    } else {
        float cmax = -CUDART_INF_F;
        for (int r = 0; r < C; r++) cmax = fmaxf(cmax, sh.cmax[r]);
        for (int r = 0; r < C; r++) {
            const float f = exp2_approx((sh.cmax[r] - cmax) * kLog2E);
            if (r == rank) { base = all; own = f; }
            all += sh.tot[0][r] * (double)f;
        }
    }
    guess_tiles(sh, tp, t0, t1, base, (double)own, all, CUDART_INF);
    tick(tk, 3);

    // P2: exp values, the tiles' compositions, and the histogram of the exp values (where the override table leaves room;
    // else in P3).  Masses are of the upper 13 mantissa bits, completed by the lower 11 (less their middle, in the increments'
    // array) of the at most 16,383 values that weigh something: their signed sum stays within 2^24.  Values below tau are left
    // out: all of them together cannot be more than half of what the nucleus may leave behind.
    // Values below minp_e cannot reach min-p's threshold, whatever the sum is: fl(e * inv) >= fl(min_p * inv) takes an
    // e >= min_p * (1 - 2^-23).  A mass that holds more than the survivors' makes the bound too high.
    const float minp_e = min_p > 0.f ? min_p * (1.0f - 1.0f / 1048576.0f) : 0.f;
    const float tau = 0.5f * (1.0f - top_p) * (float)(all / (double)n);
    const float floor_e = fmaxf(tau, minp_e), heavy_e = (float)(all * (1.0 / 16384.0));
    auto to_bins = [&](const float (&x)[8]) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t eb = __float_as_uint(x[j]), m = (eb & 0x7FFFFFu) | 0x800000u;
            const int b = row_bin(eb);
            add_if(x[j] > floor_e, mass + b, m >> 11);
            add_if(x[j] > fmaxf(floor_e, heavy_e), dd + b, (m & 2047u) - 1024u);
        }
    };
    if (CLOSE && ids != nullptr) {
        for (int t = t0 + warp; t < t1; t += kRW) {
            const int b = t * kSub + lane * 8;
            float x[8];
            load_e(e, b, x);
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = b + j < n ? expf(__fsub_rn(x[j], mx)) : 0.f;
            store_e(e, b, x);
            compose_tile(sh, wa, dst, x, t, t0);
            if (want_topp && small_table) to_bins(x);
        }
    } else {
        // one tile at a time, the next one's logits on the way
        float nx[8];
        unsigned nbits = 0u;
        if (t0 + warp < t1) src.fetch((t0 + warp) * kSub + lane * 8, nx, nbits);
#pragma unroll 1
        for (int t = t0 + warp; t < t1; t += kRW) {
            const int at = t * kSub + lane * 8;
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = nx[j];
            const unsigned bits = nbits;
            if (t + kRW < t1) src.fetch(at + kRW * kSub, nx, nbits);
            src.mask(x, bits, at);
            src.adjust(x, at);
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = expf(__fsub_rn(x[j], mx));  // 0 beyond the row, whose logits read as -inf
            store_e(e, at, x);
            compose_tile(sh, wa, dst, x, t, t0);
            if (want_topp && small_table) to_bins(x);
        }
    }
    __syncthreads();
    runs_of_tiles(sh, wa, dst, t0, t1);
    if (want_topp && !small_table) clear_bins();
    cl.sync();
    tick(tk, 4);

    auto get_e = [&](int t, float x[8]) { load_e(e, t * kSub + lane * 8, x); };
    // P3: the exact sum on rank 0's first warp; beside it the other CTAs' histograms go to rank 0
    if (rank == 0 && warp == 0) {
        const WalkOut o = row_walk(wa, get_e, n, nsub, 0.f, false);
        if (lane < C) cl.map_shared_rank(&sh, lane)->sum = o.s;
    } else if (want_topp && !small_table) {
        const int w0 = rank == 0 ? warp - 1 : warp, wn = rank == 0 ? kRW - 1 : kRW;
        for (int t = t0 + w0; t < t1; t += wn) {
            float x[8];
            get_e(t, x);
            to_bins(x);
        }
    }
    if (!small_table) __syncthreads();
    if (want_topp && rank != 0) {
        unsigned *m0 = cl.map_shared_rank(mass, 0), *h0 = cl.map_shared_rank(dd, 0);
        for (int b = tid; b < kBins; b += kRT) {
            const unsigned v = mass[b], w = dd[b];
            if (v) atomicAdd(&m0[b], v);
            if (w) { atomicAdd(&h0[b], w); dd[b] = 0u; }
        }
    }
    cl.sync();
    tick(tk, 5);
    const float sum = sh.sum;
    RowDist d;
    d.flags = 0;
    d.inv_t = src.inv_t;
    d.max_x = mx;
    d.tie_idx_max = INT_MAX;
    d.kth = 0.f; d.inv2 = 1.f; d.minp_thr = 0.f; d.tstar = 0.f; d.inv3 = 1.f; d.inv1 = 1.f;
    d.uniform_p = 0.f; d.sum_end = 0.f; d.argmax = rk ? key_idx(rk) : 0;
    if (sum > 0.f && sum != 1.0f) { d.flags |= kDistScale1; d.inv1 = __fdiv_rn(1.0f, sum); }
    RowProb fin{d.inv1, 0.f};  // an exp value's final probability, before Normalize
    bool in_reach = true;      // the filters' smallest exp values were found
    if (min_p > 0.f) {
        // ApplyMinP (Sampler.cs:493-503): the largest probability belongs to exp value 1
        d.minp_thr = __fmul_rn(min_p, d.inv1);
        d.flags |= kDistMinP;
        if (d.minp_thr > 0.f) in_reach = smallest_e(d.minp_thr, d.inv1, fin.e_min);
    }
    if (!in_reach) {  // the same for every thread of the cluster
        if (rank == 0 && tid == 0) ws.redo[fi] = 1;
        return;
    }
    const RowProb prob = fin;
    const bool dist_mode = (a.mode == 1 || a.mode == 3) && a.dist_out;
    const float u01 = a.uniforms ? __ldg(a.uniforms + row) : 0.5f;
    auto write_dist = [&]() {
        float *o = a.dist_out + (int64_t)row * n;
        for (int t = t0 + warp; t < t1; t += kRW) {
            const int b = t * kSub + lane * 8;
            float x[8];
            load_e(e, b, x);
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = eval_p3(x[j], b + j, d);
            if (b + 8 <= n && ((uintptr_t)(o + b) & 15) == 0) {
                *(float4 *)(o + b) = make_float4(x[0], x[1], x[2], x[3]);
                *(float4 *)(o + b + 4) = make_float4(x[4], x[5], x[6], x[7]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (b + j < n) o[b + j] = x[j];
            }
        }
    };
    // hit: the element of the row the draw met, -1: none.  One thread.
    auto write_row = [&](int hit, uint32_t fl) {
        if (a.row_drill == 2) { ws.redo[fi] = 1; return; }
        int tok = hit >= 0 ? (CLOSE && ids ? ids[hit] : hit) : a.vocab - 1, at = hit >= 0 ? hit : n - 1;
        if (hit < 0) fl |= 1u << 5;
        if (!(u01 > 0.f)) { tok = 0; at = 0; fl &= ~(1u << 5); }  // the first token meets such a target whatever its probability
        const float prob_tok = CLOSE && ids && ids[at] != tok ? 0.f : eval_p3(__ldcg(e + at), at, d);
        a.tokens[row] = tok;
        if (a.token_probs) a.token_probs[row] = prob_tok;
        if (a.row_flags) a.row_flags[row] = fl;
        count_row_flags(a.counters, fl);
        ws.redo[fi] = 0;
    };

    if (want_topp) {
        if (rank == 0) {
            // every survivor is in the histogram when the min-p threshold lies above tau
            plan_bins(sh, dyn, top_p, (double)d.inv1, minp_e > tau);
            if (tid < C) {
                RowSh *o = cl.map_shared_rank(&sh, tid);
                o->c_lo = sh.c_lo;
                o->narrow = sh.n_cand <= kNarrow - 64 ? 1 : 0;
            }
            __syncthreads();
            if (tid == 0) sh.n_cand = 0;
        }
        cl.sync();
        tick(tk, 6);
        const int c_lo = sh.c_lo;
        const float lo_e = __uint_as_float(c_lo > 0 ? row_bin_floor(c_lo) : 1u);
        if (sh.narrow) {
            u64 *keys = (u64 *)(dyn + kOffList);
            u64 *keys0 = rank == 0 ? keys : cl.map_shared_rank(keys, 0);
            for_tiles(t0 + warp, t1, kRW, get_e, [&](int t, float (&x)[8]) {
                unsigned take = 0u;
#pragma unroll
                for (int j = 0; j < 8; j++) take |= x[j] >= lo_e && prob(x[j]) > 0.f ? 1u << j : 0u;
                append(keys, kNarrow, rank == 0 ? &sh.n_cand : &sh.list_n, take, [&](int j) {
                    return ((u64)__float_as_uint(prob(x[j])) << 32) | (u64)(0xFFFFFFFFu - (uint32_t)(t * kSub + lane * 8 + j));
                });
            });
            __syncthreads();
            if (rank != 0 && sh.list_n > 0) {
                if (tid == 0) sh.n_cand = atomicAdd(&sh0->n_cand, sh.list_n);
                __syncthreads();
                const int at = sh.n_cand;
                for (int i = tid; i < min(sh.list_n, kNarrow); i += kRT)
                    if (at + i < kNarrow) keys0[at + i] = keys[i];
            }
            cl.sync();
            tick(tk, 7);
            if (rank != 0) {
                if (!dist_mode) return;
                cl.sync();
                if (sh.stop) return;
                d = sh.dist;
                write_dist();
                return;
            }
            const int nc = sh.n_cand;
            bool redo = nc > kNarrow || nc == 0;
            int kept = 0;
            if (!redo) {
                int p2 = 64;
                while (p2 < nc) p2 <<= 1;
                for (int i = nc + tid; i < p2; i += kRT) keys[i] = 0ull;
                __syncthreads();
                row_sort_desc(keys, p2);
                tick(tk, 8);
                if (warp == 0) {
                    float s = 0.f, before = 0.f;
                    const uint32_t *hi = (const uint32_t *)keys + 1;
                    const int hit = serial_sum([&](int i, float x[8]) {
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            const uint4 q = *(const uint4 *)(keys + i + j);
                            x[j] = __uint_as_float(q.y);
                            x[j + 1] = __uint_as_float(q.w);
                        }
                    }, (nc + 7) & ~7, top_p, s, before);
                    const int last = hit >= 0 ? hit : nc - 1;
                    if (lane == 0) {
                        sh.stop = hit < 0 && c_lo > 0 ? 1 : 0;
                        sh.cut_lo = last;
                        sh.tstar = hit >= 0 ? __uint_as_float(hi[2 * hit]) : 0.f;
                        sh.tie_idx = INT_MAX;
                        if (hit >= 0 && (s - top_p <= kNearTol || top_p - before <= kNearTol)) sh.flags |= kFlagNearCut;
                        if (hit >= 0 && hit + 1 < nc && hi[2 * hit] == hi[2 * hit + 2]) {
                            // equal probabilities at the cut: the kept ones are a prefix by token id
                            sh.flags |= 1u << 4;
                            sh.tie_idx = key_idx(keys[hit]);
                        }
                    }
                }
                __syncthreads();
                redo = sh.stop != 0;
                kept = sh.cut_lo + 1;
            }
            if (redo) {
                if (tid == 0) ws.redo[fi] = 1;
                if (dist_mode) {
                    if (tid < C) cl.map_shared_rank(&sh, tid)->stop = 1;
                    cl.sync();
                }
                return;
            }
            double part = 0.0;
            for (int i = tid; i < kept; i += kRT) part += (double)__uint_as_float((uint32_t)(keys[i] >> 32));
            const float s3 = (float)block_sum_d(part, sh.red_d);
            d.flags |= kDistTopP;
            d.tstar = sh.tstar;
            d.tie_idx_max = sh.tie_idx;
            if (s3 > 0.f && s3 != 1.0f) { d.flags |= kDistScale3; d.inv3 = __fdiv_rn(1.0f, s3); }
            if (dist_mode) {
                if (tid < C) cl.map_shared_rank(&sh, tid)->dist = d;
                cl.sync();
                write_dist();
            }
            if (a.mode == 1) {
                if (tid == 0) { if (a.row_flags) a.row_flags[row] = kPathFull | sh.flags; ws.redo[fi] = 0; }
                return;
            }
            if (a.mode == 2) {
                if (tid == 0) { a.dists[row] = d; ws.redo[fi] = 0; }
                return;
            }
            // the draw (SampleFromDistribution, Sampler.cs:564-576) over the kept tokens in token order: the
            // others add nothing to the sum
            int p2 = 64;
            while (p2 < kept) p2 <<= 1;
            for (int i = tid; i < p2; i += kRT) {
                const u64 k = keys[i];
                keys[i] = i < kept ? (k << 32) | (k >> 32) : 0ull;
            }
            __syncthreads();
            row_sort_desc(keys, p2);
            tick(tk, 9);
            if (warp == 0) {
                float s = 0.f, before = 0.f;
                const int hit = serial_sum([&](int i, float x[8]) {
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const uint4 q = *(const uint4 *)(keys + i + j);
                        x[j] = __fmul_rn(__uint_as_float(q.x), d.inv3);
                        x[j + 1] = __fmul_rn(__uint_as_float(q.z), d.inv3);
                    }
                }, (kept + 7) & ~7, u01, s, before);
                if (lane == 0) {
                    uint32_t fl = kPathFull | sh.flags;
                    if (hit >= 0 && u01 > 0.f && (u01 - before <= kNearTol || s - u01 <= kNearTol)) fl |= kFlagNearBoundary;
                    write_row(hit >= 0 ? key_idx(keys[hit] >> 32) : -1, fl);
                }
            }
            tick(tk, 10);
            return;
        }
        // P5: increments per bin
        if (rank != 0) {
            const uint4 *s4 = (const uint4 *)cl.map_shared_rank(bin_e, 0);
            if (tid < kBins / 16) ((uint4 *)bin_e)[tid] = s4[tid];
            __syncthreads();
        }
        unsigned *dd0 = rank == 0 ? dd : cl.map_shared_rank(dd, 0);
        uint32_t *list = (uint32_t *)(dyn + kOffList);
        uint32_t *list0 = rank == 0 ? list : cl.map_shared_rank(list, 0);
        // this CTA's part of the elements to sort goes to rank 0 in one piece
        auto hand_over = [&]() {
            __syncthreads();
            const int m = sh.list_n;
            if (rank != 0 && m > 0) {
                if (tid == 0) sh.n_cand = atomicAdd(&sh0->list_n, m);
                __syncthreads();
                const int at = sh.n_cand;
                for (int i = tid; i < min(m, kRowList); i += kRT)
                    if (at + i < kRowList) list0[at + i] = list[i];
            }
        };
        for_tiles(t0 + warp, t1, kRW, get_e, [&](int, float (&x)[8]) {
            unsigned take = 0u, odd = 0u;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float p = prob(x[j]);
                const int b = row_bin(__float_as_uint(x[j])), be = bin_e[b];
                const bool in = x[j] >= lo_e && p > 0.f, order = be == kBinOrder;
                // the increment in units of the running sum, as in tile_composite
                const float c = __uint_as_float(((uint32_t)be << 23) | 0x400000u), y = __fadd_rn(p, c);
                const bool plain = be >= 48 && p < __uint_as_float((uint32_t)(be - 1) << 23) &&
                                   fabsf(__fsub_rn(p, __fsub_rn(y, c))) != __uint_as_float((uint32_t)(be - 24) << 23);
                take |= in && order ? 1u << j : 0u;
                odd |= in && !order && !plain ? 1u << j : 0u;
                add_if(in && !order && plain, dd + b, (unsigned)(__float_as_int(y) - __float_as_int(c)));
            }
            // a rounding tie, or nearly as large as the sum
#pragma unroll 1
            while (odd) {
                const int q = __ffs(odd) - 1;
                odd &= odd - 1u;
                float v = x[0];
#pragma unroll
                for (int j = 1; j < 8; j++) v = j == q ? x[j] : v;
                const int b = row_bin(__float_as_uint(v));
                int d0, d1;
                unit_incr(prob(v), bin_e[b], d0, d1);
                if (d0 != d1) atomicOr(&sh0->tie_bits[b >> 5], 1u << (b & 31));
                if (d0) atomicAdd(&dd[b], (unsigned)d0);
            }
            append(list, kRowList, &sh.list_n, take, [&](int j) { return __float_as_uint(x[j]); });
        });
        hand_over();
        if (rank != 0)
            for (int b = tid; b < kBins; b += kRT) {
                const unsigned v = dd[b];
                if (v) atomicAdd(&dd0[b], v);
            }
        cl.sync();
        tick(tk, 7);
        for (int round = 0;; round++) {
            // bins with an exact rounding tie, or that the sum asked for: their order counts too.  Whether there are any
            // decides about the barrier below, so every CTA has to see the same bits: rank 0's tie_bits stand still
            // from the barrier above until all have passed the one that ends the first round, and its
            // new_bits from there to the barrier in the block (a further round always has a bit).
            if (tid < kBins / 32) {
                const unsigned bits = round == 0 ? sh0->tie_bits[tid] : sh0->new_bits[tid];
                sh.new_bits[tid] = bits;
                if (rank == 0 && round > 0) sh.tie_bits[tid] |= bits;
            }
            if (__syncthreads_or(tid < kBins / 32 && sh.new_bits[tid] != 0u)) {
                if (rank != 0) {
                    if (tid == 0) sh.list_n = 0;
                    __syncthreads();
                }
                for_tiles(t0 + warp, t1, kRW, get_e, [&](int, float (&x)[8]) {
                    unsigned take = 0u;
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (x[j] >= lo_e) {
                            const int b = row_bin(__float_as_uint(x[j]));
                            if (((sh.new_bits[b >> 5] >> (b & 31)) & 1u) && prob(x[j]) > 0.f) take |= 1u << j;
                        }
                    append(list, kRowList, &sh.list_n, take, [&](int j) { return __float_as_uint(x[j]); });
                });
                hand_over();
                cl.sync();
            }
            tick(tk, 8);
            if (rank == 0) {
                int r = cut_bins(sh, dyn, top_p, prob);
                if (r == 2 && round >= 8) r = 1;
                __syncthreads();
                if (tid < C) {
                    RowSh *o = cl.map_shared_rank(&sh, tid);
                    o->stop = r;
                    o->tstar = sh.tstar;
                    o->hit_keep = sh.hit_keep;
                }
                if (r == 1 && tid == 0) ws.redo[fi] = 1;
            }
            cl.sync();
            if (sh.stop != 2) break;
        }
        tick(tk, 9);
        if (sh.stop) return;
        d.flags |= kDistTopP;
        d.tstar = sh.tstar;
        if (d.tstar > 0.f) {
            float em;
            if (!smallest_e(d.tstar, d.inv1, em)) {  // the same for every thread of the cluster
                if (rank == 0 && tid == 0) ws.redo[fi] = 1;
                return;
            }
            fin.e_min = fmaxf(fin.e_min, em);
        }
        const int keep = sh.hit_keep;
        if (keep > 0) {
            // the keep-th token, in token order, whose probability equals the threshold
            int *tile_cnt = (int *)sh.tile_sum;
            auto matches = [&](int t) {
                float x[8];
                get_e(t, x);
                unsigned m = 0u;
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (prob(x[j]) == d.tstar) m |= 1u << j;
                return m;
            };
            for (int t = t0 + warp; t < t1; t += kRW) {
                const int m = __reduce_add_sync(0xFFFFFFFFu, __popc(matches(t)));
                if (lane == 0) tile_cnt[t - t0] = m;
            }
            __syncthreads();
            if (warp == 0) {
                int v = 0;
                for (int t = lane; t < t1 - t0; t += 32) v += tile_cnt[t];
                v = __reduce_add_sync(0xFFFFFFFFu, v);
                if (lane < C) cl.map_shared_rank(&sh, lane)->cnt[rank] = v;
            }
            cl.sync();
            int first = 0;
            for (int r = 0; r < rank; r++) first += sh.cnt[r];
            if (warp == 0 && keep > first && keep <= first + sh.cnt[rank]) {
                int want = keep - first;  // 1-based among this CTA's matches
                for (int t = t0; t < t1; t++) {
                    const int c = tile_cnt[t - t0];
                    if (want > c) { want -= c; continue; }
                    const unsigned m = matches(t);
                    const int inc = warp_scan_i(__popc(m)), excl = inc - __popc(m);
                    int idx = -1;
                    if (want > excl && want <= inc) {
                        int k = want - excl;
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            if ((m >> j) & 1u) { if (--k == 0) idx = t * kSub + lane * 8 + j; }
                    }
                    idx = __reduce_max_sync(0xFFFFFFFFu, idx);
                    if (lane < C) cl.map_shared_rank(&sh, lane)->tie_idx = idx;
                    break;
                }
            }
            cl.sync();
            d.tie_idx_max = sh.tie_idx;
        }
    }

    // P7: Normalize (Sampler.cs:553-562): the fp64 sum of what is left, and the tile sums of it
    const bool tied = d.tie_idx_max != INT_MAX;
    {
        double part[2] = {0.0, 0.0};
        // two tiles to a turn: little is done with them, and it is their loads that count
        for (int t = t0 + warp; t < t1; t += 2 * kRW) {
            float x[2][8];
            get_e(t, x[0]);
            const bool two = t + kRW < t1;
            if (two) get_e(t + kRW, x[1]);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (u == 1 && !two) break;
                float acc = 0.f;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    float p = fin(x[u][j]);
                    if (tied && p == d.tstar && (t + u * kRW) * kSub + lane * 8 + j > d.tie_idx_max) p = 0.f;
                    part[j & 1] += widen(p);
                    acc += p;
                }
                acc = warp_sum_f(acc);
                if (lane == 0) sh.tile_sum[t - t0 + u * kRW] = acc;
            }
        }
        const double all_part = block_sum_d(part[0] + part[1], sh.red_d);
        tp = tile_prefix(sh.tile_sum, t1 - t0, sh.red_d);
        if (tid < C) {
            RowSh *o = cl.map_shared_rank(&sh, tid);
            o->part[rank] = all_part;
            o->tot[1][rank] = tp.all;
        }
    }
    cl.sync();
    tick(tk, 10);
    double sum3 = 0.0;
    for (int r = 0; r < C; r++) sum3 += sh.part[r];
    const float s3 = (float)sum3;
    if (s3 > 0.f && s3 != 1.0f) { d.flags |= kDistScale3; d.inv3 = __fdiv_rn(1.0f, s3); }
    if (a.mode == 2) {
        if (rank == 0 && tid == 0) { a.dists[row] = d; ws.redo[fi] = 0; }
        return;
    }
    if (dist_mode) write_dist();
    if (a.mode == 1) {
        if (rank == 0 && tid == 0) { if (a.row_flags) a.row_flags[row] = kPathFull | sh.flags; ws.redo[fi] = 0; }
        return;
    }
    base = all = 0.0;
    for (int r = 0; r < C; r++) {
        if (r == rank) base = all;
        all += sh.tot[1][r];
    }
    auto final_p = [&](int t, float (&x)[8]) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float p = fin(x[j]);
            if (tied && p == d.tstar && t * kSub + lane * 8 + j > d.tie_idx_max) p = 0.f;
            x[j] = __fmul_rn(p, d.inv3);
        }
    };
    auto get_p = [&](int t, float (&x)[8]) { get_e(t, x); final_p(t, x); };
    summarise(sh, wa, dst, get_e, final_p, t0, t1, tp, base, all, (double)d.inv3, (double)u01);
    cl.sync();
    tick(tk, 11);
    if (rank != 0 || warp != 0) return;
    const WalkOut o = row_walk(wa, get_p, n, nsub, u01, true);
    tick(tk, 12);
    if (lane == 0) {
        uint32_t fl = kPathFull | sh.flags;
        if (o.hit >= 0 && u01 > 0.f && (u01 - o.before <= kNearTol || o.s - u01 <= kNearTol)) fl |= kFlagNearBoundary;
        write_row(o.hit, fl);
    }
}

// ---- speculative verification: accept chain and draw -------------------------------------------------------
// What k_spec_finish (stg_spec_kernels.cu) does with one CTA per sequence, by a cluster per sequence: the accept
// chain by a warp of every CTA (the draft positions side by side), then the values the draw runs over - the
// target row's final probabilities (bonus draw, looser rule) or the residual max(p - q, 0), recomputed from
// the logits - to the sequence's scratch row, and the walk of stg_walk.cuh; for the residual first to its sum, then
// to u * sum.  As three kernels, one of them a CTA per sequence, a lone sequence took 110 us.  Sequences
// that need a rare fall-back (an empty residual, a walk off the end) are left to k_spec_finish.
template <bool BF16>
__global__ void __launch_bounds__(kRT, 2) k_spec_row(const __grid_constant__ SpecArgs a, const RowWs ws, int32_t *fallback)
{
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ RowSh sh;
    __shared__ int s_acc, s_bad;
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = blockIdx.x / C;
    const int L = a.n_draft, n = a.vocab, nsub = (n + kSub - 1) / kSub;
    const int per = (nsub + C - 1) / C;
    const int t0 = min(rank * per, nsub), t1 = min(t0 + per, nsub);
    WalkArea *wa = (WalkArea *)dyn;
    WalkArea *dst = rank == 0 ? wa : (WalkArea *)cl.map_shared_rank((unsigned char *)wa, 0);
    float *e = ws.e + (size_t)s * ws.e_stride;
    const int esz = BF16 ? 2 : 4;
    const RowDist *td = a.tdist + (int64_t)s * (L + 1);
    const RowDist *dd = a.ddist ? a.ddist + (int64_t)s * L : nullptr;
    const char *trows = (const char *)a.target + (int64_t)s * (L + 1) * n * esz;
    const char *drows = a.draft ? (const char *)a.draft + (int64_t)s * L * n * esz : nullptr;
    const double *u = a.uniforms + (int64_t)s * (L + 2);
    const bool greedy = (td[0].flags & kDistOneHot) != 0;
    if (warp == 0) {
        bool ok = true, bad = false;
        float shown = 0.f;
        if (lane < L) {
            const int i = lane;
            const int tok = a.draft_tokens[(int64_t)s * L + i];
            if ((unsigned)tok >= (unsigned)n) {
                // a draft token outside the vocabulary (the reference's pDist[tokens[i]] throws,
                // SpeculativeDecoder.cs:534): never read, rejected, and reported in the flags
                ok = false;
                bad = true;
            } else if (greedy) {
                ok = (tok == td[i].tie_idx_max);  // SpeculativeDecoder.Step, SpeculativeDecoder.cs:400-405
                shown = ok ? 1.f : 0.f;
            } else {
                const float px = eval_point<BF16>(LogitRow{trows + (int64_t)i * n * esz, a.target_cap}, tok, td[i]);
                if (a.mode == 0) {
                    const float qx = eval_point<BF16>(LogitRow{drows + (int64_t)i * n * esz, a.draft_cap}, tok, dd[i]);
                    const float r = qx > 0.f ? fminf(1.f, __fdiv_rn(px, qx)) : (px > 0.f ? 1.f : 0.f);
                    ok = u[i] < (double)r;
                    shown = r;
                } else {
                    ok = px >= a.p_min || tok == td[i].argmax;
                    shown = px;
                }
            }
        }
        const unsigned rej = __ballot_sync(0xFFFFFFFFu, lane < L && !ok);
        const int acc = rej ? __ffs(rej) - 1 : L;
        const bool bad_draft = acc < L && __shfl_sync(0xFFFFFFFFu, bad ? 1 : 0, min(acc, 31)) != 0;
        if (rank == 0) {
            // positions after the first rejection are not tested
            if (a.accept_probs && lane < L) a.accept_probs[(int64_t)s * L + lane] = lane <= acc ? shown : 0.f;
            if (lane == 0) {
                fallback[s] = 0;
                a.accepted[s] = acc;
                if (greedy) {
                    a.correction[s] = td[acc].tie_idx_max;
                    if (a.seq_flags) a.seq_flags[s] = bad_draft ? (1u << 9) : 0u;
                }
            }
        }
        if (lane == 0) { s_acc = acc; s_bad = bad_draft ? 1 : 0; }
    }
    if (greedy) return;
    cl.barrier_arrive();  // waited for before the first push, as in k_row
    __syncthreads();
    const int acc = s_acc;
    const bool residual = !(acc == L || a.mode == 1);
    {
        const bool al = a.vec == 4;
        const RowDist tdr = td[acc];
        const LogitRow prow{trows + (int64_t)acc * n * esz, a.target_cap};
        const ProvRow<BF16> pp{SrcLogits<BF16>{prow, nullptr, al, tdr.inv_t, tdr.inv_t != 1.0f}, tdr};
        auto tile = [&](int t, const float (&x)[8]) {
            store_e(e, t * kSub + lane * 8, x);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 8; j++) sum += x[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
            if (lane == 0) sh.tile_sum[t - t0] = sum;
        };
        if (residual) {
            const RowDist dq = dd[acc];
            const LogitRow qrow{drows + (int64_t)acc * n * esz, a.draft_cap};
            const ProvRow<BF16> qq{SrcLogits<BF16>{qrow, nullptr, al, dq.inv_t, dq.inv_t != 1.0f}, dq};
            const ProvResidual<BF16> rr{pp, qq};
#pragma unroll 1
            for (int t = t0 + warp; t < t1; t += kRW) {
                float x[8];
                rr.load(t * kSub + lane * 8, n, x);  // zeros beyond the row
                tile(t, x);
            }
        } else {
#pragma unroll 1
            for (int t = t0 + warp; t < t1; t += kRW) {
                float x[8];
                pp.load(t * kSub + lane * 8, n, x);
                tile(t, x);
            }
        }
    }
    cl.barrier_wait();
    const TilePrefix tp = tile_prefix(sh.tile_sum, t1 - t0, sh.red_d);
    if (tid < C) cl.map_shared_rank(&sh, tid)->tot[0][rank] = tp.all;
    cl.sync();
    double base = 0.0, all = 0.0;
    for (int r = 0; r < C; r++) {
        if (r == rank) base = all;
        all += sh.tot[0][r];
    }
    const float u0 = __double2float_rn(u[L]);
    auto get = [&](int t, float x[8]) { load_e(e, t * kSub + lane * 8, x); };
    // the target of a residual is u times its sum: where it should lie is known well enough
    summarise(sh, wa, dst, get, [](int, float (&)[8]) {}, t0, t1, tp, base, all, 1.0, residual ? (double)u0 * all : (double)u0);
    cl.sync();
    pdl_release();
    if (rank != 0 || warp != 0) return;
    float target = u0;
    if (residual) {
        // ResampleResidual (Sampler.cs:587-618): the sum of the residual, then the draw to u * sum
        const float sum = row_walk(wa, get, n, nsub, 0.f, false).s;
        if (!(sum > 0.f)) {  // nothing left of p - q (or NaN): the draw from p with the spare uniform
            if (lane == 0) fallback[s] = 1;
            return;
        }
        target = __fmul_rn(u0, sum);
    }
    const WalkOut o = row_walk(wa, get, n, nsub, target, true);
    if (lane == 0) {
        uint32_t fl = s_bad ? (1u << 9) : 0u;
        int corr = o.hit;
        if (corr < 0) {
            if (residual) { fallback[s] = 1; return; }  // the rounding fall-back of the residual draw
            corr = n - 1;
            fl |= 1u << 5;
        }
        a.correction[s] = corr;
        if (a.seq_flags) a.seq_flags[s] = fl;
    }
}

}  // namespace

// Launches `rows` clusters as large as the rows leave room for, one wave: a lone row is spread over 16 CTAs, several
// hundred rows get one each (two CTAs fit an SM).  A CTA has a tile for every other warp at least (a row of 32,000 by
// eight CTAs: 55.4 -> 51.5 us against four).
template <class... Params, class... Args>
static cudaError_t launch_clusters(void (*fn)(Params...), size_t smem, int rows, int vocab, cudaStream_t stream, const Args &...args)
{
    cudaError_t e = ensure_dynamic_smem((const void *)fn, smem);
    if (e != cudaSuccess) return e;
    const int nsub = (vocab + kSub - 1) / kSub;
    struct Fit { int n[5]; };
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, Fit> fits;
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kRT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    Fit fit;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = fits.find({(const void *)fn, dev});
        if (it == fits.end()) {
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e != cudaSuccess) return e;
            for (int k = 0; k < 5; k++) {
                at.val.clusterDim = {1u << k, 1, 1};
                cfg.gridDim = dim3(1u << k);
                e = cudaOccupancyMaxActiveClusters(&fit.n[k], fn, &cfg);
                if (e != cudaSuccess) { cudaGetLastError(); fit.n[k] = 0; }
            }
            fits[{(const void *)fn, dev}] = fit;
        } else {
            fit = it->second;
        }
    }
    int k = 0;
    for (int j = 4; j > 0; j--)
        if (fit.n[j] >= rows && (1 << j) * kRW <= 2 * nsub) { k = j; break; }
    at.val.clusterDim = {1u << k, 1, 1};
    cfg.gridDim = dim3((unsigned)rows << k);
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

cudaError_t launch_row_clusters(const SampleArgs &a, const RowWs &ws, bool want_argmax, cudaStream_t stream)
{
    const auto fn = a.mask != nullptr && a.mode == 0 ? (a.dtype == 1 ? k_row<true, true> : k_row<false, true>)
                                                     : (a.dtype == 1 ? k_row<true, false> : k_row<false, false>);
    return launch_clusters(fn, kRowSmem, a.n_items, a.vocab, stream, a, ws, want_argmax ? 1 : 0);
}

cudaError_t launch_spec_rows(const SpecArgs &a, const RowWs &ws, int32_t *fallback, cudaStream_t stream)
{
    return launch_clusters(a.dtype == 1 ? k_spec_row<true> : k_spec_row<false>, sizeof(WalkArea), a.n_seq, a.vocab, stream, a, ws, fallback);
}

}  // namespace stg
