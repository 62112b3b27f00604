// The finish of a top-k row from its candidate list, without sorting or radix-selecting the list.
//
// Every warp sorts its share of the list in registers (bitonic, keys exchanged by shuffles) and keeps its best
// K2 = 32 * KPL keys; a tree of merges over the warps leaves the row's best K2 in the first warp, which
// also runs the softmax, the filters and the draw of Sampler.cs:296-349.  The radix selection it stands in
// for crosses two block barriers per digit and ranks ties against the whole list: on 96 rows of bf16 logits
// (which tie in droves) with 256-token histories the finish took 70 us and takes 27, a lone row's step of
// 151,936 logits went from 25 to 19 us.  Bound: latency of a few dozen dependent shuffles.
//
// The row's order is (penalised value descending, raw order among equals).  Keys hold the penalised value, a
// bit that says a penalty lowered it - its raw logit was higher than those of its equals that none did, so it
// comes first - and the token.  Lowered logits that come out equal from different raw values (common with bf16:
// 11 / 1.1^2 = 10 / 1.1) are put into raw order at the end; left to the general path they made a step of 96
// rows of 151,936 with histories of their own sampled tokens take 102 us instead of 47.
#pragma once
#include <math_constants.h>

#include "stg_select.cuh"

namespace stg {

constexpr int kFastK = 255;       // largest top_k: one more key than k has to be seen

struct FastShared {
    float vals[256], probs[256], pre[256];
    int ids[256];
    int fail, pad[3];
};

__device__ __forceinline__ int fast_idx(u64 k) { return (int)(0x7FFFFFFFu - ((uint32_t)k & 0x7FFFFFFFu)); }

// steps j0 .. 1 of stage k of a bitonic sort (descending) of 32 * KPL keys; key i is r[i / 32] of lane i % 32.
// Unrolled: in loops the same steps made a lone row's step 21.5 us instead of 18.8.
template <int KPL>
__device__ __forceinline__ void warp_steps(u64 (&r)[KPL], int k, int j0)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 16 * KPL; j > 0; j >>= 1) {
        if (j > j0) continue;
        if (j >= 32) {
            const int dj = j / 32;
#pragma unroll
            for (int q = 0; q < KPL; q++) {
                if ((q & dj) == 0) {
                    const bool desc = ((q * 32 + lane) & k) == 0;
                    const u64 x = r[q], y = r[q | dj];
                    if ((x < y) == desc) { r[q] = y; r[q | dj] = x; }
                }
            }
        } else {
            const bool lower = (lane & j) == 0;
#pragma unroll
            for (int q = 0; q < KPL; q++) {
                const bool desc = ((q * 32 + lane) & k) == 0;
                const u64 o = __shfl_xor_sync(0xFFFFFFFFu, r[q], j);
                r[q] = (lower == desc) ? (r[q] > o ? r[q] : o) : (r[q] < o ? r[q] : o);
            }
        }
    }
}
template <int KPL>
__device__ __forceinline__ void warp_sort(u64 (&r)[KPL])
{
#pragma unroll
    for (int k = 2; k <= 32 * KPL; k <<= 1) warp_steps<KPL>(r, k == 32 * KPL ? 1 << 30 : k, k >> 1);
}
// r = the best keys of r and of another descending list given reversed: rev[q] holds key 32 * KPL - 1 - (32 q + lane)
template <int KPL>
__device__ __forceinline__ void warp_best(u64 (&r)[KPL], const u64 (&rev)[KPL])
{
#pragma unroll
    for (int q = 0; q < KPL; q++) r[q] = r[q] > rev[q] ? r[q] : rev[q];
    warp_steps<KPL>(r, 1 << 30, 16 * KPL);
}

// o[i] = fl(o[i - 1] + x[i]) from 0 for i < m (a multiple of 8); one warp, returns the last
__device__ __forceinline__ float warp_prefix_serial(const float *x, float *o, int m)
{
    const int lane = threadIdx.x & 31;
    float acc = 0.f;
    float4 a = *(const float4 *)x, b = *(const float4 *)(x + 4);
#pragma unroll 1
    for (int i = 0; i < m; i += 8) {
        const float4 p = a, q = b;
        const int nx = i + 8 < m ? i + 8 : 0;
        a = *(const float4 *)(x + nx);
        b = *(const float4 *)(x + nx + 4);
        float4 u, v;
        u.x = acc = __fadd_rn(acc, p.x); u.y = acc = __fadd_rn(acc, p.y); u.z = acc = __fadd_rn(acc, p.z); u.w = acc = __fadd_rn(acc, p.w);
        v.x = acc = __fadd_rn(acc, q.x); v.y = acc = __fadd_rn(acc, q.y); v.z = acc = __fadd_rn(acc, q.z); v.w = acc = __fadd_rn(acc, q.w);
        if (lane == 0) { *(float4 *)(o + i) = u; *(float4 *)(o + i + 4) = v; }
    }
    __syncwarp();
    return acc;
}

// What is left of the row for one warp: softmax over the k ordered candidates, min-p, top-p, the draw
// (Sampler.cs:296-349; every fp32 operation as in finish_topk_draw).  vals / ids [k] are in `fs`.
__device__ __forceinline__ void fast_draw(FastShared &fs, const RowPlan &rp, float uniform, FinishOut *out)
{
    const int lane = threadIdx.x & 31, k = rp.top_k, k8 = (k + 7) & ~7;
    const float inv_t = rp.temperature == 1.0f ? 1.0f : __fdiv_rn(1.0f, rp.temperature);
    const float mx = __fmul_rn(fs.vals[0], inv_t);
#pragma unroll 1
    for (int t = lane; t < k8; t += 32) {
        float e = 0.f;
        if (t < k) {
            const float v = fs.vals[t];
            if (!(isinf(v) && v < 0.f)) e = (float)exp((double)__fsub_rn(__fmul_rn(v, inv_t), mx));
        }
        fs.probs[t] = e;
    }
    __syncwarp();
    const float sum = warp_prefix_serial(fs.probs, fs.pre, k8);
    const float inv_sum = sum > 0.f ? __fdiv_rn(1.0f, sum) : 0.f;
#pragma unroll 1
    for (int t = lane; t < k8; t += 32) fs.probs[t] = __fmul_rn(fs.probs[t], inv_sum);
    __syncwarp();
    warp_prefix_serial(fs.probs, fs.pre, k8);
    // the first index at which a condition holds, `none` when it never does
    auto first = [&](int m, int none, auto cond) {
#pragma unroll 1
        for (int b = 0; b < m; b += 32) {
            const unsigned hit = __ballot_sync(0xFFFFFFFFu, b + lane < m && cond(b + lane));
            if (hit) return b + __ffs(hit) - 1;
        }
        return none;
    };
    int count = k;
    if (rp.min_p > 0.f) {
        const float thr = __fmul_rn(rp.min_p, fs.probs[0]);
        count = first(k, k, [&](int t) { return fs.probs[t] < thr; });
    }
    if (rp.top_p < 1.0f && rp.top_p > 0.f) count = first(count, count - 1, [&](int t) { return fs.pre[t] >= rp.top_p; }) + 1;
    const float kept = count > 0 ? fs.pre[count - 1] : 0.f;
    const float r = __fmul_rn(uniform, kept);
    const int t = first(count, -1, [&](int i) { return r <= fs.pre[i] && fs.ids[i] >= 0; });
    if (lane == 0) {
        uint32_t fl = kPathTopK;
        float pr = fs.probs[0];
        int tok = fs.ids[0];
        if (t >= 0) {
            const float cacc = fs.pre[t], prev = t > 0 ? fs.pre[t - 1] : 0.f;
            tok = fs.ids[t];
            pr = fs.probs[t];
            if (r - prev <= kNearTol * kept || cacc - r <= kNearTol * kept) fl |= kFlagNearBoundary;
        } else {
            fl |= 1u << 5;
        }
        out->token = tok;
        out->prob = kept > 0.f ? pr / kept : 0.f;
        out->flags = fl;
    }
}

// Whether the list qualifies: no penalty can raise a logit, so that any superset of the N best raw logits holds
// the k best penalised ones (see finish_topk_select), and the shared memory suffices.
__device__ __forceinline__ bool fast_eligible(const RowPlan &rp, size_t arena_bytes)
{
    int hslots = 0;
    if (rp.has_penalty)
        for (hslots = 64; hslots < 2 * rp.hist_len;) hslots <<= 1;
    return sizeof(FastShared) + (kThreads / 64) * 256 * 8 + (size_t)hslots * 8 <= arena_bytes && rp.top_k <= kFastK &&
           (!rp.has_penalty || (rp.rep >= 1.0f && rp.pres >= 0.f && rp.freq >= 0.f));
}

// Occurrences of `id` in the history | inside the window << 16.  Whole warps call it, and the warp leaves the loop
// together, when the last of its lanes is done: with a loop that each lane left by itself the lane that had found its
// token stayed apart from the others through the shuffles of the sort behind it, and its warp's candidates were lost
// (rows of 262,144 bf16 logits behind 700-token histories: once in 400 to 9,000 steps, a `__syncwarp` notwithstanding).
__device__ __forceinline__ unsigned fast_occurrences(const int *hkey, const unsigned *hcnt, int hmask, int id)
{
    int h = (int)(((unsigned)id * 2654435761u) >> 7) & hmask;
    int at = -1;
    bool open = true;
#pragma unroll 1
    while (__any_sync(0xFFFFFFFFu, open)) {
        const int kx = hkey[h];
        at = open && kx == id ? h : at;
        open = open && kx != id && kx != -1;
        h = (h + 1) & hmask;
    }
    return at >= 0 ? hcnt[at] : 0u;
}
// the keys of a warp's candidates (0: none) with the penalties applied (Sampler.cs:263-287)
__device__ __forceinline__ u64 fast_penalise(u64 key, const int *hkey, const unsigned *hcnt, int hmask, const RowPlan &rp, const float *pow_tab)
{
    key &= 0xFFFFFFFF7FFFFFFFull;
    unsigned c = fast_occurrences(hkey, hcnt, hmask, fast_idx(key));
    if (key == 0ull) c = 0u;  // reads as token 2^31 - 1
    if (!__any_sync(0xFFFFFFFFu, c != 0u)) return key;
    float x = key_val(key);
    const int occ_all = (int)(c & 0xFFFFu), occ_w = (int)(c >> 16);
    if (rp.rep != 1.0f && occ_w > 0) {
        const float pw = pow_rep(pow_tab, rp.rep, occ_w);
        x = x > 0.f ? __fdiv_rn(x, pw) : __fmul_rn(x, pw);
    }
    x = __fsub_rn(x, __fadd_rn(rp.pres, __fmul_rn(rp.freq, (float)occ_all)));
    __syncwarp();
    const uint32_t was = (uint32_t)(key >> 32), now = ord32(x);
    return c != 0u ? ((u64)now << 32) | (key & 0x7FFFFFFFull) | (now != was ? 0x80000000ull : 0ull) : key;
}

// The sorted keys of one warp, with every run of equal lowered values put into the order of the raw logits.  Keys behind
// the last one were dropped, so a run that reaches it may lack members; that, or a run beyond 32, is answered
// with true: the general path.  `buf`: the 32 * KPL keys, in shared memory.
template <int KPL, class Raw>
__device__ __noinline__ bool order_by_raw(const Raw raw, u64 *buf, int k)
{
    constexpr int K2 = 32 * KPL;
    const int lane = threadIdx.x & 31;
    bool fail = false;
    u64 r[KPL];
    int to[KPL];
#pragma unroll
    for (int q = 0; q < KPL; q++) {
        const int i = q * 32 + lane;
        const u64 key = buf[i];
        r[q] = key;
        int at = i;
        if ((key >> 31) & 1ull) {
            int lo = i, hi = i;
            while (lo > 0 && i - lo < 32 && (buf[lo - 1] >> 31) == (key >> 31)) lo--;
            while (hi + 1 < K2 && hi - i < 32 && (buf[hi + 1] >> 31) == (key >> 31)) hi++;
            if (lo < k && (hi == K2 - 1 || hi - lo >= 32)) {
                fail = true;
            } else if (lo < k && lo < hi) {
                const uint32_t mine = ord32(__fadd_rn(raw(fast_idx(key)), 0.f));
                at = lo;
                for (int j = lo; j <= hi; j++) {
                    if (j == i) continue;
                    const uint32_t other = ord32(__fadd_rn(raw(fast_idx(buf[j])), 0.f));
                    at += other > mine || (other == mine && j < i) ? 1 : 0;
                }
            }
        }
        to[q] = at;
    }
    __syncwarp();
    if (__any_sync(0xFFFFFFFFu, fail)) return true;
#pragma unroll
    for (int q = 0; q < KPL; q++) buf[to[q]] = r[q];
    __syncwarp();
    return false;
}

// Where a row's hash of its history lies in the arena, and its slots
__device__ __forceinline__ int *fast_hash_at(const RowPlan &rp, unsigned char *arena)
{
    return (int *)(arena + sizeof(FastShared) + (kThreads / 64) * 32 * (rp.top_k < 64 ? 2 : rp.top_k < 128 ? 4 : 8) * 8);
}
__device__ __forceinline__ int fast_hash_slots(const RowPlan &rp)
{
    int n = 64;
    while (n < 2 * rp.hist_len) n <<= 1;
    return n;
}
// One CTA, all threads: what the finish of a row needs besides its candidates, done while those are still being found.
// Ends in a block barrier.
__device__ __forceinline__ void finish_fast_begin(const RowPlan &rp, const int32_t *hist, unsigned char *arena)
{
    const int tid = threadIdx.x;
    if (tid == 0) ((FastShared *)arena)->fail = 0;
    if (rp.has_penalty) {
        int *hkey = fast_hash_at(rp, arena);
        const int hslots = fast_hash_slots(rp);
        unsigned *hcnt = (unsigned *)(hkey + hslots);
#pragma unroll 1
        for (int t = tid; t < hslots; t += kThreads) { hkey[t] = -1; hcnt[t] = 0u; }
        __syncthreads();
#pragma unroll 1
        for (int t = tid; t < rp.hist_len; t += kThreads) {
            const int id = __ldg(hist + t);
            if (id < 0) continue;  // never a candidate, and -1 marks an empty slot
            int h = (int)(((unsigned)id * 2654435761u) >> 7) & (hslots - 1);
#pragma unroll 1
            for (;;) {
                const int old = atomicCAS(&hkey[h], -1, id);
                if (old == -1 || old == id) break;
                h = (h + 1) & (hslots - 1);
            }
            atomicAdd(&hcnt[h], 1u + (t >= rp.window_start ? 65536u : 0u));
        }
    }
    __syncthreads();
}

// One CTA, all threads, behind finish_fast_begin; `list`: cnt keys in device memory, `arena`: shared memory, (kThreads / 64) *
// 32 * KPL * 8 bytes for the merges and, behind them, 8 bytes per slot of the history's hash.  False: nothing was written,
// the general path has to do the row.  raw(id): the row's logit at token id.
template <int KPL, class Raw>
__device__ __forceinline__ bool finish_fast_k(const Raw &raw, const u64 *list, int cnt, const RowPlan &rp, const float *pow_tab,
                                              float uniform, unsigned char *arena, FastShared &fs, FinishOut *out)
{
    constexpr int K2 = 32 * KPL, W = kThreads / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    u64 *merge = (u64 *)arena;
    const int *hkey = (const int *)(arena + (W / 2) * K2 * 8);
    const int hslots = fast_hash_slots(rp);
    const unsigned *hcnt = (const unsigned *)(hkey + hslots);
    const bool pen = rp.has_penalty != 0;
    u64 r[KPL], nx[KPL];
#pragma unroll
    for (int q = 0; q < KPL; q++) {
        const int i = warp * K2 + q * 32 + lane;
        r[q] = i < cnt ? __ldcg(list + i) : 0ull;
    }
    const int lists = (cnt + K2 - 1) / K2;
    if (pen) {
#pragma unroll
        for (int q = 0; q < KPL; q++) r[q] = fast_penalise(r[q], hkey, hcnt, hslots - 1, rp, pow_tab);
    }
    warp_sort<KPL>(r);
#pragma unroll 1
    for (int l = warp + W; l < lists; l += W) {
#pragma unroll
        for (int q = 0; q < KPL; q++) {
            const int i = l * K2 + q * 32 + lane;
            nx[q] = i < cnt ? __ldcg(list + i) : 0ull;
        }
        if (pen) {
#pragma unroll
            for (int q = 0; q < KPL; q++) nx[q] = fast_penalise(nx[q], hkey, hcnt, hslots - 1, rp, pow_tab);
        }
        warp_sort<KPL>(nx);
        u64 rev[KPL];
#pragma unroll
        for (int q = 0; q < KPL; q++) rev[q] = __shfl_xor_sync(0xFFFFFFFFu, nx[KPL - 1 - q], 31);
        warp_best<KPL>(r, rev);
    }
#pragma unroll 1
    for (int w = W / 2; w > 0; w >>= 1) {
        if (w < lists) {  // the warps from `lists` on hold nothing
            if (warp >= w && warp < 2 * w) {
#pragma unroll
                for (int q = 0; q < KPL; q++) merge[(size_t)(warp - w) * K2 + q * 32 + lane] = r[q];
            }
            __syncthreads();
            if (warp < w) {
                u64 rev[KPL];
#pragma unroll
                for (int q = 0; q < KPL; q++) rev[q] = merge[(size_t)warp * K2 + K2 - 1 - (q * 32 + lane)];
                warp_best<KPL>(r, rev);
            }
            __syncthreads();
        }
    }
    if (warp == 0) {
        const int k = rp.top_k;
        bool fail = false;
        if (pen) {
            bool tie = false;
#pragma unroll
            for (int q = 0; q < KPL; q++) {
                // the key behind this one
                u64 next = __shfl_down_sync(0xFFFFFFFFu, r[q], 1);
                const u64 head = q + 1 < KPL ? __shfl_sync(0xFFFFFFFFu, r[q + 1 < KPL ? q + 1 : q], 0) : 0ull;
                if (lane == 31) next = head;
                tie |= q * 32 + lane < k && next != 0ull && (r[q] >> 31) == (next >> 31) && ((r[q] >> 31) & 1ull);
            }
            if (__any_sync(0xFFFFFFFFu, tie)) {
#pragma unroll
                for (int q = 0; q < KPL; q++) merge[q * 32 + lane] = r[q];
                __syncwarp();
                fail = order_by_raw<KPL>(raw, merge, k);
#pragma unroll
                for (int q = 0; q < KPL; q++) r[q] = merge[q * 32 + lane];
            }
        }
#pragma unroll
        for (int q = 0; q < KPL; q++) {
            const int i = q * 32 + lane;
            if (i < k) {
                fs.vals[i] = r[q] ? key_val(r[q]) : -CUDART_INF_F;
                fs.ids[i] = r[q] ? fast_idx(r[q]) : -1;
            }
        }
        fail = __any_sync(0xFFFFFFFFu, fail);
        __syncwarp();
        if (!fail) fast_draw(fs, rp, uniform, out);
        else if (lane == 0) fs.fail = 1;
    }
    __syncthreads();
    return fs.fail == 0;
}

template <class Raw>
__device__ __forceinline__ bool finish_fast(const Raw &raw, const u64 *list, int cnt, const RowPlan &rp,
                                            const float *pow_tab, float uniform, unsigned char *arena, FinishOut *out, int32_t *o_ids,
                                            float *o_vals, float *o_probs)
{
    FastShared &fs = *(FastShared *)arena;
    arena += sizeof(FastShared);
    static_assert(sizeof(FastShared) % 16 == 0, "what follows is aligned");
    bool ok;
    if (rp.top_k < 64) ok = finish_fast_k<2>(raw, list, cnt, rp, pow_tab, uniform, arena, fs, out);
    else if (rp.top_k < 128) ok = finish_fast_k<4>(raw, list, cnt, rp, pow_tab, uniform, arena, fs, out);
    else ok = finish_fast_k<8>(raw, list, cnt, rp, pow_tab, uniform, arena, fs, out);
    if (!ok) return false;
#pragma unroll 1
    for (int t = threadIdx.x; t < rp.top_k; t += kThreads) {
        if (o_ids) o_ids[t] = fs.ids[t];
        if (o_vals) o_vals[t] = fs.vals[t];
        if (o_probs) o_probs[t] = fs.probs[t];
    }
    return true;
}

}  // namespace stg
