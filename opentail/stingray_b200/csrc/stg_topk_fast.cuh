// The finish of a top-k row from its candidate list, without sorting the list.
//
// The row's order is (penalised value, raw logit, lower token first): a candidate is the pair (penalised value, raw logit)
// in one 64-bit word, and its token.  The k best are fenced off by a histogram over the range of the penalised values, refined
// inside the bin that holds the k-th until no more than kFastM candidates lie above its lower edge; those are put in
// order by counting, each by a thread, which also computes its exp; then one warp runs the filters and the draw of
// Sampler.cs:296-349.  Equal values share a bin, so ties at the k-th are all there to be ordered; more of them than that are
// divided by their raw logits and tokens first.
//
// Bound: latency of a dozen dependent steps, six block barriers: 6 us for a lone row of 549 candidates (2.4 of them the loads and
// the history's lookups, 1.4 the ranks and exps, 1.3 the draw), 11 where four CTAs share an SM.  A register sort of every
// warp's share and a tree of merges in its place: 16 there, and 96 rows of bf16 logits took 45.5 us a step, now 34.8.
#pragma once
#include <math_constants.h>

#include "stg_select.cuh"

namespace stg {

constexpr int kFastK = 256;       // largest top_k
constexpr int kFastM = 512;       // candidates put in order at most
constexpr int kFastU = kThreads >= 512 ? 2 : 3;  // candidates a thread takes at a time

struct FastShared {
    float vals[256], probs[256], pre[256];
    int ids[256];
    u64 best[kFastM];
    int tok[kFastM];
    unsigned hist[256];
    unsigned lo[32], hi[32];   // smallest and largest penalised value of each warp
    unsigned base;             // lower edge of the window, then of the k best's bin
    int shift;                 // bins of 2^shift values
    int want;                  // how many of the k best lie in the window
    int above;                 // candidates above the window
    int state;                 // 0: another round, 1: fenced off, 2: too many of one value
    int n, pad[2];
};

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
// (Sampler.cs:296-349; every fp32 operation as in finish_topk_draw).  vals, their exps in probs, and ids [k] are in `fs`, zeros
// in probs behind them up to a multiple of eight.
__device__ __forceinline__ void fast_draw(FastShared &fs, const RowPlan &rp, float uniform, FinishOut *out)
{
    const int lane = threadIdx.x & 31, k = rp.top_k, k8 = (k + 7) & ~7;
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

// Whether the row qualifies: no penalty can raise a logit, so that any superset of the N best raw logits holds
// the k best penalised ones (see finish_topk_select), and the shared memory suffices.
__device__ __forceinline__ int fast_hash_slots(const RowPlan &rp)
{
    int n = 0;
    if (rp.has_penalty)
        for (n = 64; n < 2 * rp.hist_len;) n <<= 1;
    return n;
}
__device__ __forceinline__ bool fast_eligible(const RowPlan &rp, size_t arena_bytes)
{
    return sizeof(FastShared) + (size_t)fast_hash_slots(rp) * 8 <= arena_bytes && rp.top_k <= kFastK &&
           (!rp.has_penalty || (rp.rep >= 1.0f && rp.pres >= 0.f && rp.freq >= 0.f));
}

// One CTA, all threads: what the finish of a row needs besides its candidates, done while those are still being found: the
// hash of its history, token -> occurrences | inside the window << 16, behind the FastShared.
__device__ __forceinline__ void finish_fast_begin(const RowPlan &rp, const int32_t *hist, unsigned char *arena)
{
    const int tid = threadIdx.x;
    if (rp.has_penalty) {
        const int hslots = fast_hash_slots(rp);
        int *hkey = (int *)(arena + sizeof(FastShared));
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

// The penalised values of a warp's candidates (Sampler.cs:263-287), as ordered bits; key 0: none.  Whole warps call it, and the
// warp leaves the lookup's loop together, when the last of its lanes is done: with a loop that each lane left by itself a
// warp's candidates were now and then lost in the register sort that followed then (rows of 262,144 bf16 logits behind
// 700-token histories: once in 400 to 9,000 steps), for a reason that was not found.  A lane's keys are looked up side
// by side.
template <int U>
__device__ __forceinline__ void fast_penalise(const u64 (&key)[U], uint32_t (&pv)[U], const int *hkey, const unsigned *hcnt, int hmask,
                                              const RowPlan &rp, const float *pow_tab)
{
    int h[U], at[U];
    unsigned open = 0u;
#pragma unroll
    for (int q = 0; q < U; q++) {
        pv[q] = (uint32_t)(key[q] >> 32);
        h[q] = (int)(((unsigned)key_idx(key[q]) * 2654435761u) >> 7) & hmask;
        at[q] = -1;
        open |= key[q] != 0ull ? 1u << q : 0u;
    }
#pragma unroll 1
    while (__any_sync(0xFFFFFFFFu, open != 0u)) {
#pragma unroll
        for (int q = 0; q < U; q++) {
            const int kx = hkey[h[q]], id = key_idx(key[q]);
            at[q] = ((open >> q) & 1u) && kx == id ? h[q] : at[q];
            open &= kx == id || kx == -1 ? ~(1u << q) : 0xFFFFFFFFu;
            h[q] = (h[q] + 1) & hmask;
        }
    }
#pragma unroll
    for (int q = 0; q < U; q++) {
        if (!__any_sync(0xFFFFFFFFu, at[q] >= 0)) continue;
        const unsigned c = at[q] >= 0 ? hcnt[at[q]] : 0u;
        float x = key_val(key[q]);
        const int occ_all = (int)(c & 0xFFFFu), occ_w = (int)(c >> 16);
        if (rp.rep != 1.0f && occ_w > 0) {
            const float pw = pow_rep(pow_tab, rp.rep, occ_w);
            x = x > 0.f ? __fdiv_rn(x, pw) : __fmul_rn(x, pw);
        }
        x = __fsub_rn(x, __fadd_rn(rp.pres, __fmul_rn(rp.freq, (float)occ_all)));
        __syncwarp();
        if (c != 0u) pv[q] = ord32(x);
    }
}

// penalised value << 32 | raw logit of a candidate there was no room for: the list holds its penalised value in the raw
// logit's place, which raw(token) reads from the row again
template <class Raw>
__device__ __noinline__ u64 fast_reread(const Raw raw, u64 x) { return (x & ~0xFFFFFFFFull) | ord32(raw(key_idx(x))); }

// One CTA, all threads, behind finish_fast_begin; `list`: cnt keys in device memory, `arena`: shared memory, the FastShared, the
// history's hash, then 12 bytes per candidate.  Of those that do not fit the penalised value goes back to the list, so that
// all are looked up and penalised once.  (Penalised again in every pass: 300 rows behind 1,000 tokens took 193 us, and rows
// of 1,500, whose hash leaves little room, took 1,100 on the general path.)  `ahead`: entries tid + q kThreads of the
// list, loaded before its length was known.  False: nothing was written, the row has to be done from its logits.
template <class Raw>
__device__ __forceinline__ bool finish_fast(const Raw &raw, u64 *list, const u64 (&ahead)[kFastU], int cnt, const RowPlan &rp, const float *pow_tab, float uniform,
                                            unsigned char *arena, size_t arena_bytes, FinishOut *out, int32_t *o_ids, float *o_vals,
                                            float *o_probs)
{
    constexpr int U = kFastU;
    FastShared &fs = *(FastShared *)arena;
    static_assert(sizeof(FastShared) % 16 == 0, "what follows is aligned");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, k = rp.top_k, hslots = fast_hash_slots(rp);
    const int *hkey = (const int *)(arena + sizeof(FastShared));
    const unsigned *hcnt = (const unsigned *)(hkey + hslots);
    const int room = (int)((arena_bytes - sizeof(FastShared) - (size_t)hslots * 8) / 12), held = min(cnt, room);
    u64 *pk = (u64 *)(arena + sizeof(FastShared) + (size_t)hslots * 8);  // penalised value << 32 | raw logit, ordered bits
    int *pt = (int *)(pk + room);
    if (tid < 256) fs.hist[tid] = 0u;
    if (tid < 8) fs.probs[(k + tid) & 255] = 0.f;  // behind the last, where the sums read
    uint32_t lo = 0xFFFFFFFFu, hi = 0u;
#pragma unroll 1
    for (int b = 0; b < cnt; b += U * kThreads) {
        u64 key[U];
        uint32_t pv[U];
#pragma unroll
        for (int q = 0; q < U; q++) {
            const int i = b + q * kThreads + tid;
            key[q] = i >= cnt ? 0ull : b == 0 ? ahead[q] : __ldcg(list + i);
            pv[q] = (uint32_t)(key[q] >> 32);
        }
        if (rp.has_penalty) fast_penalise<U>(key, pv, hkey, hcnt, hslots - 1, rp, pow_tab);
#pragma unroll
        for (int q = 0; q < U; q++) {
            const int i = b + q * kThreads + tid;
            if (i < cnt) {
                lo = min(lo, pv[q]);
                hi = max(hi, pv[q]);
                if (i < room) {
                    pk[i] = (u64)pv[q] << 32 | (key[q] >> 32);
                    pt[i] = key_idx(key[q]);
                } else {
                    __stcg(list + i, (u64)pv[q] << 32 | (uint32_t)key[q]);
                }
            }
        }
    }
    {
        const uint32_t l = __reduce_min_sync(0xFFFFFFFFu, lo), h = __reduce_max_sync(0xFFFFFFFFu, hi);
        if (lane == 0) { fs.lo[warp] = l; fs.hi[warp] = h; }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kThreads / 32; w++) { lo = min(lo, fs.lo[w]); hi = max(hi, fs.hi[w]); }
    }
    // A window of 256 bins from the largest value downwards, value v in bin (top - v) >> shift; then the same inside the bin that
    // holds the k-th, until no more than kFastM candidates lie above its lower edge (to go on until 128 do gives nothing).
    // Where more have one value at the cut, their raw logits are divided in the same way (`by` 1), and where those are
    // equal too, their tokens (`by` 2), of which no two are the same.
    int by = 0, shift = max(24 - __clz((int)(hi - lo)), 0), want = k, above = 0;
    uint32_t top = hi, cut = 0u, cut_raw = 0u;
    // body(x, tok): x = penalised value << 32 | raw logit, of which the latter may be missing where it does not matter
    auto for_all = [&](auto body) {
#pragma unroll 1
        for (int i = tid; i < held; i += kThreads) body(pk[i], pt[i], true);
#pragma unroll 1
        for (int i = held + tid; i < cnt; i += kThreads) {
            const u64 x = __ldcg(list + i);
            body(by == 0 ? x : fast_reread(raw, x), key_idx(x), by != 0);
        }
    };
    // the value in question of a candidate at the cut
    auto value = [&](u64 x, int tok) { return by == 0 ? (uint32_t)(x >> 32) : by == 1 ? (uint32_t)x : ~(uint32_t)tok; };
    auto at_cut = [&](u64 x) { return by == 0 || ((uint32_t)(x >> 32) == cut && (by == 1 || (uint32_t)x == cut_raw)); };
#pragma unroll 1
    for (;;) {
        for_all([&](u64 x, int tok, bool) {
            const uint32_t v = value(x, tok), d = (top - v) >> shift;
            if (at_cut(x) && v <= top && d < 256u) atomicAdd(&fs.hist[d], 1u);
        });
        __syncthreads();
        if (warp == 0) {
            if (lane == 0) { fs.state = 3; fs.n = 0; }
            __syncwarp();
            unsigned h[8], sum = 0u;
#pragma unroll
            for (int j = 0; j < 8; j++) { h[j] = fs.hist[lane * 8 + j]; fs.hist[lane * 8 + j] = 0u; sum += h[j]; }
            unsigned run = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xFFFFFFFFu, run, o);
                if (lane >= o) run += t;
            }
            run -= sum;
            if ((int)run < want && want <= (int)(run + sum)) {  // one lane
                bool found = false;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (!found && want <= (int)(run + h[j])) {
                        found = true;
                        const int bin = lane * 8 + j, all = above + (int)(run + h[j]);
                        const int state = all <= kFastM ? 1 : shift == 0 ? 2 : 0;
                        // the bin's lower edge where the k best are fenced off, else its upper one: it is the next window
                        fs.base = state == 1 ? top - min(top, (uint32_t)((((u64)bin + 1) << shift) - 1)) : top - ((uint32_t)bin << shift);
                        fs.want = want - (int)run;
                        fs.above = above + (int)run;
                        fs.state = state;
                    }
                    run += found ? 0u : h[j];
                }
            }
        }
        __syncthreads();
        const int state = fs.state;
        top = fs.base;
        if (state == 1) break;
        if (state == 3) return false;  // not met: the k-th lies in every window
        want = fs.want;
        above = fs.above;
        shift = max(shift - 8, 0);  // 256 bins inside that one
        if (state == 2) {
            if (by == 0) cut = top;
            else cut_raw = top;
            by++;
            top = 0xFFFFFFFFu;
            shift = 24;
        }
    }
    const u64 fence = by == 0 ? (u64)top << 32 : (u64)cut << 32 | (by == 1 ? top : cut_raw);
    for_all([&](u64 x, int tok, bool whole) {
        if (x >= fence && (by < 2 || x > fence || ~(uint32_t)tok >= top)) {
            const int slot = atomicAdd(&fs.n, 1);
            if (slot < kFastM) {
                fs.best[slot] = whole ? x : fast_reread(raw, (x & ~0xFFFFFFFFull) | (uint32_t)~tok);
                fs.tok[slot] = tok;
            }
        }
    });
    __syncthreads();
    const int m = min(fs.n, kFastM);
    const float inv_t = rp.temperature == 1.0f ? 1.0f : __fdiv_rn(1.0f, rp.temperature);
    const float mx = __fmul_rn(unord32(hi), inv_t);
    for (int i = tid; i < m; i += kThreads) {
        const u64 x = fs.best[i];
        const int tok = fs.tok[i];
        int rank = 0;
#pragma unroll 8
        for (int j = 0; j < m; j++) {  // no branches: bf16 logits tie in droves
            const u64 y = fs.best[j];
            rank += (int)(y > x) | ((int)(y == x) & (int)(fs.tok[j] < tok));
        }
        if (rank < k) {
            const float v = unord32((uint32_t)(x >> 32));
            fs.vals[rank] = v;
            fs.ids[rank] = tok;
            fs.probs[rank] = isinf(v) && v < 0.f ? 0.f : (float)exp((double)__fsub_rn(__fmul_rn(v, inv_t), mx));
        }
    }
    __syncthreads();
    if (warp == 0) fast_draw(fs, rp, uniform, out);
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < k; t += kThreads) {
        if (o_ids) o_ids[t] = fs.ids[t];
        if (o_vals) o_vals[t] = fs.vals[t];
        if (o_probs) o_probs[t] = fs.probs[t];
    }
    return true;
}

}  // namespace stg
