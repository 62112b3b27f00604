// Speculative verification in the flat form (see stg_flat.cuh): every pass over V as small CTAs over pieces of
// all sequences at once, every serial part as one CTA per sequence over summaries.  The arithmetic is that
// of stg_rowdist.cuh, whose device functions are reused.
#include <cuda_runtime.h>
#include <limits.h>
#include <math_constants.h>
#include <stdint.h>

#include "stg_flat.cuh"
#include "stg_spec_prov.cuh"
#include "stg_launch.h"
#include "stg_rowdist.cuh"

namespace stg {

constexpr int kFullThreads = 256;              // threads of a per-piece kernel: 8 warps, one sub-tile each at a time
constexpr int kPhasePiece = 8192;                  // elements of a row one CTA of a per-piece phase kernel covers
constexpr int kPieceSubTiles = kPhasePiece / kSub;  // 32 sub-tiles of 256 elements: 4 per warp, two in flight at a time
static_assert(kSub * kMaxSubTiles / kPhasePiece <= kFullMaxParts, "FullRow::part has one entry per phase piece");

// ---- look-back over the pieces of a row; guesses and composites of a piece --------------------------------
// A per-piece phase kernel needs, for every sub-tile, the binade the sequential running sum is in
// when it gets there - a guess from the fp64 prefix of the sub-tile sums (stg_emul2.cuh, phase B).
// Inside a piece that is a warp scan; across pieces every CTA publishes the total of its piece
// (FullRow::ptotal, then the flag, release order) and collects the totals of the pieces before it.
// Those belong to CTAs with a lower linear block index, which the hardware has dispatched before this
// one, so they are running or done and none of them waits for a later piece.  The wait is bounded all
// the same: when it runs out the row is flagged `redo` (the self-contained row kernel takes it) and
// the CTA leaves.
constexpr int kLookbackSpins = 100000;  // x 40 ns: a few milliseconds at most

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Warp 0 of the CTA of piece `p` (k: 0 exp values, 1 final probabilities), given the sums of the
// piece's sub-tiles in shared memory (s_sum[0..nloc)): publishes the piece total, looks back, and
// leaves the guessed binade and the crossing slot of every sub-tile of the piece in shared memory
// and in the row's Emul2Work.  Returns false (to every lane) when the look-back timed out.
__device__ __forceinline__ bool piece_guesses(FullRow *fr, Emul2Work *ew, int k, int p, int t0, int nloc, int nsub,
                                              const float *s_sum, unsigned char *s_guess, unsigned char *s_xslot)
{
    const int lane = threadIdx.x & 31;
    const double mine = lane < nloc ? (double)s_sum[lane] : 0.0;
    double tot = mine;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xFFFFFFFFu, tot, o);
    if (lane == 0) {
        __stcg(&fr->ptotal[k][p], tot);
        __threadfence();
        atomicExch(&fr->pflag[k][p], 1u);
    }
    bool ok = true;
    double before = 0.0;
    if (lane < p) {
        int it = 0;
        while (ld_acquire_u32(&fr->pflag[k][lane]) == 0u) {
            if (++it > kLookbackSpins) { ok = false; break; }
            __nanosleep(40);
        }
        if (ok) before = __ldcg(&fr->ptotal[k][lane]);
    }
    ok = __all_sync(0xFFFFFFFFu, ok);
    // sum of the earlier pieces' totals in piece order (lane 0 adds them: a guess needs no more, but
    // every CTA of the row must see the same prefix at a piece boundary whoever computes it)
    double base = 0.0;
    for (int q = 0; q < p; q++) base += __shfl_sync(0xFFFFFFFFu, before, q);
    double inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    const int g = exp_of_double(base + (inc - mine));
    const int gnext = exp_of_double(base + inc);  // the guess at the sub-tile behind this one
    int xs = 0;
    if (ok && lane < nloc && t0 + lane + 1 < nsub && gnext == g + 1 && s_sum[lane] > 0.f) {
        // the sum should pass into the next binade inside this sub-tile: it gets a CrossSlot
        const int slot = atomicAdd(&fr->n_cross[k], 1);
        if (slot < kMaxCross) xs = slot + 1;
    }
    if (lane < nloc) {
        s_guess[lane] = (unsigned char)g;
        s_xslot[lane] = (unsigned char)xs;
        ew->guess[t0 + lane] = (unsigned char)g;
        ew->xslot[t0 + lane] = (unsigned char)xs;
    }
    if (!ok && lane == 0) fr->redo = 1;
    return ok;
}

// Composite increment of every sub-tile of the piece under its guess (phase C), CrossSlots included.
// FINAL: over the final probabilities, else over the exp values.  All threads of the CTA.
// The values come in registers: xs[i] holds the warp's i-th sub-tile of the piece (sub-tile warp + 8 i,
// this lane's 8 elements, zeros beyond the row's end) as the first stage of the kernel left them.
constexpr int kWarpSubTiles = kPieceSubTiles / (kFullThreads / 32);  // 4
__device__ __forceinline__ void piece_composites(Emul2Work *ew, const float (&xs)[kWarpSubTiles][8], int begin, int n,
                                                 const float *s_sum, const unsigned char *s_guess, const unsigned char *s_xslot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W = kFullThreads / 32;
#pragma unroll
    for (int i = 0; i < kWarpSubTiles; i++) {
        const int st = warp + i * W;
        const int t = (begin >> 8) + st;
        if (t * kSub >= n) continue;
        int a0 = 0, a1 = 0;
        if (!(s_sum[st] == 0.f)) {  // else nothing to add: composite 0
            const int g = s_guess[st];
            subtile_composite<false>(xs[i], g, a0, a1);
            const int xsl = s_xslot[st];
            if (xsl) {
                CrossSlot &cs = ew->xs[xsl - 1];
                int l0, l1, h0, h1;
                lane_composite(xs[i], g, l0, l1);
                lane_composite(xs[i], g + 1, h0, h1);
                cs.lo[lane][0] = l0; cs.lo[lane][1] = l1;
                cs.hi[lane][0] = h0; cs.hi[lane][1] = h1;
            }
        }
        if (lane == 0) { ew->comp[t][0] = a0; ew->comp[t][1] = a1; }
    }
}

// the tail both per-piece kernels share: look-back and guesses by warp 0, composites by everyone
template <bool FINAL>
__device__ __forceinline__ void piece_tail(FullRow *fr, Emul2Work *ew, const float (&xs)[kWarpSubTiles][8], int begin, int n,
                                           float *s_sum, unsigned char *s_guess, unsigned char *s_xslot, int *s_ok)
{
    const int t0 = begin >> 8, nsub = (n + kSub - 1) / kSub;
    const int nloc = min(kPieceSubTiles, nsub - t0);
    __syncthreads();  // s_sum is complete
    if (threadIdx.x < 32) {
        const bool ok = piece_guesses(fr, ew, FINAL ? 1 : 0, begin / kPhasePiece, t0, nloc, nsub, s_sum, s_guess, s_xslot);
        if (threadIdx.x == 0) *s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    if (!*s_ok) return;
    piece_composites(ew, xs, begin, n, s_sum, s_guess, s_xslot);
}

// copies a row's sub-tile summaries from device memory into the shared-memory work area of the walk
__device__ __forceinline__ void load_work(Emul2Work *dst, const Emul2Work *src)
{
    const uint4 *s = (const uint4 *)src;
    uint4 *d = (uint4 *)dst;
    for (int i = threadIdx.x; i < (int)(sizeof(Emul2Work) / 16); i += kThreads) d[i] = __ldcg(s + i);
    __syncthreads();
}
static_assert(sizeof(Emul2Work) % 16 == 0, "Emul2Work is copied in 16-byte words");

// exp values of a row as the walk replays them (ProvExp's reload without its load side)
struct ProvE {
    const float *scratch;
    __device__ __forceinline__ void load(int base, int n, float x[8]) const { reload(base, n, x); }
    __device__ __forceinline__ void reload(int base, int n, float x[8]) const
    {
        if (base >= n) {
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = 0.f;
            return;
        }
        SrcScratch s{scratch, 1.f, false};
        s.get8(base, n, x);
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (base + j >= n) x[j] = 0.f;
    }
};

// ---- a shared-memory cache of the sub-tiles a walk will replay ------------------------------------------
// The walk (emul2_walk) consumes most sub-tiles by their composites and touches elements only where
// the running sum changes binade, where a guess was off by one sub-tile, or where the target is met.
// Those places are known in advance from the fp64 prefix of the sub-tile sums: the sub-tiles with a
// crossing slot and their neighbours, the first sub-tiles (the sum climbs through many binades
// there), and the sub-tile in which the prefix reaches the target.  All warps copy them into shared
// memory before the one walking warp starts, so that its replays do not wait on L2.
constexpr int kXcEntries = 64;
struct XCache {
    int of[kMaxSubTiles];      // 0: not cached, else 1 + entry
    int tile[kXcEntries];
    int n;
    int hit_tile;
    double wsum[32];
};

template <class P>
struct ProvCached {
    P base;
    const float *xc;
    const int *of;
    __device__ __forceinline__ void load(int b, int n, float x[8]) const { reload(b, n, x); }
    __device__ __forceinline__ void reload(int b, int n, float x[8]) const
    {
        const int idx = of[b >> 8];
        if (idx > 0) {
            const float4 *q = (const float4 *)(xc + (size_t)(idx - 1) * kSub + (b & (kSub - 1)));
            const float4 q0 = q[0], q1 = q[1];
            x[0] = q0.x; x[1] = q0.y; x[2] = q0.z; x[3] = q0.w; x[4] = q1.x; x[5] = q1.y; x[6] = q1.z; x[7] = q1.w;
        } else {
            base.reload(b, n, x);
        }
    }
};

// Fills the cache for the sequence behind `pv` (n elements, nsub sub-tiles, summaries in wk).  With
// has_target the sub-tile in which the fp64 prefix of the sums reaches `target` is cached too.
// All kThreads threads call it.
template <class P>
__device__ void build_xcache(XCache *xc, float *xdata, const Emul2Work *wk, const P &pv, int n, int nsub, float target,
                             bool has_target)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int t = tid; t < kMaxSubTiles; t += kThreads) xc->of[t] = 0;
    if (tid == 0) { xc->n = 0; xc->hit_tile = INT_MAX; }
    __syncthreads();
    if (has_target) {
        double v = tid < nsub ? (double)wk->sums[tid] : 0.0, inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) xc->wsum[warp] = inc;
        __syncthreads();
        double before = 0.0;
        for (int w = 0; w < warp; w++) before += xc->wsum[w];
        if (tid < nsub && before + inc >= (double)target * (1.0 - 1e-5)) atomicMin(&xc->hit_tile, tid);
        __syncthreads();
    }
    auto mark = [&](int t) {
        if (t >= 0 && t < nsub && atomicCAS(&xc->of[t], 0, -1) == 0) {
            const int e = atomicAdd(&xc->n, 1);
            if (e < kXcEntries) { xc->tile[e] = t; xc->of[t] = e + 1; } else { xc->of[t] = 0; }
        }
    };
    if (tid < 4) mark(tid);
    if (tid < nsub && wk->xslot[tid]) { mark(tid - 1); mark(tid); mark(tid + 1); mark(tid + 2); }
    if (has_target && tid == 0 && xc->hit_tile != INT_MAX) { mark(xc->hit_tile - 1); mark(xc->hit_tile); mark(xc->hit_tile + 1); }
    __syncthreads();
    const int ne = min(xc->n, kXcEntries);
    for (int e = warp; e < ne; e += kThreads / 32) {
        float x[8];
        pv.reload(xc->tile[e] * kSub + lane * 8, n, x);
        float4 *q = (float4 *)(xdata + (size_t)e * kSub + lane * 8);
        q[0] = make_float4(x[0], x[1], x[2], x[3]);
        q[1] = make_float4(x[4], x[5], x[6], x[7]);
    }
    __syncthreads();
}

constexpr size_t kDrawSmem = sizeof(Emul2Work) + (size_t)kXcEntries * kSub * 4;

// ---- speculative verification in the flat form ---------------------------------------------------------
// What k_spec_finish (stg_spec_kernels.cu) does with one CTA per sequence - the accept chain, then one
// or two emulated sums over V whose every phase recomputes p (and q) from the logits - as three
// kernels: the accept chain (one warp per sequence, the draft positions evaluated side by side), ONE
// flat pass that writes the values the draw runs over - the final probabilities of the target row
// (bonus draw, or the looser rule's draw from p) or the residual max(p - q, 0) - into the sequence's
// scratch row with their sub-tile sums, guesses and composites (the tail k_full_psums has), and a
// per-sequence walk: for the residual first without a target (its sum), then to u * sum with the same
// composites.  Sequences whose draw needs one of the rare fall-backs (an empty residual, a walk that
// runs off the end, a look-back that ran out) are flagged, and k_spec_finish redoes exactly those.
struct SpecSeq {
    int32_t acc;       // accepted draft tokens
    int32_t kind;      // 0: done (greedy), 1: draw from the target row `acc`, 2: residual of position `acc`
    uint32_t flags;    // STG_SEQ_* gathered so far
    int32_t pad;
};

template <bool BF16>
__global__ void __launch_bounds__(256) k_spec_accept(const __grid_constant__ SpecArgs a, const FullWs ws, SpecSeq *seq,
                                                     int32_t *fallback)
{
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= a.n_seq) return;
    const int L = a.n_draft, V = a.vocab;
    const int esz = BF16 ? 2 : 4;
    const RowDist *td = a.tdist + (int64_t)s * (L + 1);
    const RowDist *dd = a.ddist ? a.ddist + (int64_t)s * L : nullptr;
    const char *trows = (const char *)a.target + (int64_t)s * (L + 1) * V * esz;
    const char *drows = a.draft ? (const char *)a.draft + (int64_t)s * L * V * esz : nullptr;
    const double *u = a.uniforms + (int64_t)s * (L + 2);
    const bool greedy = (td[0].flags & kDistOneHot) != 0;
    bool ok = true, bad = false;
    float shown = 0.f;
    if (lane < L) {
        const int i = lane;
        const int tok = a.draft_tokens[(int64_t)s * L + i];
        if ((unsigned)tok >= (unsigned)V) {
            // a draft token outside the vocabulary (the reference's pDist[tokens[i]] throws,
            // SpeculativeDecoder.cs:534): never read, rejected, and reported in the flags
            ok = false;
            bad = true;
        } else if (greedy) {
            ok = (tok == td[i].tie_idx_max);  // SpeculativeDecoder.Step, SpeculativeDecoder.cs:400-405
            shown = ok ? 1.f : 0.f;
        } else {
            const float px = eval_point<BF16>(LogitRow{trows + (int64_t)i * V * esz, a.target_cap}, tok, td[i]);
            if (a.mode == 0) {
                const float qx = eval_point<BF16>(LogitRow{drows + (int64_t)i * V * esz, a.draft_cap}, tok, dd[i]);
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
    // positions after the first rejection are not tested
    if (a.accept_probs && lane < L) a.accept_probs[(int64_t)s * L + lane] = lane <= acc ? shown : 0.f;
    const bool bad_draft = acc < L && __shfl_sync(0xFFFFFFFFu, bad ? 1 : 0, acc) != 0;
    if (lane == 0) {
        const uint32_t fl = bad_draft ? (1u << 9) : 0u;
        SpecSeq q;
        q.acc = acc;
        q.flags = fl;
        q.pad = 0;
        q.kind = greedy ? 0 : ((acc == L || a.mode == 1) ? 1 : 2);
        seq[s] = q;
        fallback[s] = 0;
        a.accepted[s] = acc;
        if (greedy) {
            a.correction[s] = td[acc].tie_idx_max;
            if (a.seq_flags) a.seq_flags[s] = fl;
        }
        FullRow *fr = ws.rows + s;
        fr->redo = 0;
        fr->n_cross[1] = 0;
    }
    FullRow *fr = ws.rows + s;
    for (int p = lane; p < kFullMaxParts; p += 32) fr->pflag[1][p] = 0u;
}

template <bool BF16>
__global__ void __launch_bounds__(kFullThreads) k_spec_values(const __grid_constant__ SpecArgs a, const FullWs ws,
                                                              const SpecSeq *seq)
{
    __shared__ float s_sum[kPieceSubTiles];
    __shared__ unsigned char s_guess[kPieceSubTiles], s_xslot[kPieceSubTiles];
    __shared__ int s_ok;
    const int s = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SpecSeq q = seq[s];
    if (q.kind == 0) return;
    const int L = a.n_draft, n = a.vocab;
    const int begin = blockIdx.x * kPhasePiece;
    if (begin >= n) return;
    const int esz = BF16 ? 2 : 4;
    const bool al = a.vec == 4;
    const RowDist td = a.tdist[(int64_t)s * (L + 1) + q.acc];
    const LogitRow prow{(const char *)a.target + ((int64_t)s * (L + 1) + q.acc) * n * esz, a.target_cap};
    const ProvRow<BF16> pp{SrcLogits<BF16>{prow, nullptr, al, td.inv_t, td.inv_t != 1.0f}, td};
    FullRow *fr = ws.rows + s;
    Emul2Work *ew = ws.ew + s;
    float *e = ws.e + (size_t)s * ws.e_stride;
    constexpr int W = kFullThreads / 32;
    float xs[kWarpSubTiles][8];
    if (q.kind == 2) {
        const RowDist dq = a.ddist[(int64_t)s * L + q.acc];
        const LogitRow qrow{(const char *)a.draft + ((int64_t)s * L + q.acc) * n * esz, a.draft_cap};
        const ProvRow<BF16> qq{SrcLogits<BF16>{qrow, nullptr, al, dq.inv_t, dq.inv_t != 1.0f}, dq};
        const ProvResidual<BF16> rr{pp, qq};
#pragma unroll
        for (int i = 0; i < kWarpSubTiles; i++) {
            const int st = warp + i * W;
            rr.load(begin + st * kSub + lane * 8, n, xs[i]);  // zeros beyond the row
        }
    } else {
#pragma unroll
        for (int i = 0; i < kWarpSubTiles; i++) {
            const int st = warp + i * W;
            pp.load(begin + st * kSub + lane * 8, n, xs[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < kWarpSubTiles; i++) {
        const int st = warp + i * W;
        const int base = begin + st * kSub + lane * 8;
        if (begin + st * kSub >= n) continue;  // the same for the whole warp
        if (base < n) store8(e, base, n, xs[i]);
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++) acc += xs[i][j] > 0.f ? xs[i][j] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        if (lane == 0) { ew->sums[(begin >> 8) + st] = acc; s_sum[st] = acc; }
    }
    piece_tail<true>(fr, ew, xs, begin, n, s_sum, s_guess, s_xslot, &s_ok);
}

__global__ void __launch_bounds__(kThreads, 1) k_spec_draw(const __grid_constant__ SpecArgs a, const FullWs ws,
                                                           const SpecSeq *seq, int32_t *fallback)
{
    extern __shared__ __align__(16) unsigned char arena[];
    __shared__ Emul2Ctl ctl;
    __shared__ XCache xcache;
    const int s = blockIdx.x, tid = threadIdx.x;
    const SpecSeq q = seq[s];
    if (q.kind == 0) return;
    const FullRow *fr = ws.rows + s;
    if (fr->redo) {
        if (tid == 0) fallback[s] = 1;
        return;
    }
    const int L = a.n_draft, n = a.vocab;
    const int nsub = (n + kSub - 1) / kSub;
    Emul2Work *wk2 = (Emul2Work *)arena;
    float *xdata = (float *)(arena + sizeof(Emul2Work));
    load_work(wk2, ws.ew + s);
    const ProvE pe{ws.e + (size_t)s * ws.e_stride};
    const float u0 = __double2float_rn(a.uniforms[(int64_t)s * (L + 2) + L]);
    float target = u0;
    if (q.kind == 2) {
        // ResampleResidual (Sampler.cs:587-618): the sum of the residual, then the draw to u * sum
        build_xcache(&xcache, xdata, wk2, pe, n, nsub, 0.f, false);
        if (tid < 32) {
            const ProvCached<ProvE> pc{pe, xdata, xcache.of};
            emul2_walk<ProvCached<ProvE>, false, false>(&ctl, wk2, pc, n, nsub, 0.f, false, nullptr, nullptr);
        }
        __syncthreads();
        const float sum = ctl.s;
        __syncthreads();
        if (!(sum > 0.f)) {  // nothing left of p - q (or NaN): the draw from p with the spare uniform
            if (tid == 0) fallback[s] = 1;
            return;
        }
        target = __fmul_rn(u0, sum);
    }
    build_xcache(&xcache, xdata, wk2, pe, n, nsub, target, true);
    if (tid < 32) {
        const ProvCached<ProvE> pc{pe, xdata, xcache.of};
        emul2_walk<ProvCached<ProvE>, false, false>(&ctl, wk2, pc, n, nsub, target, true, nullptr, nullptr);
    }
    __syncthreads();
    if (tid == 0) {
        int corr = ctl.hit;
        uint32_t fl = q.flags;
        if (corr < 0) {
            if (q.kind == 2) { fallback[s] = 1; return; }  // the rounding fall-back of the residual draw
            corr = n - 1;
            fl |= (1u << 5);
        }
        a.correction[s] = corr;
        if (a.seq_flags) a.seq_flags[s] = fl;
    }
}

cudaError_t launch_spec_flat(const SpecArgs &a, const FullWs &ws, void *seq_ctl, int32_t *fallback, cudaStream_t stream)
{
    SpecSeq *seq = (SpecSeq *)seq_ctl;
    cudaError_t e = ensure_dynamic_smem((const void *)k_spec_draw, kDrawSmem);
    if (e != cudaSuccess) return e;
    const dim3 pg((unsigned)((a.vocab + kPhasePiece - 1) / kPhasePiece), (unsigned)a.n_seq);
    if (a.dtype == 1) {
        k_spec_accept<true><<<(a.n_seq + 7) / 8, 256, 0, stream>>>(a, ws, seq, fallback);
        k_spec_values<true><<<pg, kFullThreads, 0, stream>>>(a, ws, seq);
    } else {
        k_spec_accept<false><<<(a.n_seq + 7) / 8, 256, 0, stream>>>(a, ws, seq, fallback);
        k_spec_values<false><<<pg, kFullThreads, 0, stream>>>(a, ws, seq);
    }
    k_spec_draw<<<a.n_seq, kThreads, kDrawSmem, stream>>>(a, ws, seq, fallback);
    return cudaGetLastError();
}

}  // namespace stg
