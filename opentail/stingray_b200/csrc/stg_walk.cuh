// The exact sequential fp32 sum of a row, walked by one warp over per-tile summaries.
//
// The arithmetic is that of stg_emul.cuh / stg_emul2.cuh: inside a binade the running sum is an
// integer number of units, an element is the pair of its increments for an even and an odd sum, pairs
// compose, and a tile of 256 elements is the composition of its elements under the binade the sum is
// guessed to be in when it gets there (from an fp64 prefix of the tiles' plain sums).  What this file
// adds to emul2_walk is that almost nothing is left to do serially:
//
//   * consecutive tiles with one guessed binade form a run, whose composition is computed beside the
//     walk: a run costs one load, one addition and one comparison;
//   * a tile in which the sum should pass into the next binade carries, per lane (8 elements), the
//     composition of the lanes before it under the old binade and of the lanes behind it under the new
//     one: a crossing is one ballot, one lane's 8 additions and one lookup;
//   * the tiles in which neither holds - the first one, where the sum starts from zero and changes binade
//     every few elements, a jump over two binades, the tile the target should lie in - are added element
//     by element from shared memory (an fp32 addition is four cycles, a warp scan several hundred).
//
// Whatever does not go as guessed is replayed exactly (replay_subtile).  The result never depends on the
// guesses.  Measured on a lone row of 151,936: 16-20 thousand cycles with a warp scan per run and per
// crossing, some 10 thousand so.
#pragma once
#include "stg_emul2.cuh"

namespace stg {

constexpr int kWalkCross = 16;  // binades that have a slot: the last 16 of the sum

// kind of a tile: the first of a run, another one of it, 1 + slot: a prepared crossing, kTileSlot + slot: serial
// with its elements in the slot, kTileReplay: serial without
enum : int { kTileRun = 0, kTileMid = 127, kTileSlot = 128, kTileReplay = 255 };

struct WalkCross {
    int2 lo[32];    // composition of lanes 0 .. l under binade g
    int2 hi[34];    // composition of lanes l .. 31 under binade g + 1 ([32]: nothing)
    float x[kSub];
    int tile;       // whose slot this is
    int pad[3];
};

struct WalkArea {
    uint32_t desc[kMaxSubTiles];  // guessed biased exponent of the sum in front of the tile | kind << 8 | last tile of the run << 16
    int2 tot[kMaxSubTiles];       // first tile of a run: composition of the run
    int2 comp[kMaxSubTiles];      // composition of every tile under its guess: even / odd start
    WalkCross xs[kWalkCross + 1]; // [kWalkCross]: the tile the target should lie in
    float head[kSub];             // elements of tile 0
};

// What few tiles need lies out of line: inlined into the loops that all tiles go through it made those wait for their
// own instructions.
struct Lane8 { float v[8]; };  // by value: a called function gets a lane's elements in registers
__device__ __forceinline__ Lane8 lane8(const float x[8])
{
    Lane8 l;
#pragma unroll
    for (int j = 0; j < 8; j++) l.v[j] = x[j];
    return l;
}
static __device__ __noinline__ int2 composite_any(const Lane8 x, int g)
{
    int r0, r1;
    subtile_composite<false>(x.v, g, r0, r1);
    return make_int2(r0, r1);
}

struct WalkOut {
    float s;        // the sum at the hit, or the final sum
    float before;   // the sum just before the element that met the target
    int hit;        // first element at which the sum is >= target, -1: none
};

// s = fl(s + x[i]) over `m` elements (a multiple of 8; zeros pad) until s >= target.  The same in every lane.
__device__ __forceinline__ int serial_tile(const float *xp, int m, float target, bool has_target, float &s, float &before)
{
    const float4 *q = (const float4 *)xp;
    float4 a = q[0], b = q[1];
    for (int i = 0; i < m; i += 8) {
        const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        const int nx = i + 8 < m ? (i + 8) >> 2 : 0;
        a = q[nx];
        b = q[nx + 1];
        float r = s;
#pragma unroll
        for (int j = 0; j < 8; j++) r = __fadd_rn(r, x[j]);
        if (has_target && r >= target) {
            float c = s;
            int h = -1;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (h < 0) {
                    before = c;
                    c = __fadd_rn(c, x[j]);
                    if (c >= target) h = i + j;
                }
            }
            s = c;
            return h;
        }
        s = r;
    }
    return -1;
}

// `get(t, x)`: this lane's 8 elements of tile t (zeros beyond the row).  All 32 lanes of one warp.
template <class Get>
__device__ __forceinline__ WalkOut row_walk(const WalkArea *w, const Get &get, int n, int nsub, float target, bool has_target)
{
    const int lane = threadIdx.x & 31;
    WalkOut o;
    o.before = 0.f;
    o.s = 0.f;
    o.hit = serial_tile(w->head, kSub, target, has_target, o.s, o.before);
    if (o.hit >= 0) {
        if (o.hit >= n) o.hit = -1;
        return o;
    }
    int t = 1;
    while (t < nsub) {
        const uint32_t sb = __float_as_uint(o.s);
        const int eb = (int)(sb >> 23) & 255;  // the sum is >= 0
        if (eb == 255) break;                  // inf / NaN: nothing changes any more
        if (sb == 0u) {
            // Nothing yet: a run without a positive element leaves it so (under the lowest guess every positive one counts).
            // Near-greedy rows are nothing else up to their maximum: 64 rows of 151,936 at T = 1e-5 516 -> 56 us.
            const uint32_t d = w->desc[t];
            const int2 v = w->tot[t];
            if ((d & 0xFFFFu) == (1u | (kTileRun << 8)) && (v.x | v.y) == 0) {
                t = (int)(d >> 16) + 1;
                continue;
            }
        }
        int sint = (int)((sb & 0x7FFFFFu) | 0x800000u);
        bool replay = eb < 24;                 // sums that small have no summaries
        if (!replay) {
            const long long tl = target_units(target, has_target, eb);
            const int tint = (int)(tl > (1 << 30) ? (1 << 30) : tl), lim = min(tint, 1 << 24);
            uint32_t d = w->desc[t];
            // the runs that stay in this binade
            while ((d & 0xFFFFu) == (uint32_t)(eb | (kTileRun << 8))) {
                const int2 v = w->tot[t];
                const int S = sint + ((sint & 1) ? v.y : v.x);
                if (S >= lim) break;
                sint = S;
                t = (int)(d >> 16) + 1;
                if (t >= nsub) break;
                d = w->desc[t];
            }
            o.s = __uint_as_float(((uint32_t)eb << 23) | ((uint32_t)sint & 0x7FFFFFu));
            if (t >= nsub) break;
            const int kind = (int)(d >> 8) & 255;
            const bool right = (int)(d & 255u) == eb;
            if (kind >= kTileSlot && kind != kTileReplay && w->xs[kind - kTileSlot].tile == t) {
                const int h = serial_tile(w->xs[kind - kTileSlot].x, kSub, target, has_target, o.s, o.before);
                if (h >= 0) { o.hit = t * kSub + h < n ? t * kSub + h : -1; return o; }
                t++;
                continue;
            }
            if (right && kind >= 1 && kind <= kWalkCross) {
                const WalkCross &c = w->xs[kind - 1];
                const int2 lo = c.lo[lane];
                const int S1 = sint + ((sint & 1) ? lo.y : lo.x);  // sum after lanes 0 .. lane
                const unsigned over = __ballot_sync(0xFFFFFFFFu, S1 >= (1 << 24));
                const unsigned met = __ballot_sync(0xFFFFFFFFu, S1 >= tint);
                if (c.tile == t && over && !(met & ((over & (0u - over)) - 1u))) {
                    const int L = __ffs(over) - 1;
                    const float4 *q = (const float4 *)(c.x + L * 8);  // every lane adds lane L's elements
                    const float4 q0 = q[0], q1 = q[1];
                    const int2 hi = c.hi[L + 1];
                    const int pv = __shfl_sync(0xFFFFFFFFu, S1, L > 0 ? L - 1 : 0);
                    const int prev = L > 0 ? pv : sint;
                    float acc = __uint_as_float(((uint32_t)eb << 23) | ((uint32_t)prev & 0x7FFFFFu));
                    acc = __fadd_rn(acc, q0.x); acc = __fadd_rn(acc, q0.y); acc = __fadd_rn(acc, q0.z); acc = __fadd_rn(acc, q0.w);
                    acc = __fadd_rn(acc, q1.x); acc = __fadd_rn(acc, q1.y); acc = __fadd_rn(acc, q1.z); acc = __fadd_rn(acc, q1.w);
                    const uint32_t ab = __float_as_uint(acc);
                    if ((int)(ab >> 23) == eb + 1 && eb < 253 && !(has_target && acc >= target)) {
                        const int sint2 = (int)((ab & 0x7FFFFFu) | 0x800000u);
                        const int S2 = sint2 + ((sint2 & 1) ? hi.y : hi.x);
                        if (S2 < (1 << 24) && (long long)S2 < target_units(target, has_target, eb + 1)) {
                            o.s = __uint_as_float(((uint32_t)(eb + 1) << 23) | ((uint32_t)S2 & 0x7FFFFFu));
                            t++;
                            continue;
                        }
                    }
                }
            } else if (right && (kind == kTileRun || kind == kTileMid)) {
                // the sum leaves the binade or meets the target inside a run, or a run is entered in its middle
                // (behind a tile that was guessed wrongly): 32 tiles at a time
                const int tt = t + lane;
                int i0 = 0, i1 = 0;
                bool valid = false;
                if (tt < nsub) {
                    const int2 v = w->comp[tt];
                    i0 = v.x;
                    i1 = v.y;
                    const uint32_t dd = w->desc[tt];
                    const int k = (int)(dd >> 8) & 255;
                    valid = (k == kTileRun || k == kTileMid) && (int)(dd & 255u) == eb;
                }
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) {
                    const int p0 = __shfl_up_sync(0xFFFFFFFFu, i0, s), p1 = __shfl_up_sync(0xFFFFFFFFu, i1, s);
                    if (lane >= s) { int r0, r1; comp(p0, p1, i0, i1, r0, r1); i0 = r0; i1 = r1; }
                }
                const int S = sat_add(sint, (sint & 1) ? i1 : i0);
                const unsigned m = __ballot_sync(0xFFFFFFFFu, !valid || S >= lim);
                const int ok = m ? __ffs(m) - 1 : 32;
                if (ok > 0) {
                    const int S2 = __shfl_sync(0xFFFFFFFFu, S, ok - 1);
                    o.s = __uint_as_float(((uint32_t)eb << 23) | ((uint32_t)S2 & 0x7FFFFFu));
                    t += ok;
                    continue;
                }
            }
        }
        // exact replay of one tile
        float x[8];
        get(t, x);
        const int h = replay_subtile<false>(x, t * kSub, n, target, has_target, o.s, o.before);
        if (h >= 0) { o.hit = h; return o; }
        t++;
    }
    return o;
}

// One warp: runs and descriptors of the tiles [t0, t1) from their guesses, kinds (kTileRun for every tile of
// a run) and compositions (arrays indexed by t - t0, shared memory), written to `dst`, the area of the CTA
// that walks.  A run never crosses t0.
__device__ __forceinline__ void walk_runs(WalkArea *dst, const int2 *cmp, const unsigned char *guess, const unsigned char *kind,
                                          int t0, int t1)
{
    const int lane = threadIdx.x & 31;
    int c0 = 0, c1 = 0, c_first = t0;  // composition and first tile of the run the previous 32 tiles ended in
    for (int b = t0; b < t1; b += 32) {
        const int t = b + lane, i = t - t0;
        const bool in = t < t1;
        const int k = in ? kind[i] : (int)kTileReplay, g = in ? guess[i] : 0;
        const bool run = in && k == kTileRun;
        const bool joins = run && t > t0 && kind[i - 1] == kTileRun && guess[i - 1] == g;
        const bool ends = run && (t + 1 >= t1 || kind[i + 1] != kTileRun || guess[i + 1] != g);
        const int2 v = run ? cmp[i] : make_int2(0, 0);
        int a0 = v.x, a1 = v.y;
        const unsigned heads = __ballot_sync(0xFFFFFFFFu, !joins);
        const unsigned mine = heads & (0xFFFFFFFFu >> (31 - lane));
        const int first_lane = mine ? 31 - __clz(mine) : -1;  // -1: the run began in an earlier round
        const unsigned tails = __ballot_sync(0xFFFFFFFFu, ends);
        if (!__any_sync(0xFFFFFFFFu, a0 != a1 || c0 != c1)) {
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int p0 = __shfl_up_sync(0xFFFFFFFFu, a0, d);
                if (lane - d >= max(first_lane, 0)) a0 = sat_add(a0, p0);
            }
            if (first_lane < 0) a0 = sat_add(a0, c0);
            a1 = a0;
        } else {
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int p0 = __shfl_up_sync(0xFFFFFFFFu, a0, d), p1 = __shfl_up_sync(0xFFFFFFFFu, a1, d);
                if (lane - d >= max(first_lane, 0)) { int r0, r1; comp(p0, p1, a0, a1, r0, r1); a0 = r0; a1 = r1; }
            }
            if (first_lane < 0) { int r0, r1; comp(c0, c1, a0, a1, r0, r1); a0 = r0; a1 = r1; }
        }
        const int first = first_lane < 0 ? c_first : b + first_lane;
        if (ends) {
            dst->tot[first] = make_int2(a0, a1);
            if (first_lane < 0) dst->desc[first] = (uint32_t)g | (kTileRun << 8) | ((uint32_t)t << 16);
        }
        if (in) {
            // a first tile whose run ends in this round names its last tile; the others are named when it is known
            const unsigned after = tails & (0xFFFFFFFFu << lane);
            const int last = after ? b + __ffs(after) - 1 : t;
            const int kk = run ? (first == t ? (int)kTileRun : (int)kTileMid) : k;
            if (!(run && first == t && !after)) dst->desc[t] = (uint32_t)g | ((uint32_t)kk << 8) | ((uint32_t)last << 16);
        }
        c0 = __shfl_sync(0xFFFFFFFFu, a0, 31);
        c1 = __shfl_sync(0xFFFFFFFFu, a1, 31);
        c_first = __shfl_sync(0xFFFFFFFFu, first, 31);
    }
}

// One warp: prepares the crossing of a tile from binade g (this lane's 8 elements in x)
static __device__ __noinline__ void walk_cross(WalkCross *dst, const Lane8 e, int g)
{
    const float (&x)[8] = e.v;
    const int lane = threadIdx.x & 31;
    int l0, l1, h0, h1;
    lane_composite(x, g, l0, l1);
    lane_composite(x, g + 1, h0, h1);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int p0 = __shfl_up_sync(0xFFFFFFFFu, l0, d), p1 = __shfl_up_sync(0xFFFFFFFFu, l1, d);
        if (lane >= d) { int r0, r1; comp(p0, p1, l0, l1, r0, r1); l0 = r0; l1 = r1; }
        const int q0 = __shfl_down_sync(0xFFFFFFFFu, h0, d), q1 = __shfl_down_sync(0xFFFFFFFFu, h1, d);
        if (lane + d < 32) { int r0, r1; comp(h0, h1, q0, q1, r0, r1); h0 = r0; h1 = r1; }
    }
    dst->lo[lane] = make_int2(l0, l1);
    dst->hi[lane] = make_int2(h0, h1);
    if (lane == 0) dst->hi[32] = make_int2(0, 0);
}

// kind of tile t given the guesses in front of it and behind it and that of the whole sum.  At most one tile
// leaves a binade upwards, so the binade names the slot.
__device__ __forceinline__ int walk_kind(int t, int g, int g_next, int g_end)
{
    if (t == 0) return kTileReplay;  // added from WalkArea::head
    if (g_next == g) return kTileRun;
    if (g <= g_end - kWalkCross) return kTileReplay;
    const int slot = g & (kWalkCross - 1);
    return g_next == g + 1 ? 1 + slot : kTileSlot + slot;
}

__device__ __forceinline__ float max_or_nan(float a, float b)
{
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}

// composition of a tile (8 consecutive elements per lane) under binade g; every lane gets it.  Where g >= 48 and no element
// reaches 2^(g - 128), half of the binade, adding 1.5 * 2^(g - 127) rounds each of them to the unit of the running sum, to even
// on a tie, in one addition.  Both are asked of the elements themselves: what a tile weighs is known beforehand, but only
// about (estimate_tile, stg_row.cu), and an element too large for its guess has other increments than the addition shows.
__device__ __forceinline__ void tile_composite(const float x[8], int g, int &r0, int &r1)
{
    if (g >= 48 && g < 250) {
        const float c = __uint_as_float(((uint32_t)g << 23) | 0x400000u);
        unsigned a = 0u;  // modulo 2^32
        float m = 0.f, top = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j += 2) {  // two elements to an instruction
            const float2 v = make_float2(x[j], x[j + 1]), y = __fadd2_rn(v, make_float2(c, c)), z = __fadd2_rn(y, make_float2(-c, -c));
            const float2 w = __ffma2_rn(z, make_float2(-1.f, -1.f), v);
            a += __float_as_uint(y.x) + __float_as_uint(y.y);
            m = fmaxf(m, fmaxf(fabsf(w.x), fabsf(w.y)));
            top = max_or_nan(top, max_or_nan(y.x, y.y));
        }
        a -= 8u * __float_as_uint(c);
        const bool odd = m == __uint_as_float((uint32_t)(g - 24) << 23) || !(top < __uint_as_float((uint32_t)(g + 1) << 23));
        if (__ballot_sync(0xFFFFFFFFu, odd) == 0u) {
            r0 = r1 = min((int)__reduce_add_sync(0xFFFFFFFFu, a), 1 << 28);  // at most 2^30, and two of them are to be added (sat_add)
            return;
        }
    }
    float any = x[0];
#pragma unroll
    for (int j = 1; j < 8; j++) any = fmaxf(any, x[j]);
    r0 = r1 = 0;
    if (__any_sync(0xFFFFFFFFu, any > 0.f)) {
        const int2 r = composite_any(lane8(x), g);
        r0 = r.x;
        r1 = r.y;
    }
}

}  // namespace stg
