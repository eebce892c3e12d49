// gi_contact.cuh -- device code of the contact pass shared by gi_grid.cu and
// the paired far field's kernel: the cell torus, the contact law, the
// fixed-point sums and the row path (see gi_grid.cu for the pass as a whole).
#pragma once

#include "gi_force_impl.cuh"

namespace gi {

__device__ __forceinline__ int cell_of(float x)
{
    float f = floorf(x);
    f = fminf(fmaxf(f, -1.0e9f), 1.0e9f);  // far debris shares edge cells; NaN -> -1e9
    return (int)f;
}

__device__ __forceinline__ int3 cell_of(float4 p)
{
    return make_int3(cell_of(p.x), cell_of(p.y), cell_of(p.z));
}

// The torus of a run's buckets: glog bits, x >= y >= z of them (z at least 3 for a
// run of more than kDirectAlways bodies: the 3 x 3 x 3 neighbours of a cell are
// distinct buckets, and cells that share one are too far apart to touch).
struct Torus {
    unsigned int base;
    int xb, yb;      // bits of x and y
    int xm, ym, zm;  // masks
};

__device__ __forceinline__ Torus torus_of(const RunDev &R)
{
    Torus t;
    const int zb = R.glog / 3;
    t.base = (unsigned int)R.gbase;
    t.yb = (R.glog - zb) >> 1;
    t.xb = R.glog - zb - t.yb;
    t.xm = (1 << t.xb) - 1;
    t.ym = (1 << t.yb) - 1;
    t.zm = (1 << zb) - 1;
    return t;
}

// First bucket of the x-row of cells (., cy, cz); then the bucket of a cell.
__device__ __forceinline__ unsigned int row_of(const Torus &t, int cy, int cz)
{
    return t.base + ((unsigned int)((cz & t.zm) << t.yb | (cy & t.ym)) << t.xb);
}

__device__ __forceinline__ unsigned int bucket_of(const Torus &t, int cx, int cy, int cz)
{
    return row_of(t, cy, cz) + (unsigned int)(cx & t.xm);
}

__device__ __forceinline__ unsigned int bucket_size(const unsigned int *start, unsigned int b)
{
    return start[b + 1] - start[b];
}

// Counters of the tiled path, in one block of kCtrWords words that start at
// zero: item count, tiled-bucket count, queue head, candidate buckets, then
// the items per cost class and the fill of each class while ordering,
// then a bit per run: has candidate buckets.
constexpr int kCtrItems = 0, kCtrTiled = 1, kCtrHead = 2, kCtrCand = 3, kCtrClass = 4,
              kCtrFill = kCtrClass + (int)kItemClasses, kCtrCrowds = kCtrFill + (int)kItemClasses;
static_assert(kCtrCrowds + GI_MAX_RUNS / 32 == kCtrWords, "tiled-path counter block");

__device__ __forceinline__ void set_crowds(unsigned int *ctr, unsigned int run)
{
    atomicOr(&ctr[kCtrCrowds + (run >> 5)], 1u << (run & 31u));
}

__device__ __forceinline__ bool has_crowds(const unsigned int *ctr, unsigned int run)
{
    return (__ldg(&ctr[kCtrCrowds + (run >> 5)]) >> (run & 31u)) & 1u;
}

// The bodies of a bucket that share its majority cell take the tiled path when
// they are at least tab.dense_min (kDenseMin unless set), or at least a quarter of
// that next to a bucket of that many: near a crowded remnant its bodies have
// enough contacts to pay the tiled path's fixed costs per item, while cells
// of ordinary settled bodies stay on the row path.  Either bound is at least
// kDenseFloor, which bounds the item count.  Buckets of at least dense_lo
// bodies are listed as candidates while they are counted.
// (kDenseFloor itself lives in gi_internal.h: it sizes the scratch.)
__host__ __device__ __forceinline__ unsigned int dense_hi(unsigned int dmin)
{
    return dmin > kDenseFloor ? dmin : kDenseFloor;
}

__host__ __device__ __forceinline__ unsigned int dense_lo(unsigned int dmin)
{
    return dmin / 4u > kDenseFloor ? dmin / 4u : kDenseFloor;
}

// Pair constants of body i against a j of one material: the class row of
// the table and the far-field term of a contact pair.
struct PairRow {
    float G, K, Tband, Tmid, KRmid, KRin;
    float far;  // -(gm_i gm_j) s_far, the clamped far-field coefficient at r2 < 1
};

__device__ __forceinline__ PairRow pair_row(const PairDev &P, bool ife, bool jfe)
{
    const int test = (int)ife + (int)jfe;
    PairRow w;
    w.G = P.G[test];
    w.K = P.K[test];
    w.Tband = P.Tband[test];
    w.Tmid = P.Tmid[test];
    w.KRmid = P.KRmid[test];
    w.KRin = P.KRin[test];
    // every contact pair has r2 < 1, where the all-pairs pass clamps r2 to 1
    const float ri = rsqrt_mufu(1.0f);
    const float s_far = (ri * ri) * ri;
    const float gmi = ife ? P.gm_fe : P.gm_si;
    const float gmj = jfe ? P.gm_fe : P.gm_si;
    w.far = -(gmi * gmj) * s_far;
    return w;
}

__device__ __forceinline__ PairRow select_row(bool jfe, const PairRow &fe, const PairRow &si)
{
    PairRow w;
    w.G = jfe ? fe.G : si.G;
    w.K = jfe ? fe.K : si.K;
    w.Tband = jfe ? fe.Tband : si.Tband;
    w.Tmid = jfe ? fe.Tmid : si.Tmid;
    w.KRmid = jfe ? fe.KRmid : si.KRmid;
    w.KRin = jfe ? fe.KRin : si.KRin;
    w.far = jfe ? fe.far : si.far;
    return w;
}

// Contact correction of one pair with r2 < 1, as a coefficient of dp in
// force units: the reference law's contact force on i, mag dp / r, minus
// the clamped far-field term gm_i gm_j dp the all-pairs pass added.
__device__ __forceinline__ float contact_coef(const PairRow &w, int sep_test, float dx, float dy,
                                              float dz, float r2, float4 vi, float4 vj)
{
    float K = w.K;
    if (!(r2 >= w.Tband)) {
        const float dvx = __fsub_rn(vj.x, vi.x), dvy = __fsub_rn(vj.y, vi.y),
                    dvz = __fsub_rn(vj.z, vi.z);
        const float dpdv = __fmaf_rn(dz, dvz, __fmaf_rn(dx, dvx, __fmul_rn(dy, dvy)));
        // Reference: int inout = dp.dv; KR when inout > 0, i.e. dp.dv >= 1.
        const bool sep = (sep_test == GI_SEP_SIGN) ? (dpdv > 0.0f) : (dpdv >= 1.0f);
        if (sep) K = (r2 >= w.Tmid) ? w.KRmid : w.KRin;
    }
    const float mag = contact_mag(w.G, K, r2);
    // 1 / r: MUFU rsqrt and one Newton-Raphson step (about 1 ulp)
    float invr = rsqrt_mufu(r2);
    invr = invr * __fmaf_rn(-0.5f * r2 * invr, invr, 1.5f);
    return __fmaf_rn(mag, invr, w.far);
}

// contact_coef with the velocities read (from shared memory) only for pairs
// inside the shell band, where the separation test needs it.  Same
// arithmetic, same result.
__device__ __forceinline__ float contact_coef_at(const PairRow &w, int sep_test, float dx,
                                                 float dy, float dz, float r2,
                                                 const float4 *vi, const float4 *vj)
{
    float K = w.K;
    if (!(r2 >= w.Tband)) {
        const float4 u = *vi, v = *vj;
        const float dvx = __fsub_rn(v.x, u.x), dvy = __fsub_rn(v.y, u.y),
                    dvz = __fsub_rn(v.z, u.z);
        const float dpdv = __fmaf_rn(dz, dvz, __fmaf_rn(dx, dvx, __fmul_rn(dy, dvy)));
        const bool sep = (sep_test == GI_SEP_SIGN) ? (dpdv > 0.0f) : (dpdv >= 1.0f);
        if (sep) K = (r2 >= w.Tmid) ? w.KRmid : w.KRin;
    }
    const float mag = contact_mag(w.G, K, r2);
    float invr = rsqrt_mufu(r2);
    invr = invr * __fmaf_rn(-0.5f * r2 * invr, invr, 1.5f);
    return __fmaf_rn(mag, invr, w.far);
}

// Fixed-point sums without the FP64 unit.  Each pair term x (FP32, in
// units of the fixed point) is rounded to the nearest integer, ties to
// even, exactly as cvt.rni.s64.f32 would; that instruction issues on the
// FP64 unit, the slowest unit of this GPU, so the terms are split on the
// FP32 pipe instead.  For |x| < 2^45:
//   s = fl(x + 1.5 2^46) is x rounded to a multiple of 2^23 (ulp 2^23) plus
//       1.5 2^46, and stays in [2^46, 2^47], so its bit pattern minus that
//       of 1.5 2^46 is hi = (s - 1.5 2^46) / 2^23;
//   lo = x - hi 2^23 is exact (|lo| <= 2^22), and fl(lo + 1.5 2^23) rounds
//       it to an integer (ulp 1, ties to even), read back the same way.
// round(x) = hi 2^23 + round(lo) because 2^23 is even.  Bit patterns are
// summed mod 2^32 and folded into 64 bits at most every kFixFold terms,
// before the 32-bit sums of hi and lo (each |.| <= 2^22 a term) can wrap.
constexpr float kFixM = 0x1.8p46f;  // 1.5 * 2^46
constexpr float kFixC = 0x1.8p23f;  // 1.5 * 2^23
constexpr float kFixMax = 0x1p45f;  // largest |term| the split takes
constexpr unsigned int kFixFold = 256;
// A pair term is at most 2^40 (1 + 2^-16) units (see fix_in_range).
static_assert(0x1p40f * (1.0f + 0x1p-16f) < kFixMax, "the split must take every pair term");
// kFixFold terms of at most 2^22 each fit the 32-bit pending sums.
static_assert((double)kFixFold * 0x1p22 < 0x1p31, "pending sums must not wrap");

struct FixSum3 {
    long long x, y, z;           // folded sums
    unsigned int hx, hy, hz;     // pending bit-pattern sums of s
    unsigned int lx, ly, lz;     // pending bit-pattern sums of fl(lo + 1.5 2^23)
    unsigned int n;              // pending terms
};

__device__ __forceinline__ void fix_zero(FixSum3 &a)
{
    a.x = a.y = a.z = 0;
    a.hx = a.hy = a.hz = a.lx = a.ly = a.lz = a.n = 0u;
}

__device__ __forceinline__ void fix_split(float x, unsigned int &h, unsigned int &l)
{
    const float s = __fadd_rn(x, kFixM);
    const float lo = __fsub_rn(x, __fsub_rn(s, kFixM));
    h += __float_as_uint(s);
    l += __float_as_uint(__fadd_rn(lo, kFixC));
}

__device__ __forceinline__ long long fix_value(unsigned int h, unsigned int l, unsigned int n)
{
    const int hi = (int)(h - n * __float_as_uint(kFixM));
    const int lo = (int)(l - n * __float_as_uint(kFixC));
    return (long long)hi * (1ll << 23) + lo;
}

__device__ __forceinline__ void fix_fold(FixSum3 &a)
{
    a.x += fix_value(a.hx, a.lx, a.n);
    a.y += fix_value(a.hy, a.ly, a.n);
    a.z += fix_value(a.hz, a.lz, a.n);
    a.hx = a.hy = a.hz = a.lx = a.ly = a.lz = a.n = 0u;
}

// The split is exact for every term of a pair with a normal r2: there
// 1 / r is finite, |d| <= r (up to rounding), so |c d| <= (|mag| + G m m) /
// unit <= 2^40 (1 + 2^-16) < kFixMax, the fixed-point unit being
// (2 Gmax + Kmax) 2^-40.  Coincident bodies (r2 = 0), a denormal r2 (the
// MUFU rsqrt flushes it to zero) or NaN take the hardware conversion,
// which rounds the same way; so the choice never changes a result.
__device__ __forceinline__ bool fix_in_range(float r2) { return r2 >= 0x1p-126f; }

// Adds round(c dx), round(c dy), round(c dz) for a pair of squared
// distance r2 (see fix_in_range); x and y in packed FP32x2 instructions,
// with the roundings of fix_split (s = fl(t + M); lo = fl(t - fl(s - M)),
// here as fma(fl(s - M), -1, t); fl(lo + C)).  FOLD: fold when kFixFold
// terms are pending (a caller that adds fewer terms between its own folds
// passes false).
template <bool FOLD = true>
__device__ __forceinline__ void fix_add3(FixSum3 &a, float c, float dx, float dy, float dz,
                                         float r2)
{
    const float2 txy = __fmul2_rn(make_float2(c, c), make_float2(dx, dy));
    const float tz = __fmul_rn(c, dz);
    if (fix_in_range(r2)) {
        const float2 s = __fadd2_rn(txy, make_float2(kFixM, kFixM));
        const float2 lo = __ffma2_rn(__fadd2_rn(s, make_float2(-kFixM, -kFixM)),
                                     make_float2(-1.0f, -1.0f), txy);
        const float2 l = __fadd2_rn(lo, make_float2(kFixC, kFixC));
        a.hx += __float_as_uint(s.x);
        a.hy += __float_as_uint(s.y);
        a.lx += __float_as_uint(l.x);
        a.ly += __float_as_uint(l.y);
        fix_split(tz, a.hz, a.lz);
        ++a.n;
        if (FOLD && a.n == kFixFold) fix_fold(a);
    } else {
        a.x += __float2ll_rn(txy.x);
        a.y += __float2ll_rn(txy.y);
        a.z += __float2ll_rn(tz);
    }
}

// The bodies of bucket b (of the torus T) that take the tiled path (see
// dense_hi), by one warp: their number and their cell c, 0 for none.  They are
// the bucket's majority cell; bodies of another cell that share the bucket
// (the torus is at least 8 cells wide, so they are far away) stay on the row
// path.
__device__ __forceinline__ unsigned int bucket_tiled(const Torus &T, const unsigned int *start,
                                                     const float4 *spos, unsigned int b,
                                                     unsigned int dmin, int lane, int3 &c)
{
    const unsigned int beg = start[b], end = start[b + 1], lo = dense_lo(dmin);
    if (end - beg < lo) return 0u;
    unsigned int same = 0u, first = beg;
    for (int tries = 0; tries < 2; ++tries) {
        // the bodies of the cell of slot `first`, and the first of another one
        c = cell_of(spos[first]);
        unsigned int n = 0u, other = end;
        for (unsigned int u = beg + lane; u < end; u += 128) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const unsigned int k = u + 32 * v;
                const int3 d = cell_of(spos[min(k, end - 1u)]);
                const bool eq = d.x == c.x && d.y == c.y && d.z == c.z;
                if (k < end) {
                    n += eq;
                    if (!eq) other = min(other, k);
                }
            }
        }
        same = __reduce_add_sync(0xffffffffu, n);
        first = __reduce_min_sync(0xffffffffu, other);
        if (2u * same > end - beg || first == end) break;
    }
    if (2u * same <= end - beg || same < lo) return 0u;
    bool crowded = same >= dense_hi(dmin);
    if (!crowded && lane < 27)
        crowded = bucket_size(start, bucket_of(T, c.x + lane % 3 - 1, c.y + (lane / 3) % 3 - 1,
                                               c.z + lane / 9 - 1)) >= dense_hi(dmin);
    return __any_sync(0xffffffffu, crowded) ? same : 0u;
}

// Whether bucket b's tiled bodies, if it has any, are those of cell c.  The
// states are written for buckets of at least dense_lo bodies alone.
__device__ __forceinline__ bool cell_tiled(const GridView &g, unsigned int b, int3 c,
                                           unsigned int dmin)
{
    const unsigned int beg = __ldg(&g.start[b]);
    if (__ldg(&g.start[b + 1]) - beg < dense_lo(dmin) || __ldg(&g.state[b]) == 0u) return false;
    const int3 d = cell_of(__ldg(&g.dpos[beg]));
    return c.x == d.x && c.y == d.y && c.z == d.z;
}

// The row path: one warp, a few consecutive bodies of a run.  Bodies that
// share their candidates form a group; the warp's lanes are split evenly among
// a group's bodies (1 to 8 of them, 32 to 4 lanes each), so a lone body gets
// all of them.  The candidates come as up to 32 slot ranges, one per lane; the
// warp stages their positions in shared memory kRowStage at a time (cp.async,
// the next batch while this one is tested, so that a warp waits for memory
// once and not once per range), and a body's lanes test them in turn.  Hits
// (r2 < 1) go to the body's shared list, and its lanes share the list when the
// law is evaluated, so the law runs on nearly full warps.
//
// What bounds it is the issue rate: at 66,000 settled bodies (about 150
// candidates and 18 contacts a body) one warp per body, with its own 27
// bucket look-ups, a candidate search over them and half-empty evaluations,
// took 70 us alone, this path 31.
//
// A tiled cell is no candidate here: its items give both sides of its pairs
// with its neighbours, and add to the corrections beside this path.  The few
// bodies around a remnant's core had thousands of such candidates, a warp
// with the longest list lasting 130 us (4,500 bodies) to 330 us (66,000) after
// the rest were done: a step of 20,000 remnant bodies took 531 us with them,
// 391 without.
constexpr int kRowStage = 128;  // candidates staged at a time
constexpr int kRowList = 512;   // hits listed: 16 per lane before they are drained
constexpr int kRowLaw = 4;      // hits of a lane evaluated at a time

struct RowSmem {
    float4 stage[2][kRowStage];
    unsigned int slot[2][kRowStage];
    unsigned int list[kRowList];
};

__device__ __forceinline__ void copy_async16(void *smem, const void *global)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned int)__cvta_generic_to_shared(smem)),
                 "l"(global)
                 : "memory");
}

// The batch of candidates at `base`: lane's range starts at slot beg, its
// candidates at excl.  DIRECT: slot t is candidate t.  Places past the last
// candidate get a position that is never a hit.
template <bool DIRECT>
__device__ __forceinline__ void row_fetch(RowSmem &sm, const float4 *__restrict__ cpos, int buf,
                                          unsigned int base, unsigned int total, unsigned int beg,
                                          unsigned int excl, int lane)
{
#pragma unroll
    for (int v = 0; v < kRowStage / 32; ++v) {
        const unsigned int t = base + 32 * v + lane;
        unsigned int slot = t;
        if (!DIRECT) {
            // the lane whose range holds t: the last one with excl <= t
            int src = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const unsigned int e = __shfl_sync(0xffffffffu, excl, (src + step) & 31);
                if (src + step < 32 && e <= t) src += step;
            }
            slot = __shfl_sync(0xffffffffu, beg - excl, src) + t;
        }
        if (t < total) {
            copy_async16(&sm.stage[buf][32 * v + lane], cpos + slot);
            sm.slot[buf][32 * v + lane] = slot;
        } else {
            sm.stage[buf][32 * v + lane].x = __int_as_float(0x7fffffff);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// A body as its lanes see it.
struct RowBody {
    float4 pi, vi;
    int i;              // body index (-1: none)
    unsigned int self;  // own slot, listed as a hit and passed over by the law
};

// One group: the lanes [k W, (k + 1) W) have body k of it, W = 1 << wlog.
// [beg, beg + cnt): the lane's range of candidates (ranges without candidates
// come last, or have the next one's excl).  add: to delta, else stored there.
template <bool DIRECT>
__device__ __forceinline__ void row_group(RowSmem &sm, const float4 *__restrict__ cpos,
                                          const float4 *__restrict__ cvel,
                                          long long *__restrict__ delta, const LaunchTable &tab,
                                          const RunDev &R, const PairDev &P, const RowBody &B,
                                          int wlog, unsigned int beg, unsigned int cnt, bool add, int lane)
{
    const int W = 1 << wlog, way = lane & (W - 1);
    const unsigned int mine = (wlog == 5 ? 0xffffffffu : (1u << W) - 1u) << (lane & ~(W - 1));
    const unsigned int below = mine & ((1u << lane) - 1u);
    unsigned int *const list = sm.list + 16 * (lane & ~(W - 1));  // 16 W places
    const unsigned int full = 16u * W - 4u * W;
    const float nan = __int_as_float(0x7fffffff);
    const float px = B.i >= 0 ? B.pi.x : nan;  // no body: no hits
    const int sw = R.offset + R.nfe;
    const float inv_unit = P.inv_unit;
    const PairRow row_fe = pair_row(P, B.i < sw, true), row_si = pair_row(P, B.i < sw, false);
    FixSum3 acc;
    fix_zero(acc);
    unsigned int nh = 0;  // hits listed, the same in the body's lanes

    // the contact law on the listed hits, kRowLaw of a lane's at a time with
    // all their loads in flight
    const auto drain = [&]() {
        __syncwarp();
        for (unsigned int k = way; k < nh; k += kRowLaw * W) {
            unsigned int u[kRowLaw];
            float4 p[kRowLaw], v[kRowLaw];
#pragma unroll
            for (int q = 0; q < kRowLaw; ++q) {
                u[q] = k + q * W < nh ? list[k + q * W] : B.self;
                p[q] = __ldg(&cpos[u[q]]);
                v[q] = __ldg(&cvel[u[q]]);
            }
#pragma unroll
            for (int q = 0; q < kRowLaw; ++q) {
                if (u[q] == B.self) continue;
                const bool jfe = DIRECT ? (int)u[q] < R.nfe : __float_as_int(p[q].w) < sw;
                const float dx = p[q].x - B.pi.x, dy = p[q].y - B.pi.y, dz = p[q].z - B.pi.z;
                const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
                const float c = contact_coef(select_row(jfe, row_fe, row_si), tab.sep_test, dx, dy,
                                             dz, r2, B.vi, v[q]) * inv_unit;
                fix_add3(acc, c, dx, dy, dz, r2);
            }
        }
        __syncwarp();  // the list is read before it refills
        nh = 0;
    };

    unsigned int incl = cnt;
    if (!DIRECT) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
    }
    const unsigned int total = DIRECT ? cnt : __shfl_sync(0xffffffffu, incl, 31), excl = incl - cnt;
    row_fetch<DIRECT>(sm, cpos, 0, 0u, total, beg, excl, lane);
    int buf = 0;
    for (unsigned int base = 0; base < total; base += kRowStage, buf ^= 1) {
        if (base + kRowStage < total) {
            row_fetch<DIRECT>(sm, cpos, buf ^ 1, base + kRowStage, total, beg, excl, lane);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const int n = (int)min((unsigned int)kRowStage, total - base);
        for (int t0 = way; t0 < n + way; t0 += 4 * W) {
            bool hit[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const float4 pj = sm.stage[buf][t0 + v * W];  // < kRowStage: 4 W divides it
                const float dx = pj.x - px, dy = pj.y - B.pi.y, dz = pj.z - B.pi.z;
                const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
                hit[v] = r2 < 1.0f;
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const unsigned int m = __ballot_sync(0xffffffffu, hit[v]);
                if (hit[v]) list[nh + __popc(m & below)] = sm.slot[buf][t0 + v * W];
                nh += __popc(m & mine);
            }
            if (__any_sync(0xffffffffu, nh > full)) drain();
        }
        __syncwarp();  // the batch is tested before its buffer refills
    }
    drain();
    fix_fold(acc);
    long long a[3] = {acc.x, acc.y, acc.z};
    for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
        for (int d = 0; d < 3; ++d) a[d] += __shfl_xor_sync(0xffffffffu, a[d], o);
    if (B.i >= 0 && way < 3) {
        long long *const d = &delta[3 * (size_t)B.i + way];
        const long long v = way == 0 ? a[0] : way == 1 ? a[1] : a[2];
        if (!add) *d = v;
        else if (v) atomicAdd(reinterpret_cast<unsigned long long *>(d), (unsigned long long)v);
    }
}

// A lone body with at most 32 candidates, one to a lane, straight from memory: no
// staging, no list.  [beg, beg + cnt): the lane's range, excl the candidates before it.
__device__ __forceinline__ void row_few(const GridView &g, long long *__restrict__ delta,
                                        const LaunchTable &tab, const RunDev &R, const PairDev &P,
                                        unsigned int self, unsigned int beg, unsigned int cnt,
                                        unsigned int total, bool add, int lane)
{
    unsigned int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const unsigned int excl = incl - cnt;
    int src = 0;  // the lane whose range holds candidate `lane`: the last one with excl <= it
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const unsigned int e = __shfl_sync(0xffffffffu, excl, (src + step) & 31);
        if (src + step < 32 && e <= (unsigned int)lane) src += step;
    }
    const unsigned int slot = __shfl_sync(0xffffffffu, beg - excl, src) + (unsigned int)lane;
    const float4 pi = __ldg(&g.spos[self]);
    float4 p = make_float4(__int_as_float(0x7fffffff), 0.f, 0.f, 0.f);
    if ((unsigned int)lane < total) p = __ldg(&g.spos[slot]);
    const float dx = p.x - pi.x, dy = p.y - pi.y, dz = p.z - pi.z;
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    const bool hit = r2 < 1.0f && slot != self;
    FixSum3 acc;
    fix_zero(acc);
    if (hit) {
        const int sw = R.offset + R.nfe;
        const PairRow row = pair_row(P, __float_as_int(pi.w) < sw, __float_as_int(p.w) < sw);
        const float c = contact_coef(row, tab.sep_test, dx, dy, dz, r2, __ldg(&g.svel[self]),
                                     __ldg(&g.svel[slot])) * P.inv_unit;
        fix_add3<false>(acc, c, dx, dy, dz, r2);
        fix_fold(acc);
    }
    long long a[3] = {0, 0, 0};
    for (unsigned int m = __ballot_sync(0xffffffffu, hit); m; m &= m - 1u) {
        const int l = __ffs(m) - 1;
        a[0] += __shfl_sync(0xffffffffu, acc.x, l);
        a[1] += __shfl_sync(0xffffffffu, acc.y, l);
        a[2] += __shfl_sync(0xffffffffu, acc.z, l);
    }
    if (lane < 3) {
        long long *const d = &delta[3 * (size_t)__float_as_int(pi.w) + lane];
        const long long v = lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
        if (!add) *d = v;
        else if (v) atomicAdd(reinterpret_cast<unsigned long long *>(d), (unsigned long long)v);
    }
}

// Runs without a grid: kDirectBodies bodies from `first` on, every body of the
// run a candidate.
__device__ __forceinline__ void row_direct(RowSmem &sm, const float4 *__restrict__ pos,
                                           const float4 *__restrict__ vel,
                                           long long *__restrict__ delta, const LaunchTable &tab,
                                           const RunDev &R, int first, int lane)
{
    constexpr int kWlog = kDirectBodies == 1 ? 5 : kDirectBodies == 2 ? 4 : 3;
    static_assert(kDirectBodies == 1 || kDirectBodies == 2 || kDirectBodies == 4, "lanes per body");
    const int k = first + (lane >> kWlog);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    RowBody B;
    B.i = k < R.n ? R.offset + k : -1;
    B.self = (unsigned int)k;
    B.pi = k < R.n ? __ldg(&pos[B.i]) : z;
    B.vi = k < R.n ? __ldg(&vel[B.i]) : z;
    row_group<true>(sm, pos + R.offset, vel + R.offset, delta, tab, R, tab.params[R.param], B, kWlog,
                    0u, (unsigned int)R.n, false, lane);
}

// Runs with a grid: kRowBodies (8) consecutive slots.  Slots run along x, so
// the bodies of one cell row (same y and z cell) a few cells apart share their
// candidates: nine rows' slots over the bodies' x range and one cell to either
// side, each one contiguous range (two where the torus wraps).  FEW: with row_few.
template <bool FEW>
__device__ __forceinline__ void row_slots(RowSmem &sm, const GridView &g,
                                          long long *__restrict__ delta, const LaunchTable &tab,
                                          const RunDev &R, unsigned int run, int first, int lane)
{
    const bool crowds = has_crowds(g.ctr, run);
    const PairDev &P = tab.params[R.param];
    const Torus T = torus_of(R);
    const unsigned int dmin = (unsigned int)tab.dense_min;
    // lane k < 8 has slot k; tiled bodies are left to contact_tile_kernel
    const bool valid = lane < kRowBodies && first + lane < R.n;
    const unsigned int slot = (unsigned int)(R.gslot + first + lane);
    const int3 c = valid ? cell_of(__ldg(&g.spos[slot])) : make_int3(0, 0, 0);
    const unsigned int key = bucket_of(T, c.x, c.y, c.z);
    const bool in = valid && !(crowds && cell_tiled(g, key, c, dmin));
    // a body joins the one before it where their x ranges meet; a group is a
    // chain of joined bodies
    const int bx = __shfl_up_sync(0xffffffffu, c.x, 1), by = __shfl_up_sync(0xffffffffu, c.y, 1),
              bz = __shfl_up_sync(0xffffffffu, c.z, 1);
    unsigned int rest = __ballot_sync(0xffffffffu, in);
    const unsigned int joined = __ballot_sync(
        0xffffffffu, in && lane > 0 && ((rest >> (lane - 1)) & 1u) && c.y == by && c.z == bz &&
                         c.x >= bx && c.x <= bx + 3);
    while (rest) {
        const int src = __ffs(rest) - 1;
        int n = __ffs(~(joined >> src >> 1));  // bodies of the group (8 at most)
        const int xlo = __shfl_sync(0xffffffffu, c.x, src) - 1,
                  width = __shfl_sync(0xffffffffu, c.x, src + n - 1) + 2 - xlo,
                  gy = __shfl_sync(0xffffffffu, c.y, src), gz = __shfl_sync(0xffffffffu, c.z, src);
        unsigned int beg = 0u, end = 0u;
        bool crowd = false;
        if (lane < 18) {  // the two pieces of each of the nine rows
            const int r = lane >> 1, side = T.xm + 1;
            const unsigned int base = row_of(T, gy + r % 3 - 1, gz + r / 3 - 1);
            const int a = width >= side ? 0 : xlo & T.xm, z = a + min(width, side);
            const int lo = lane & 1 ? 0 : a, hi = lane & 1 ? z - side : min(z, side);
            if (hi > lo) {
                beg = __ldg(&g.start[base + lo]);
                end = __ldg(&g.start[base + hi]);
            }
            if (crowds && end - beg >= dense_lo(dmin))
                for (int x = lo; x < hi; ++x)
                    crowd |= bucket_size(g.start, base + x) >= dense_lo(dmin) && g.state[base + x];
        }
        if (__any_sync(0xffffffffu, crowd)) {
            // Next to a tiled bucket; a tiled neighbour cell's items give both
            // sides of its pairs.  The first cell's bodies alone, its other
            // neighbours one to a lane.
            n = min(n, __ffs(~(__ballot_sync(0xffffffffu, in && c.x == xlo + 1) >> src)) - 1);
            beg = end = 0u;
            if (lane < 27) {
                const int3 d = make_int3(xlo + lane % 3, gy + lane / 3 % 3 - 1, gz + lane / 9 - 1);
                const unsigned int b = bucket_of(T, d.x, d.y, d.z);
                if (!cell_tiled(g, b, d, dmin)) {
                    beg = __ldg(&g.start[b]);
                    end = __ldg(&g.start[b + 1]);
                }
            }
        }
        rest &= ~(((1u << n) - 1u) << src);
        if (FEW && n == 1) {
            const unsigned int total = __reduce_add_sync(0xffffffffu, end - beg);
            if (total <= 32u) {
                row_few(g, delta, tab, R, P, (unsigned int)(R.gslot + first + src), beg, end - beg, total,
                        crowds, lane);
                continue;
            }
        }
        // the lanes among the group's bodies
        const int wlog = n > 4 ? 2 : n > 2 ? 3 : n > 1 ? 4 : 5;
        const int k = lane >> wlog;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        RowBody B;
        B.self = (unsigned int)(R.gslot + first + src + k);
        B.pi = k < n ? __ldg(&g.spos[B.self]) : z;
        B.vi = k < n ? __ldg(&g.svel[B.self]) : z;
        B.i = k < n ? __float_as_int(B.pi.w) : -1;
        row_group<false>(sm, g.spos, g.svel, delta, tab, R, P, B, wlog, beg, end - beg, crowds, lane);
    }
}

// Row-path CTA (one warp) w of the table: bodies of one run.
template <bool FEW>
__device__ __forceinline__ void contact_rows(RowSmem &sm, const float4 *__restrict__ pos,
                                             const float4 *__restrict__ vel, const GridView &g,
                                             long long *__restrict__ delta, const LaunchTable &tab,
                                             int w)
{
    int lo = 0, hi = tab.nruns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tab.runs[mid].row_start <= w) lo = mid;
        else hi = mid - 1;
    }
    const RunDev &R = tab.runs[lo];
    const int first = (w - R.row_start) * (R.glog ? kRowBodies : kDirectBodies);
    if (R.glog) row_slots<FEW>(sm, g, delta, tab, R, lo, first, threadIdx.x);
    else row_direct(sm, pos, vel, delta, tab, R, first, threadIdx.x);
}

}  // namespace gi
