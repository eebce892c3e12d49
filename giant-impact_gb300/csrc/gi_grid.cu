// gi_grid.cu -- contact forces through a cell grid.
//
// The all-pairs kernel evaluates far-field gravity for every pair with r2
// clamped at one diameter.  The pairs inside one diameter (r2 < 1, the only
// ones where the reference law departs from gravity) are handled here:
//
//   1. grid: every body gets the cell floor(x), floor(y), floor(z) (cell size
//      D = 1, so two bodies within r < 1 are in the same or adjacent cells).
//      Each run has 2^k buckets of its own, a torus of cells: the low bits of
//      the three cell coordinates, x fastest.  Cells next to each other along
//      x are neighbouring buckets, and no two cells closer than the torus is
//      wide share one.  A counting sort lists the bodies bucket by bucket as
//      slots, with their state and index (spos.w).
//   2. contact law: for each j of the same run with FP32 r2 < 1, the pass
//      adds the contact force of the reference law minus the clamped
//      far-field term the all-pairs pass added for that pair.  Band and K/KR
//      choices use the reference's FP32 r2 and dp.dv (bit-identical
//      decisions).
//   3. each pair's correction is evaluated in FP32, rounded to an integer
//      of the fixed point (unit = (2 Gmax + Kmax) 2^-40 per pair table) and
//      summed in 64 bits: integer adds are exact, so the sum does not depend
//      on the order in which bodies landed in buckets or lanes found them,
//      and the result is bit-reproducible.
// The all-pairs epilogue adds the correction before its single rounding.
//
// Two passes share the bodies.  contact_row_kernel takes a few consecutive
// slots per warp, an ordinary body's path.  The bodies of a crowded bucket's
// majority cell (gi_options.dense_min of them, 128 by default, or a quarter of
// that next to such a cell; e.g. an interpenetrating collision remnant with
// thousands of contacts per body) are sorted by sub-cell and go through
// contact_tile_kernel: a work item is (bucket, neighbour bucket, chunk of 128 of
// its bodies); its CTA stages the neighbour bucket in shared memory 128 bodies at
// a time, evaluates the law on the hits only, or on whole blocks of pairs that are
// mostly hits, and a pair of two dense cells is evaluated once for both bodies.
// The candidate sets, the pair law and the fixed-point terms are the same on both
// paths and integer addition is exact, so the corrections are bit-identical
// whichever path a body takes.
//
// Short runs (kDirectMax) need no grid where a table has few: every body of the run
// is a candidate.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>

#include "gi_contact.cuh"

namespace cg = cooperative_groups;

namespace gi {

__device__ __forceinline__ void put_body(const float4 *__restrict__ pos,
                                         const float4 *__restrict__ vel, int i, unsigned int slot,
                                         float4 *__restrict__ spos, float4 *__restrict__ svel)
{
    float4 p = __ldg(&pos[i]);
    p.w = __int_as_float(i);
    spos[slot] = p;
    svel[slot] = __ldg(&vel[i]);
}

// Clears the corrections of a run with candidates for the tiled path (other
// runs' are stored by the row path): thread t of nt.
__device__ __forceinline__ void clear_delta(long long *__restrict__ delta, const RunDev &R, int t,
                                            int nt)
{
    long long *const d = delta + 3 * (size_t)R.offset;
    for (long long k = t; k < 3 * (long long)R.n; k += nt) d[k] = 0;
}

// Pair form of fix_add3 for an unordered pair evaluated once: adds
// round(c d) to body i's sums and -round(c d), exactly the term body j's own
// evaluation would give (dp and dv change sign exactly, c is symmetric, and
// rounding to nearest even is odd-symmetric), to the shared sums js[.][k]
// of j's staged slot: true values mod 2^32, hi in js[0..2], lo in js[3..5].
// A term out of the split's range goes to j's global sums directly.  The
// caller folds (at most kFixFold terms between its folds).
__device__ __forceinline__ void fix_add3_pair(FixSum3 &a, unsigned int (*js)[128], int k,
                                              long long *dj, float c, float dx, float dy, float dz,
                                              float r2)
{
    const float2 txy = __fmul2_rn(make_float2(c, c), make_float2(dx, dy));
    const float tz = __fmul_rn(c, dz);
    if (fix_in_range(r2)) {
        const float2 s = __fadd2_rn(txy, make_float2(kFixM, kFixM));
        const float2 lo = __ffma2_rn(__fadd2_rn(s, make_float2(-kFixM, -kFixM)),
                                     make_float2(-1.0f, -1.0f), txy);
        const float2 l = __fadd2_rn(lo, make_float2(kFixC, kFixC));
        const float sz = __fadd_rn(tz, kFixM);
        const float lz = __fadd_rn(__fsub_rn(tz, __fsub_rn(sz, kFixM)), kFixC);
        const unsigned int sb[3] = {__float_as_uint(s.x), __float_as_uint(s.y), __float_as_uint(sz)};
        const unsigned int lb[3] = {__float_as_uint(l.x), __float_as_uint(l.y), __float_as_uint(lz)};
        a.hx += sb[0]; a.hy += sb[1]; a.hz += sb[2];
        a.lx += lb[0]; a.ly += lb[1]; a.lz += lb[2];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            atomicAdd(&js[d][k], __float_as_uint(kFixM) - sb[d]);
            atomicAdd(&js[3 + d][k], __float_as_uint(kFixC) - lb[d]);
        }
        ++a.n;
    } else {
        const long long vx = __float2ll_rn(txy.x), vy = __float2ll_rn(txy.y),
                        vz = __float2ll_rn(tz);
        a.x += vx;
        a.y += vy;
        a.z += vz;
        unsigned long long *d = reinterpret_cast<unsigned long long *>(dj);
        atomicAdd(d + 0, 0ull - (unsigned long long)vx);
        atomicAdd(d + 1, 0ull - (unsigned long long)vy);
        atomicAdd(d + 2, 0ull - (unsigned long long)vz);
    }
}

// Adds the shared j-side sums of slot t to body j's correction and clears them.
__device__ __forceinline__ void flush_slot(unsigned int (*js)[128], int t, int j, long long *delta)
{
    long long v[3];
    bool any = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        v[d] = (long long)(int)js[d][t] * (1ll << 23) + (int)js[3 + d][t];
        any |= v[d] != 0;
        js[d][t] = 0u;
        js[3 + d][t] = 0u;
    }
    if (any) {
        unsigned long long *p = reinterpret_cast<unsigned long long *>(delta + 3 * (size_t)j);
        atomicAdd(p + 0, (unsigned long long)v[0]);
        atomicAdd(p + 1, (unsigned long long)v[1]);
        atomicAdd(p + 2, (unsigned long long)v[2]);
    }
}

// The row path on its own (beside the one-sided far field); the paired far
// field's kernel takes the same CTAs itself.
__global__ void __maxnreg__(96)
contact_row_kernel(const float4 *__restrict__ pos, const float4 *__restrict__ vel, const GridView g,
                   long long *__restrict__ delta, const __grid_constant__ LaunchTable tab)
{
    __shared__ RowSmem sm;
    contact_rows<true>(sm, pos, vel, g, delta, tab, blockIdx.x);
}
// Work item of the tiled path, self-contained so that the tile kernel reads
// it in one load, with no hop through the bucket bounds:
//   x = first slot of the chunk of (up to) 128 bodies of bucket b,
//   y = first slot of the neighbour bucket nb to stage (the chunk's own
//       first slot when nb == b, else the start of nb),
//   z = end of nb,
//   w = run | cost class << 8 | tiled << 12 | self << 13 | bodies of the
//       chunk << 16.
// The cost class is the number of 128-body tiles the item stages, minus
// one, capped at kItemClasses - 1; tiled: nb's tiled bodies (dpos), else all
// of its bodies (spos); self: nb == b.
// (kItemClasses lives in gi_internal.h.)

// Sub-cell of a body inside its unit cell: 4 x 4 x 4 sub-cells of D/4,
// numbered in Morton order.
__device__ __forceinline__ unsigned int subcell_of(float4 p)
{
    const auto q = [](float x) {
        const int s = (int)((x - floorf(x)) * 4.0f);  // NaN -> 0
        return (unsigned int)min(max(s, 0), 3);
    };
    const unsigned int sx = q(p.x), sy = q(p.y), sz = q(p.z);
    return (sx & 1u) | (sy & 1u) << 1 | (sz & 1u) << 2 | (sx >> 1) << 3 | (sy >> 1) << 4 |
           (sz >> 1) << 5;
}

// One warp, one candidate bucket b: how many of its bodies are tiled (state, 0
// for none), and copies them to the front of the bucket's dpos / dvel, ordered by sub-cell
// (counting sort in cnt[64]), so that the 32 bodies of a warp, and the 32 of a
// staged block, sit close together.  The slots stay as they are for the row
// path.  Order within a bucket is free: the contact sums are exact integer
// sums.
__device__ __forceinline__ bool dense_prep(const Torus &T, const GridWork &g, unsigned int b,
                                           unsigned int dmin, unsigned int *cnt, unsigned int lane)
{
    int3 m;
    const unsigned int t = bucket_tiled(T, g.start, g.spos, b, dmin, (int)lane, m);
    if (lane == 0u) g.state[b] = t;
    if (!t) return false;  // the same in the whole warp
    const auto main = [&](float4 p) {
        const int3 c = cell_of(p);
        return c.x == m.x && c.y == m.y && c.z == m.z;
    };
    const unsigned int beg = g.start[b], end = g.start[b + 1];
    __syncwarp();
    cnt[lane] = cnt[lane + 32u] = 0u;
    __syncwarp();
    for (unsigned int u0 = beg + lane; u0 < end; u0 += 128u) {
        float4 p[4];  // four loads in flight
#pragma unroll
        for (int v = 0; v < 4; ++v) p[v] = g.spos[min(u0 + 32u * v, end - 1u)];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            if (u0 + 32u * v >= end || !main(p[v])) continue;
            atomicAdd(&cnt[subcell_of(p[v])], 1u);
        }
    }
    __syncwarp();
    const unsigned int c0 = cnt[2u * lane], c1 = cnt[2u * lane + 1u];
    unsigned int incl = c0 + c1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += v;
    }
    __syncwarp();
    cnt[2u * lane] = incl - c0 - c1;
    cnt[2u * lane + 1u] = incl - c1;
    __syncwarp();
    for (unsigned int u0 = beg + lane; u0 < end; u0 += 128u) {
        float4 p[4], q[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            p[v] = g.spos[min(u0 + 32u * v, end - 1u)];
            q[v] = g.svel[min(u0 + 32u * v, end - 1u)];
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            if (u0 + 32u * v >= end || !main(p[v])) continue;
            const unsigned int slot = beg + atomicAdd(&cnt[subcell_of(p[v])], 1u);
            g.dpos[slot] = p[v];
            g.dvel[slot] = q[v];
        }
    }
    __syncwarp();
    return true;
}

// One warp, one tiled bucket b of run `run`: an item per (chunk of 128 of its
// tiled bodies, non-empty neighbour bucket nb).  Lanes 0..26 look up the 27
// neighbour buckets at once.  Items evaluate each contact pair once for both
// bodies, so a pair of tiled buckets is listed once, from the lower bucket
// number (nb >= b), with nb's tiled bodies (its others are far away); where
// the neighbour cell is not nb's tiled one, the item takes all of nb, and the
// row path passes over b.  take(cls, n) is called by one lane per cost class
// for n items and returns the place of the first (one counter update per
// class, not per item); put(place, item) stores one.
template <class Take, class Put>
__device__ __forceinline__ void dense_items(const Torus &T, const GridWork &g, unsigned int b,
                                            unsigned int run, unsigned int dmin, unsigned int lane,
                                            const Take &take, const Put &put)
{
    const unsigned int beg = g.start[b], cnt = g.state[b], nch = (cnt + 127u) / 128u;
    // the cell: the first tiled body's
    const int3 c = cell_of(g.dpos[beg]);
    unsigned int nbq = 0u, nbeg = 0u, nend = 0u;
    bool keep = false, both = false;
    if (lane < 27u) {
        nbq = bucket_of(T, c.x + (int)(lane % 3u) - 1, c.y + (int)(lane / 3u % 3u) - 1,
                        c.z + (int)(lane / 9u) - 1);
        nbeg = g.start[nbq];
        nend = g.start[nbq + 1];
        if (nend - nbeg >= dense_lo(dmin)) {  // states are written for candidates alone
            const unsigned int t = g.state[nbq];
            if (t) {  // are its tiled bodies the neighbour cell's?
                const int3 d = cell_of(g.dpos[nbeg]);
                both = d.x == c.x + (int)(lane % 3u) - 1 && d.y == c.y + (int)(lane / 3u % 3u) - 1 &&
                       d.z == c.z + (int)(lane / 9u) - 1;
            }
            if (both) nend = nbeg + t;
        }
        keep = nend > nbeg && nbq != b && !(both && nbq < b);
    }
    const auto item = [&](unsigned int s0, unsigned int first, unsigned int end, unsigned int cls,
                          unsigned int flags) {
        return make_uint4(s0, first, end, run | cls << 8 | flags << 12 | min(128u, beg + cnt - s0) << 16);
    };
    // neighbours: nch items of one class each
    const unsigned int cls = keep ? min((nend - nbeg + 127u) / 128u, kItemClasses) - 1u : ~0u;
    const unsigned int same = __match_any_sync(0xffffffffu, cls);
    const int leader = __ffs(same) - 1;
    unsigned int at = 0u;
    if (keep && (int)lane == leader) at = take(cls, nch * __popc(same));
    at = __shfl_sync(0xffffffffu, at, leader) + nch * __popc(same & ((1u << lane) - 1u));
    if (keep)
        for (unsigned int k = 0; k < nch; ++k)
            put(at + k, item(beg + 128u * k, nbeg, nend, cls, both ? 1u : 0u));
    // the bucket with itself: chunk k takes the tiles from its own on
    for (unsigned int k = lane; k < nch; k += 32u) {
        const unsigned int s0 = beg + 128u * k;
        const unsigned int q = min(nch - k, kItemClasses) - 1u;
        put(take(q, 1u), item(s0, s0, beg + cnt, q, 3u));
    }
}

// The grid of one run by one thread-block cluster: counts in the distributed
// shared memory (each CTA holds an equal range of the buckets), scanned there,
// then the bodies written to their slots, and where there are crowded buckets
// the tiled path's copies and items, in cost-class order (most tiles first),
// made by the cluster's warps.  Cluster barriers instead of eleven launches: a
// launch that depends on the one before it costs 2 to 4 us, which is what
// short runs spent their step on.  One SM's bandwidth per CTA bounds it: runs
// of kClusterMax bodies or more, whose step takes milliseconds, take the
// grid-wide kernels below.  (A CTA's counts take 32 KB at most: 2^k <= 2 n
// buckets.)
constexpr int kClusterItems = 8;  // bodies per thread, at most
constexpr int kClusterSmall = 8, kClusterLarge = 16;
static_assert(kClusterSmallMax == kClusterSmall * 1024 * kClusterItems, "runs of the small cluster");
constexpr int kClusterMax = kClusterLarge * 1024 * kClusterItems;       // 131,072

// Counters of a run's crowded buckets, in the cluster's first CTA.
struct ClusterCounts {
    unsigned int cand, tiled, items, base;
    unsigned int cls[kItemClasses], fill[kItemClasses];
};

__global__ void __launch_bounds__(1024)
grid_cluster_kernel(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                    const __grid_constant__ LaunchTable tab, const GridWork g, long long *delta,
                    unsigned int *ctr)
{
    extern __shared__ unsigned int cnt[];  // this CTA's buckets; 64 words per warp at the end
    __shared__ unsigned int wsum[32];
    __shared__ unsigned int total, before;
    __shared__ ClusterCounts cc;
    const RunDev &R = tab.runs[blockIdx.y];
    if (R.glog == 0) return;  // the whole cluster: a run without a grid
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x, ctas = gridDim.x;
    const int plog = R.glog - (ctas == kClusterLarge ? 4 : 3), per = 1 << plog;
    const unsigned int dmin = (unsigned int)tab.dense_min, dlo = dense_lo(dmin);
    // the run's part of the candidate and tiled lists
    uint2 *const cand = g.cand + R.gslot / kDenseFloor + blockIdx.y,
          *const tiled = g.tiled + R.gslot / kDenseFloor + blockIdx.y;
    ClusterCounts *const c0 = cluster.map_shared_rank(&cc, 0);
    for (int u = tid; u < per; u += 1024) cnt[u] = 0u;
    if (tid < (int)(sizeof(ClusterCounts) / 4)) reinterpret_cast<unsigned int *>(&cc)[tid] = 0u;
    cluster.sync();
    const Torus T = torus_of(R);
    // all loads of a thread in flight together, then all its counts
    unsigned int key[kClusterItems], rk[kClusterItems];
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it) {
        const int k = (it * ctas + rank) * 1024 + tid;
        key[it] = 0u;
        if (k < R.n) {
            const int3 c = cell_of(__ldg(&pos[R.offset + k]));
            key[it] = bucket_of(T, c.x, c.y, c.z) - T.base;
        }
    }
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it)
        if ((it * ctas + rank) * 1024 + tid < R.n)
            rk[it] = atomicAdd(cluster.map_shared_rank(cnt, key[it] >> plog) + (key[it] & (per - 1)), 1u);
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it)
        if ((it * ctas + rank) * 1024 + tid < R.n && rk[it] == dlo - 1u)
            cand[atomicAdd(&c0->cand, 1u)] = make_uint2(T.base + key[it], 0u);
    cluster.sync();
    // exclusive scan of this CTA's counts: e consecutive ones per thread
    const int e = per > 1024 ? per >> 10 : 1;
    unsigned int sum = 0u;
    for (int q = 0; q < e; ++q) sum += tid * e + q < per ? cnt[tid * e + q] : 0u;
    unsigned int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned int w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += v;
        }
        wsum[lane] = w;
        if (lane == 31) total = w;
    }
    cluster.sync();
    if (warp == 0) {
        unsigned int t = lane < rank ? *cluster.map_shared_rank(&total, lane) : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) before = t;
    }
    __syncthreads();
    unsigned int at = (unsigned int)R.gslot + before + (warp ? wsum[warp - 1] : 0u) + incl - sum;
    for (int q = 0; q < e; ++q) {
        const int u = tid * e + q;
        if (u >= per) break;
        const unsigned int c = cnt[u];
        cnt[u] = at;
        g.start[T.base + rank * per + u] = at;
        at += c;
    }
    // the end of the last bucket (the next run writes the same value there)
    if (rank == ctas - 1 && tid == 0) g.start[T.base + ctas * per] = (unsigned int)(R.gslot + R.n);
    cluster.sync();
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it)
        if ((it * ctas + rank) * 1024 + tid < R.n)
            rk[it] += *(cluster.map_shared_rank(cnt, key[it] >> plog) + (key[it] & (per - 1)));
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it) {
        const int k = (it * ctas + rank) * 1024 + tid;
        if (k < R.n) put_body(pos, vel, R.offset + k, rk[it], g.spos, g.svel);
    }
    cluster.sync();  // the slots are written, the counts read
    const unsigned int ncand = c0->cand;
    const unsigned int gw = (unsigned int)(rank * 32 + warp), nw = (unsigned int)ctas * 32u;
    if (ncand != 0u) {
        clear_delta(delta, R, rank * 1024 + tid, ctas * 1024);
        if (rank == 0 && tid == 0) set_crowds(ctr, blockIdx.y);
    }
    for (unsigned int w = gw; w < ncand; w += nw) {
        const unsigned int b = cand[w].x;
        if (!dense_prep(T, g, b, dmin, cnt + 64 * warp, (unsigned int)lane)) continue;
        if (lane == 0) tiled[atomicAdd(&c0->tiled, 1u)] = make_uint2(b, 0u);
    }
    cluster.sync();  // no CTA leaves before its counters are read
    if (ncand == 0u) return;
    const unsigned int ntiled = c0->tiled;
    for (unsigned int w = gw; w < ntiled; w += nw)
        dense_items(T, g, tiled[w].x, blockIdx.y, dmin, (unsigned int)lane,
                    [&](unsigned int cls, unsigned int n) { return atomicAdd(&c0->cls[cls], n); },
                    [](unsigned int, uint4) {});
    cluster.sync();
    if (rank == 0 && tid == 0) {
        unsigned int n = 0u;
        for (int c = (int)kItemClasses - 1; c >= 0; --c) {
            cc.fill[c] = n;
            n += cc.cls[c];
        }
        cc.base = n ? atomicAdd(&ctr[kCtrItems], n) : 0u;
    }
    cluster.sync();
    const unsigned int base = c0->base;
    for (unsigned int w = gw; w < ntiled; w += nw)
        dense_items(T, g, tiled[w].x, blockIdx.y, dmin, (unsigned int)lane,
                    [&](unsigned int cls, unsigned int n) { return atomicAdd(&c0->fill[cls], n); },
                    [&](unsigned int at, uint4 it) { g.items[base + at] = it; });
    cluster.sync();  // the first CTA stays until its counters are done with
}

// Grid-wide form of the same (runs of any size).  Bucket of every body of
// every run, and its rank there; counts of buckets.
__global__ void __launch_bounds__(256)
grid_keys(const float4 *__restrict__ pos, const __grid_constant__ LaunchTable tab, const GridWork g,
          unsigned int *__restrict__ ctr)
{
    const RunDev &R = tab.runs[blockIdx.y];
    if (R.glog == 0) return;
    const Torus T = torus_of(R);
    const unsigned int dlo = dense_lo((unsigned int)tab.dense_min);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < R.n; k += gridDim.x * blockDim.x) {
        const int i = R.offset + k;
        const int3 c = cell_of(pos[i]);
        const unsigned int b = bucket_of(T, c.x, c.y, c.z);
        const unsigned int r = atomicAdd(&g.start[b], 1u);  // counts until they are scanned
        g.keys[i] = b;
        g.ranks[i] = r;
        if (r == dlo - 1u) {
            g.cand[atomicAdd(&ctr[kCtrCand], 1u)] = make_uint2(b, blockIdx.y);
            set_crowds(ctr, blockIdx.y);
        }
    }
}

// Exclusive scan of a[0..m), m <= 1024 * 8192 + 1, in place.
__global__ void __launch_bounds__(1024) scan_blocks(unsigned int *__restrict__ a, int m,
                                                    unsigned int *__restrict__ sums)
{
    __shared__ unsigned int sh[1024];
    const int i = blockIdx.x * 1024 + threadIdx.x;
    const unsigned int v = i < m ? a[i] : 0u;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned int t = threadIdx.x >= o ? sh[threadIdx.x - o] : 0u;
        __syncthreads();
        sh[threadIdx.x] += t;
        __syncthreads();
    }
    if (i < m) a[i] = sh[threadIdx.x] - v;
    if (threadIdx.x == 1023) sums[blockIdx.x] = sh[1023];
}

// Exclusive scan of nb <= 9216 block totals: 9 per thread, then across threads.
__global__ void __launch_bounds__(1024) scan_sums(unsigned int *__restrict__ sums, int nb)
{
    __shared__ unsigned int sh[1024];
    unsigned int loc[9];
    unsigned int tot = 0u;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int i = threadIdx.x * 9 + q;
        loc[q] = i < nb ? sums[i] : 0u;
        tot += loc[q];
    }
    sh[threadIdx.x] = tot;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned int t = threadIdx.x >= o ? sh[threadIdx.x - o] : 0u;
        __syncthreads();
        sh[threadIdx.x] += t;
        __syncthreads();
    }
    unsigned int run = sh[threadIdx.x] - tot;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int i = threadIdx.x * 9 + q;
        if (i < nb) sums[i] = run;
        run += loc[q];
    }
}

__global__ void __launch_bounds__(1024) scan_add(unsigned int *__restrict__ a, int m,
                                                 const unsigned int *__restrict__ sums)
{
    const int i = blockIdx.x * 1024 + threadIdx.x;
    if (i < m) a[i] += sums[blockIdx.x];
}

__global__ void __launch_bounds__(256)
grid_scatter(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
             const __grid_constant__ LaunchTable tab, const GridWork g,
             long long *__restrict__ delta, const unsigned int *__restrict__ ctr)
{
    const RunDev &R = tab.runs[blockIdx.y];
    if (R.glog == 0) return;
    if (has_crowds(ctr, blockIdx.y))
        clear_delta(delta, R, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < R.n; k += gridDim.x * blockDim.x) {
        const int i = R.offset + k;
        put_body(pos, vel, i, g.start[g.keys[i]] + g.ranks[i], g.spos, g.svel);
    }
}

// The crowded buckets of a grid-wide build, one warp per candidate, then one
// per tiled bucket, then the items into cost-class order.
__global__ void __launch_bounds__(64)
dense_prep_kernel(const __grid_constant__ LaunchTable tab, const GridWork g, unsigned int *ctr)
{
    __shared__ unsigned int cnt[2][64];
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned int total = ctr[kCtrCand];
    for (unsigned int w = 2u * blockIdx.x + warp; w < total; w += 2u * gridDim.x) {
        const uint2 cb = g.cand[w];
        if (dense_prep(torus_of(tab.runs[cb.y]), g, cb.x, (unsigned int)tab.dense_min,
                       cnt[warp], lane) && lane == 0u)
            g.tiled[atomicAdd(&ctr[kCtrTiled], 1u)] = cb;
    }
}

__global__ void __launch_bounds__(64)
dense_items_kernel(const __grid_constant__ LaunchTable tab, const GridWork g, unsigned int *ctr)
{
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned int total = ctr[kCtrTiled];
    for (unsigned int w = 2u * blockIdx.x + warp; w < total; w += 2u * gridDim.x) {
        const uint2 cb = g.tiled[w];
        dense_items(torus_of(tab.runs[cb.y]), g, cb.x, cb.y, (unsigned int)tab.dense_min, lane,
                    [&](unsigned int cls, unsigned int n) {
                        atomicAdd(&ctr[kCtrClass + cls], n);
                        return atomicAdd(&ctr[kCtrItems], n);
                    },
                    [&](unsigned int at, uint4 it) { g.raw[at] = it; });
    }
}

// The items, ordered by cost class, most tiles first (a counting
// sort over the classes), so that the tile kernel's queue hands out the
// longest items first and its CTAs finish together.  Order within a class
// is arbitrary; the sums do not depend on it.
__global__ void __launch_bounds__(256)
dense_order_kernel(const uint4 *__restrict__ raw, unsigned int *__restrict__ ctr,
                   uint4 *__restrict__ items)
{
    __shared__ unsigned int base[kItemClasses];
    if (threadIdx.x < kItemClasses) {
        unsigned int b = 0;
        for (unsigned int c = kItemClasses - 1; c > threadIdx.x; --c) b += ctr[kCtrClass + c];
        base[threadIdx.x] = b;
    }
    __syncthreads();
    const unsigned int total = ctr[kCtrItems];
    for (unsigned int w = blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += gridDim.x * blockDim.x) {
        const uint4 it = raw[w];
        const unsigned int cls = (it.w >> 8) & (kItemClasses - 1u);
        items[base[cls] + atomicAdd(&ctr[kCtrFill + cls], 1u)] = it;
    }
}

// Bounding box of the non-empty lanes of a warp (lo = +inf, hi = -inf for
// an empty lane), returned to every lane.  fminf / fmaxf drop NaN.
__device__ __forceinline__ void warp_box(float3 &lo, float3 &hi)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
        hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
        hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
    }
}

// Lower bound, in the rounding of the pair filter, of the FP32 r2 of every
// pair between two boxes.  Per axis, |fl(pj - pi)| >= fl(gap) because
// rounding is monotone, and the sum of squares below has the form of the
// filter's, so a result >= 1 proves that no pair passes r2 < 1.  A NaN term
// (inf - inf) is dropped by fmaxf; each remaining term bounds the finite
// pairs, and pairs with a non-finite coordinate never pass the filter.
__device__ __forceinline__ float box_gap2(float3 ilo, float3 ihi, float3 jlo, float3 jhi)
{
    const float gx = fmaxf(fmaxf(__fsub_rn(jlo.x, ihi.x), __fsub_rn(ilo.x, jhi.x)), 0.0f);
    const float gy = fmaxf(fmaxf(__fsub_rn(jlo.y, ihi.y), __fsub_rn(ilo.y, jhi.y)), 0.0f);
    const float gz = fmaxf(fmaxf(__fsub_rn(jlo.z, ihi.z), __fsub_rn(ilo.z, jhi.z)), 0.0f);
    return __fmaf_rn(gz, gz, __fmaf_rn(gx, gx, __fmul_rn(gy, gy)));
}

// Whether most pairs of two boxes of bodies are likely contacts: the mean
// square distance of evenly filled boxes is below kTileNear.
constexpr float kTileNear = 0.9f;
__device__ __forceinline__ bool box_near(float3 ilo, float3 ihi, float3 jlo, float3 jhi)
{
    const auto axis = [](float a0, float a1, float b0, float b1) {
        const float d = (b0 + b1) - (a0 + a1), a = a1 - a0, b = b1 - b0;
        return 0.25f * d * d + (a * a + b * b) * (1.0f / 12.0f);
    };
    return axis(ilo.x, ihi.x, jlo.x, jhi.x) + axis(ilo.y, ihi.y, jlo.y, jhi.y) +
               axis(ilo.z, ihi.z, jlo.z, jhi.z) < kTileNear;
}

// The tiled path's shared memory.
constexpr int kTileDense = 512;               // hits of 1,024 pairs: see tile_block
constexpr int kTileQueue = kTileDense + 32;  // pairs a warp may have queued
// An item is handed out in up to 8 units of its blocks of 32 staged bodies, as
// long as there are at most kTileUnits of them per CTA: a tile keeps a warp
// busy for 30 us or more, and a small remnant has fewer items than the GPU has
// room for.  us a step, whole items / units: 4,500 remnant bodies 211 / 108,
// 9,000 291 / 168, 20,000 392 / 305, 40,000 758 / 749; 16 and 32 units per CTA
// take 2 to 5 % more from 40,000 bodies on.
constexpr unsigned int kTilePartsLog2 = 3, kTileUnits = 8;
struct TileSmem {
    float4 sp[128], sv[128];     // the staged bodies: x, y, z, body index (bits); velocity
    float4 ip[128], iv[128];     // the chunk's bodies, the same
    unsigned int js[6][128];     // sums of the staged bodies
    unsigned int is[6][128];     // queued pairs' sums of the chunk's bodies
    float4 row[3][2];            // the law's constants per pair class (PairRow, Fe bodies of the pair)
    float3 ilo[4], ihi[4];       // box of each warp's bodies
    float3 blo[4], bhi[4];       // and of each staged block of 32
    int bcls[4];                 // its bodies: 0 Si, 1 Fe, 2 both
    unsigned short queue[4][kTileQueue];  // per warp: lane of i | staged slot of j << 5
    unsigned int units, plog;    // units in all; log2 of an item's
    unsigned int w;              // the unit to take next
};

__device__ __forceinline__ PairRow tile_row(const TileSmem &sm, int cls)
{
    const float4 a = sm.row[cls][0], b = sm.row[cls][1];
    return PairRow{a.x, a.y, a.z, a.w, b.x, b.y, b.z};
}

// The 32 bodies of a warp against a staged block of 32, all pairs: in step r
// lane l takes slot (l + r) mod 32, so that the lanes' loads and their
// additions to the slots' shared sums never meet in a bank, and no list is
// kept.  For a block with itself steps 1 to 16 cover each pair once (the
// pair's terms are the same, with opposite signs, from either body).
template <bool MIXED>
__device__ __forceinline__ void tile_block(FixSum3 &acc, TileSmem &sm, int s, bool diag, int lane,
                                           float4 pi, int cls, long long *delta, int sw,
                                           int sep_test, float inv_unit)
{
    const float4 vi = sm.iv[threadIdx.x];
    const int ife = __float_as_int(pi.w) < sw;
    const float2 npxy = make_float2(-pi.x, -pi.y);
    PairRow row = tile_row(sm, MIXED ? 0 : ife + cls);
    const int r1 = !diag ? 32 : lane < 16 ? 17 : 16;
    for (int r = diag; r < r1; ++r) {
        const int k = 32 * s + ((lane + r) & 31);
        const float4 pj = sm.sp[k];
        const float2 dxy = __fadd2_rn(make_float2(pj.x, pj.y), npxy);
        const float dx = dxy.x, dy = dxy.y, dz = pj.z - pi.z;
        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
        if (r2 < 1.0f) {
            const int j = __float_as_int(pj.w);
            if (MIXED) row = tile_row(sm, ife + (int)(j < sw));
            const float c = contact_coef_at(row, sep_test, dx, dy, dz, r2, &vi, &sm.sv[k]) * inv_unit;
            fix_add3_pair(acc, sm.js, k, delta + 3 * (size_t)j, c, dx, dy, dz, r2);
        }
    }
}

// One queued pair per lane (all of them hits), n lanes.
__device__ __forceinline__ void tile_pair(TileSmem &sm, unsigned int e, bool on, int warp,
                                          long long *delta, int sw, int sep_test, float inv_unit)
{
    if (!on) return;
    const int t = 32 * warp + (int)(e & 31u), k = (int)(e >> 5);
    const float4 pi = sm.ip[t], pj = sm.sp[k];
    const int i = __float_as_int(pi.w), j = __float_as_int(pj.w);
    const float2 dxy = __fadd2_rn(make_float2(pj.x, pj.y), make_float2(-pi.x, -pi.y));
    const float dx = dxy.x, dy = dxy.y, dz = pj.z - pi.z;
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
    const PairRow row = tile_row(sm, (int)(i < sw) + (int)(j < sw));
    const float c = contact_coef_at(row, sep_test, dx, dy, dz, r2, &sm.iv[t], &sm.sv[k]) * inv_unit;
    FixSum3 a;
    fix_zero(a);
    fix_add3<false>(a, c, dx, dy, dz, r2);
    if (a.n) {
        const unsigned int h[3] = {a.hx, a.hy, a.hz}, l[3] = {a.lx, a.ly, a.lz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            atomicAdd(&sm.is[d][t], h[d] - __float_as_uint(kFixM));
            atomicAdd(&sm.is[3 + d][t], l[d] - __float_as_uint(kFixC));
            atomicAdd(&sm.js[d][k], __float_as_uint(kFixM) - h[d]);
            atomicAdd(&sm.js[3 + d][k], __float_as_uint(kFixC) - l[d]);
        }
    } else {  // out of the split's range: to the global sums
        unsigned long long *di = reinterpret_cast<unsigned long long *>(delta + 3 * (size_t)i);
        unsigned long long *dj = reinterpret_cast<unsigned long long *>(delta + 3 * (size_t)j);
        const long long v[3] = {a.x, a.y, a.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            atomicAdd(di + d, (unsigned long long)v[d]);
            atomicAdd(dj + d, 0ull - (unsigned long long)v[d]);
        }
    }
}

// Items come from a queue, longest first.  For an item the CTA holds up to
// 128 bodies of the bucket b (one per thread, all in one cell) and stages the
// neighbour bucket nb in shared memory 128 bodies at a time.  Each warp takes
// the staged blocks of 32 in turn and skips a block whose bounding box is
// provably out of reach of its own bodies' box.  Of the others it takes those
// of which at least half the pairs are contacts as a whole (tile_block: a
// crowded core's pairs mostly are); from the rest it filters the hits
// (r2 < 1) into a queue of pairs and evaluates the law on full warps of
// those, whose sums go through shared memory on both sides.  Each pair is
// evaluated once for both bodies: a self item covers the blocks from the
// chunk's own slots on, a warp those from its own (there only slots above the
// thread's), and the staged bodies' shared sums go into their corrections
// with 64-bit global atomics once per tile.
//
// What bounds it is the issue rate.  One hit list per thread left 46 % of the
// lanes idle (a block of few hits 78 %), and the lists' scattered additions
// to shared memory took four passes each: 796 us alone on a 66,000-body
// remnant (74M pairs), 585 this way.  Thresholds from 0.6 to 0.9 (kTileNear)
// and 384 to 640 (kTileDense) are within 1 % of each other.
// Staged slots past the end and threads past the chunk hold positions at
// infinity, which no pair test passes.
__global__ void __maxnreg__(72)
contact_tile_kernel(const float4 *__restrict__ spos, const float4 *__restrict__ svel,
                    const float4 *__restrict__ dpos, const float4 *__restrict__ dvel,
                    long long *__restrict__ delta, const __grid_constant__ LaunchTable tab,
                    const uint4 *__restrict__ items, unsigned int *__restrict__ ctr)
{
    __shared__ TileSmem sm;
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const unsigned int all = 0xffffffffu;
    const float kInf = __int_as_float(0x7f800000);
    unsigned short *const queue = sm.queue[warp];
#pragma unroll
    for (int d = 0; d < 6; ++d) sm.js[d][t] = sm.is[d][t] = 0u;
    launch_wait();
    // Thread 0 takes the next unit from the queue when the current one
    // reaches its last tile: the atomic's latency hides behind that tile,
    // and the CTA still takes items close to the queue's longest-first order.
    if (t == 0) {
        sm.w = atomicAdd(&ctr[kCtrHead], 1u);
        const unsigned int total = ctr[kCtrItems];
        unsigned int plog = 0u;
        while (plog < kTilePartsLog2 && total << (plog + 1u) <= kTileUnits * gridDim.x) ++plog;
        sm.plog = plog;
        sm.units = total << plog;
    }
    __syncthreads();
    for (;;) {
        const unsigned int w = sm.w, plog = sm.plog;
        if (w >= sm.units) break;
        const uint4 rec = items[w >> plog];
        unsigned int nw = 0u;  // thread 0: the next unit
        const unsigned int s0 = rec.x;
        // the unit's part of nb, in blocks of 32 from rec.y on
        const unsigned int per = ((((rec.z - rec.y + 31u) / 32u) - 1u) >> plog) + 1u;
        const unsigned int first = rec.y + 32u * per * (w & ((1u << plog) - 1u));
        const unsigned int nend = min(rec.z, first + 32u * per);
        if (first >= nend) {
            __syncthreads();  // sm.w is read
            if (t == 0) sm.w = atomicAdd(&ctr[kCtrHead], 1u);
            __syncthreads();
            continue;
        }
        const unsigned int ni = rec.w >> 16;
        const bool tiled = (rec.w >> 12) & 1u;
        // block 0's place after the warp's own, where nb is b itself
        int rel = (rec.w >> 13) & 1u ? (int)(first - rec.y) / 32 - warp : 1;
        const bool valid = (unsigned int)t < ni;
        const RunDev &R = tab.runs[rec.w & 0xffu];
        const int sw = R.offset + R.nfe;
        const float inv_unit = tab.params[R.param].inv_unit;
        const float4 pi = valid ? dpos[s0 + t] : make_float4(kInf, kInf, kInf, __int_as_float(-1));
        const float4 *npos = tiled ? dpos : spos, *nvel = tiled ? dvel : svel;
        sm.ip[t] = pi;  // read by its own warp alone
        sm.iv[t] = valid ? dvel[s0 + t] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < 3) {
            const PairRow q = pair_row(tab.params[R.param], t > 0, t > 1);
            sm.row[t][0] = make_float4(q.G, q.K, q.Tband, q.Tmid);
            sm.row[t][1] = make_float4(q.KRmid, q.KRin, q.far, 0.0f);
        }
        float3 ilo = valid ? make_float3(pi.x, pi.y, pi.z) : make_float3(kInf, kInf, kInf);
        float3 ihi = valid ? make_float3(pi.x, pi.y, pi.z) : make_float3(-kInf, -kInf, -kInf);
        warp_box(ilo, ihi);
        if (lane == 0) {
            sm.ilo[warp] = ilo;
            sm.ihi[warp] = ihi;
        }
        const bool full = (unsigned int)(32 * warp + 32) <= ni;
        FixSum3 acc;
        fix_zero(acc);
        for (unsigned int base = first; base < nend; base += 128u, rel += 4) {
            __syncthreads();  // the previous tile is consumed
            if (base != first) flush_slot(sm.js, t, __float_as_int(sm.sp[t].w), delta);
            if (t == 0 && base + 128u >= nend) nw = atomicAdd(&ctr[kCtrHead], 1u);
            const unsigned int u = base + (unsigned int)t;
            float3 lo = make_float3(kInf, kInf, kInf), hi = make_float3(-kInf, -kInf, -kInf);
            float4 q = make_float4(kInf, kInf, kInf, 0.0f);
            if (u < nend) {
                q = npos[u];
                sm.sv[t] = nvel[u];
                lo = hi = make_float3(q.x, q.y, q.z);
            }
            sm.sp[t] = q;
            warp_box(lo, hi);
            const unsigned int in = __ballot_sync(all, u < nend);
            const unsigned int fe = __ballot_sync(all, u < nend && __float_as_int(q.w) < sw);
            if (lane == 0) {
                sm.blo[warp] = lo;
                sm.bhi[warp] = hi;
                sm.bcls[warp] = fe == 0u ? 0 : fe == in ? 1 : 2;
            }
            __syncthreads();
            const int cnt = (int)min(128u, nend - base);
            int qn = 0;                              // queued pairs, the same in the warp
            bool queued = false;
            const auto drain = [&] {
                const int n = min(qn, 32);
                qn -= n;
                __syncwarp();  // the entries are written
                const unsigned int e = lane < n ? queue[qn + lane] : 0u;
                __syncwarp();  // and read, before their places are written again
                tile_pair(sm, e, lane < n, warp, delta, sw, tab.sep_test, inv_unit);
            };
            for (int s = max(-rel, 0); 32 * s < cnt; ++s) {
                const float3 alo = sm.ilo[warp], ahi = sm.ihi[warp], jlo = sm.blo[s], jhi = sm.bhi[s];
                if (box_gap2(alo, ahi, jlo, jhi) >= 1.0f) continue;  // the same for the warp
                const bool diag = rel + s == 0;  // the warp's own bodies: each pair once
                bool dense = full && 32 * s + 32 <= cnt && box_near(alo, ahi, jlo, jhi);
                unsigned int m = 0u;
                if (!dense) {
                    for (int k = 0; k < 32 && 32 * s + k < cnt; k += 8) {
                        unsigned int g = 0u;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            const float4 pj = sm.sp[32 * s + k + c];
                            const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
                            const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
                            if (r2 < 1.0f) g |= 1u << c;
                        }
                        m |= g << k;
                    }
                    if (diag) m &= 0xfffffffeu << lane;
                    const int hits = __reduce_add_sync(all, __popc(m));
                    if (hits == 0) continue;
                    dense = hits >= (diag ? kTileDense / 2 : kTileDense);
                }
                if (dense) {
                    const int cls = sm.bcls[s];
                    if (cls == 2)
                        tile_block<true>(acc, sm, s, diag, lane, pi, cls, delta, sw, tab.sep_test,
                                         inv_unit);
                    else
                        tile_block<false>(acc, sm, s, diag, lane, pi, cls, delta, sw, tab.sep_test,
                                          inv_unit);
                    continue;
                }
                // Queue the hits, one of each lane at a time and from staggered
                // slots: 32 queued pairs are then of many bodies on either side.
                queued = true;
                for (unsigned int rm = __funnelshift_r(m, m, lane);;) {
                    const unsigned int some = __ballot_sync(all, rm != 0u);
                    if (!some) break;
                    if (rm) {
                        const int b = __ffs(rm) - 1;
                        queue[qn + __popc(some & ((1u << lane) - 1u))] =
                            (unsigned short)(lane | (32 * s + ((b + lane) & 31)) << 5);
                        rm &= rm - 1u;
                    }
                    qn += __popc(some);
                }
                while (qn >= 32) drain();
            }
            if (qn) drain();
            if (acc.n >= kFixFold - 128u) fix_fold(acc);  // a tile adds at most 128 terms
            if (queued) {
                __syncwarp();
                long long v[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    v[d] = (long long)(int)sm.is[d][t] * (1ll << 23) + (int)sm.is[3 + d][t];
                    sm.is[d][t] = sm.is[3 + d][t] = 0u;
                }
                acc.x += v[0];
                acc.y += v[1];
                acc.z += v[2];
                __syncwarp();
            }
        }
        __syncthreads();  // the last tile's j-side sums are complete; sm.w is read
        flush_slot(sm.js, t, __float_as_int(sm.sp[t].w), delta);
        if (t == 0) sm.w = nw;
        __syncthreads();  // the next unit's index is visible
        fix_fold(acc);
        const long long ax = acc.x, ay = acc.y, az = acc.z;
        if (valid && (ax | ay | az)) {
            unsigned long long *d = reinterpret_cast<unsigned long long *>(
                delta + 3 * (size_t)__float_as_int(pi.w));
            atomicAdd(d + 0, (unsigned long long)ax);
            atomicAdd(d + 1, (unsigned long long)ay);
            atomicAdd(d + 2, (unsigned long long)az);
        }
    }
}

}  // namespace gi

// gi_grid_buckets and gi_grid_words (the scratch layout) are in gi_internal.h.

void gi_grid_runs(LaunchTable &tab, long long candidates)
{
    int slots = 0, buckets = 0, rows = 0, grids = 0;
    int maxn = 0;
    for (int r = 0; r < tab.nruns; ++r)
        if (tab.runs[r].n <= gi::kDirectMax) candidates -= (long long)tab.runs[r].n * tab.runs[r].n;
    const int direct = candidates >= 0 ? gi::kDirectMax : gi::kDirectAlways;
    for (int r = 0; r < tab.nruns; ++r) {
        RunDev &d = tab.runs[r];
        d.gslot = slots;
        d.gbase = buckets;
        d.glog = 0;
        d.row_start = rows;
        const int per = d.n > direct ? gi::kRowBodies : gi::kDirectBodies;
        rows += (d.n + per - 1) / per;
        if (d.n <= direct) continue;
        while ((2LL << d.glog) <= 2LL * d.n) ++d.glog;  // the largest power of two <= 2 n
        slots += d.n;
        buckets += 1 << d.glog;
        maxn = std::max(maxn, d.n);
        ++grids;
    }
    tab.rows = rows;
    tab.gridn = maxn;
    tab.gridruns = grids;
}

cudaError_t gi_contact_setup()
{
    const cudaError_t e = gi_full_carveout(reinterpret_cast<const void *>(gi::contact_row_kernel));
    return e != cudaSuccess ? e : gi_full_carveout(reinterpret_cast<const void *>(gi::contact_tile_kernel));
}

int gi_grid_cluster_ctas()
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gi::kClusterLarge);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = (size_t)(gi::kClusterMax / gi::kClusterLarge) * sizeof(unsigned int);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned int)gi::kClusterLarge, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(gi::grid_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, gi::grid_cluster_kernel, &cfg) == cudaSuccess &&
        clusters > 0)
        return gi::kClusterLarge;
    cudaGetLastError();  // not an error of the calls that follow
    return gi::kClusterSmall;
}

cudaError_t gi_launch_grid(const float4 *pos, const float4 *vel, const LaunchTable &tab,
                           const GridWork &g, long long *delta, unsigned int *ctr, int nsm,
                           int clusters, cudaStream_t s)
{
    if (tab.gridn == 0) return cudaSuccess;
    if (g.buckets > 1024u * 8192u) return cudaErrorInvalidValue;
    int maxlog = 0;
    unsigned int m = 0;
    for (int r = 0; r < tab.nruns; ++r) {
        const RunDev &d = tab.runs[r];
        if (!d.glog) continue;
        maxlog = std::max(maxlog, d.glog);
        m = (unsigned int)d.gbase + (1u << d.glog);
    }
    if (m > g.buckets) return cudaErrorInvalidValue;
    const int ctas = tab.gridn < gi::kClusterSmallMax ? gi::kClusterSmall
                     : tab.gridn < gi::kClusterMax    ? gi::kClusterLarge
                                                      : INT_MAX;
    if (clusters >= ctas) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ctas, tab.nruns);
        cfg.blockDim = dim3(1024);
        // the counts, and later 64 words per warp
        cfg.dynamicSmemBytes = std::max(((size_t)1 << maxlog) / ctas, (size_t)(64 * 32)) * 4;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {(unsigned int)ctas, 1, 1};
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, gi::grid_cluster_kernel, pos, vel, tab, g, delta, ctr);
    }
    cudaError_t e = cudaMemsetAsync(g.start, 0, ((size_t)m + 1) * sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    const dim3 gk(std::min(4 * nsm, (tab.gridn + 255) / 256), tab.nruns);
    gi::grid_keys<<<gk, 256, 0, s>>>(pos, tab, g, ctr);
    const int sb = (int)((m + 1 + 1023) / 1024);
    gi::scan_blocks<<<sb, 1024, 0, s>>>(g.start, (int)m + 1, g.sums);
    gi::scan_sums<<<1, 1024, 0, s>>>(g.sums, sb);
    gi::scan_add<<<sb, 1024, 0, s>>>(g.start, (int)m + 1, g.sums);
    gi::grid_scatter<<<gk, 256, 0, s>>>(pos, vel, tab, g, delta, ctr);
    const int gb = (int)std::min<size_t>((g.bcap + 1) / 2, 8 * (size_t)nsm);
    gi::dense_prep_kernel<<<gb, 64, 0, s>>>(tab, g, ctr);
    gi::dense_items_kernel<<<gb, 64, 0, s>>>(tab, g, ctr);
    const int go = (int)std::min<size_t>((g.icap + 255) / 256, 4 * (size_t)nsm);
    gi::dense_order_kernel<<<go, 256, 0, s>>>(g.raw, ctr, g.items);
    return cudaGetLastError();
}

cudaError_t gi_launch_rows(const float4 *pos, const float4 *vel, const LaunchTable &tab,
                           const GridWork &g, long long *delta, const unsigned int *ctr,
                           cudaStream_t s)
{
    if (tab.rows == 0) return cudaSuccess;
    gi::contact_row_kernel<<<tab.rows, 32, 0, s>>>(pos, vel, g.view(ctr), delta, tab);
    return cudaGetLastError();
}

cudaError_t gi_launch_tiles(const LaunchTable &tab, const GridWork &g, long long *delta,
                            unsigned int *ctr, int nsm, bool early, cudaStream_t s)
{
    if (tab.gridn == 0) return cudaSuccess;  // no grid, no crowded cells
    const int gt = (int)std::min<size_t>(g.icap, 7 * (size_t)nsm);
    return gi_launch(gi::contact_tile_kernel, dim3(gt), 128, early, s, g.spos, g.svel, g.dpos, g.dvel,
                     delta, tab, g.items, ctr);
}
