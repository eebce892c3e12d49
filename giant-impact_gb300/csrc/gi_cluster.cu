// gi_cluster.cu -- Earth / Moon identification on the GPU.
//
// The reference (findEarthAndMoon, impactBasicFunctions.h:109-217) grows
// groups on the host by repeated O(N) scans: a body joins a group when its
// FP32 distance sqrtf(dx*dx + dy*dy + dz*dz) to a member is below
// touch = 1.5 D, and a group is numbered by the index of the body that
// started it, which is its smallest index.  Those groups are exactly the
// connected components of the "touching" graph, so here:
//
//   1. cells: cubes of side touch (1 - 2^-10) / sqrt(3), so the bodies of one
//      cell all touch each other; each occupied cell takes a slot of an
//      open-addressing table (exact cell coordinates, never shared by two
//      cells) and its bodies are listed together;
//   2. union: a body starts under its cell's smallest index, so a cell costs
//      one tree and no pair tests.  Touching bodies lie at most two cells
//      apart on an axis: one warp per cell looks up the neighbour cells, skips
//      those already in its tree and tests body pairs (the reference's FP32
//      test, evaluated with the same roundings) until one touches, which
//      links the two trees.  The 13 forward adjacent cells come first, the 49
//      further ones in a second launch, when most are in the same tree (small
//      cells among many bodies: all 62 at once, cluster_link_sparse).  Links
//      always hang the root with the larger index under the one with the
//      smaller index (one atomicCAS on a root), so a tree's root is its
//      smallest member: the reference's group number;
//   3. flatten: group[i] = root of i (found without writes, so that no
//      thread overwrites a final root); sizes by atomicAdd, one per warp and
//      group;
//   4. pick: Earth = largest group, smallest name on a tie (the reference's
//      first strict maximum); Moon = largest of the others; both by a 64-bit
//      atomicMax of (size << 32 | ~name);
//   5. tag: scope byte (1 Earth, 2 Moon) and the origin counts.
// What bounds it is latency: a handful of short launches over data in L2.
// A remnant's cells hold hundreds of bodies, each within touch of tens of
// thousands: testing every pair, one thread per body, took 52 ms for 66,000
// such bodies (55.0 ms for the whole end-of-impact analysis, now 0.55 ms).
// Every loop is bounded: a failed link moves to a strictly smaller index, so
// a link takes at most N tries; the kernels still stop after a set number
// (gi_options.cluster_tries, 2^22 by default) and raise an error flag that
// the host turns into GI_ERR_TIMEOUT.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "gi_internal.h"

namespace gi {

// Cell coordinate along one axis.  Two bodies of one cell differ by at most
// a cell side (up to 2^-23 of it: the double product errs by 2^-53 of at most
// 1e9), so their FP32 distance is below touch.  Coordinates beyond 1e9 cells
// and NaN have no cell: such bodies are "loose" and tested one by one.
__device__ __forceinline__ bool cluster_cell(float4 p, double inv_cell, int3 &c)
{
    const double x = floor((double)p.x * inv_cell), y = floor((double)p.y * inv_cell),
                 z = floor((double)p.z * inv_cell);
    if (!(fabs(x) < 1.0e9 && fabs(y) < 1.0e9 && fabs(z) < 1.0e9)) return false;
    c = make_int3((int)x, (int)y, (int)z);
    return true;
}

__device__ __forceinline__ unsigned int cluster_hash(int cx, int cy, int cz)
{
    unsigned int h = (unsigned int)cx * 2246822519u;
    h ^= (unsigned int)cy * 3266489917u;
    h ^= (unsigned int)cz * 668265263u;
    h ^= h >> 13;
    h *= 2654435761u;
    return h ^ h >> 16;
}

// One slot of the cell table.  All words start at ~0.
struct CellTable {
    int *rep;              // a body of the cell, -1 = free
    unsigned int *leader;  // the cell's smallest body index
    unsigned int *count;   // bodies - 1; then the next place of its list
    int4 *cell;            // coordinates and cell number
    unsigned int *absent;  // NULL, or a bit per eighth of a slot: no cell of this hash
};

// A hash's bit of the filter `absent` (see cluster_link_sparse).
__device__ __forceinline__ unsigned int filter_bit(unsigned int h, unsigned int mask)
{
    return (h ^ h >> 15) * 2654435769u >> 3 & (8u * mask + 7u);
}

// Occupied cell k: first place in the list, bodies, slot, smallest body.
struct CellInfo {
    unsigned int beg, cnt;
    int slot, leader;
};

// Counters of a call, zero at its start.
struct ClusterCounters {
    unsigned int cells, loose, placed;
};

// Every body to its cell's slot (linear probing; the table has at least two
// slots per body).
__global__ void __launch_bounds__(256)
cluster_insert(const float4 *__restrict__ pos, int n, double inv_cell, unsigned int mask,
               CellTable tab, CellInfo *__restrict__ info, int *__restrict__ slot_of,
               int *__restrict__ loose, ClusterCounters *ctr)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int3 c;
        if (!cluster_cell(pos[i], inv_cell, c)) {
            slot_of[i] = -1;
            loose[atomicAdd(&ctr->loose, 1u)] = i;
            continue;
        }
        const unsigned int h = cluster_hash(c.x, c.y, c.z);
        unsigned int s = h & mask;
        for (unsigned int t = 0; t <= mask; ++t, s = (s + 1u) & mask) {
            int cur = __ldcg(&tab.rep[s]);
            if (cur < 0) {
                cur = atomicCAS(&tab.rep[s], -1, i);
                if (cur < 0) {
                    const unsigned int k = atomicAdd(&ctr->cells, 1u);
                    tab.cell[s] = make_int4(c.x, c.y, c.z, (int)k);
                    info[k].slot = (int)s;
                    if (tab.absent) {
                        const unsigned int f = filter_bit(h, mask);
                        atomicAnd(&tab.absent[f >> 5], ~(1u << (f & 31u)));
                    }
                    break;
                }
            }
            int3 d = c;
            cluster_cell(pos[cur], inv_cell, d);  // rep bodies have a cell
            if (d.x == c.x && d.y == c.y && d.z == c.z) break;
        }
        slot_of[i] = (int)s;
        atomicMin(&tab.leader[s], (unsigned int)i);
        atomicAdd(&tab.count[s], 1u);
    }
}

// A range of the body list for every occupied cell, in any order.
__global__ void __launch_bounds__(256)
cluster_ranges(CellTable tab, CellInfo *__restrict__ info, ClusterCounters *ctr)
{
    launch_wait();
    const int lane = threadIdx.x & 31;
    const unsigned int cells = ctr->cells;
    const unsigned int stride = gridDim.x * blockDim.x;
    for (unsigned int k0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; k0 < cells; k0 += stride) {
        const unsigned int k = k0 + lane;
        int s = 0;
        unsigned int cnt = 0;
        if (k < cells) {
            s = info[k].slot;
            cnt = tab.count[s] + 1u;
        }
        unsigned int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        unsigned int base = 0;
        if (lane == 31) base = atomicAdd(&ctr->placed, incl);
        base = __shfl_sync(0xffffffffu, base, 31);
        if (k < cells) {
            info[k].beg = base + incl - cnt;
            info[k].cnt = cnt;
            info[k].leader = (int)tab.leader[s];
            tab.count[s] = base + incl - cnt;
        }
    }
}

// The bodies listed cell by cell, each under its cell's smallest index.
__global__ void __launch_bounds__(256)
cluster_scatter(const float4 *__restrict__ pos, int n, CellTable tab,
                const int *__restrict__ slot_of, float4 *__restrict__ list,
                int *__restrict__ parent)
{
    launch_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = slot_of[i];
        parent[i] = s < 0 ? i : (int)tab.leader[s];
        if (s < 0) continue;
        list[atomicAdd(&tab.count[s], 1u)] = pos[i];
    }
}

// Root of x with path halving.  Every parent pointer points to an ancestor
// with a smaller index, so x strictly decreases and the loop ends.
__device__ __forceinline__ int find_root(int *parent, int x)
{
    for (;;) {
        const int p = __ldcg(&parent[x]);
        if (p == x) return x;
        const int g = __ldcg(&parent[p]);
        if (g == p) return p;
        __stcg(&parent[x], g);
        x = g;
    }
}

// Root of x without writes.  The flatten pass writes every body's final
// root; a path-halving write from another thread, based on a parent read
// before that write, could replace it with an intermediate ancestor.
__device__ __forceinline__ int find_root_ro(const int *parent, int x)
{
    for (;;) {
        const int p = __ldcg(&parent[x]);
        if (p == x) return x;
        x = p;
    }
}

__device__ __forceinline__ bool link(int *parent, int a, int b, int tries)
{
    for (int t = 0; t < tries; ++t) {
        a = find_root(parent, a);
        b = find_root(parent, b);
        if (a == b) return true;
        if (a < b) { const int s = a; a = b; b = s; }
        const int old = atomicCAS(&parent[a], a, b);
        if (old == a) return true;
        a = old;
    }
    return false;
}

// The reference's touch test: sqrtf of ((dx*dx + dy*dy) + dz*dz), each
// operation rounded separately (host code without contraction).
__device__ __forceinline__ bool touching(float4 a, float4 b, float touch)
{
    const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
    const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return __fsqrt_rn(r2) < touch;
}

// touching() of the closest points of two boxes, in its roundings: each axis
// difference, square, sum and root is monotone, so a false result proves that
// no pair of their bodies touches.
__device__ __forceinline__ bool boxes_touch(float3 alo, float3 ahi, float3 blo, float3 bhi,
                                            float touch)
{
    const float gx = fmaxf(fmaxf(__fsub_rn(blo.x, ahi.x), __fsub_rn(alo.x, bhi.x)), 0.0f);
    const float gy = fmaxf(fmaxf(__fsub_rn(blo.y, ahi.y), __fsub_rn(alo.y, bhi.y)), 0.0f);
    const float gz = fmaxf(fmaxf(__fsub_rn(blo.z, ahi.z), __fsub_rn(alo.z, bhi.z)), 0.0f);
    return touching(make_float4(gx, gy, gz, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f), touch);
}

// Whether any body of cell a touches one of cell b, by one warp: 32 bodies of
// a at a time, one per lane, against b's in turn; lanes whose body cannot
// reach b's box sit out.
__device__ __forceinline__ bool cells_touch_warp(const float4 *__restrict__ list, CellInfo a,
                                                 CellInfo b, float touch, int lane)
{
    const float kInf = __int_as_float(0x7f800000);
    float3 lo = make_float3(kInf, kInf, kInf), hi = make_float3(-kInf, -kInf, -kInf);
    for (unsigned int u = lane; u < b.cnt; u += 32) {
        const float4 q = list[b.beg + u];
        lo = make_float3(fminf(lo.x, q.x), fminf(lo.y, q.y), fminf(lo.z, q.z));
        hi = make_float3(fmaxf(hi.x, q.x), fmaxf(hi.y, q.y), fmaxf(hi.z, q.z));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
        hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
        hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
    }
    for (unsigned int u = 0; u < a.cnt; u += 32) {
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        bool in = u + lane < a.cnt;
        if (in) {
            p = list[a.beg + u + lane];
            const float3 q = make_float3(p.x, p.y, p.z);
            in = boxes_touch(q, q, lo, hi, touch);
        }
        if (!__any_sync(0xffffffffu, in)) continue;
        for (unsigned int v = 0; v < b.cnt; v += 4) {
            bool hit = false;
#pragma unroll
            for (unsigned int w = 0; w < 4; ++w)  // the last body again past the end
                hit |= touching(p, list[b.beg + min(v + w, b.cnt - 1u)], touch);
            if (__any_sync(0xffffffffu, hit && in)) return true;
        }
    }
    return false;
}

// Pair tests a lane makes by itself; larger cell pairs go to the whole warp.
constexpr unsigned int kLanePairs = 64;

// Links cell a (the warp's) with each lane's cell b (cnt 0: none) where bodies of
// theirs touch.  Trees that are already one are not tested; of a lane's pairs of at
// most `few` bodies that is not looked at first.
__device__ __forceinline__ void link_cells(const float4 *__restrict__ list, const CellInfo &a,
                                           const CellInfo &b, float touch, unsigned int few, int tries,
                                           int *parent, int *err, int lane)
{
    const unsigned long long pairs = (unsigned long long)a.cnt * b.cnt;
    bool open = pairs > 0u &&
                (pairs <= few || find_root(parent, a.leader) != find_root(parent, b.leader));
    bool hit = false;
    if (open && pairs <= kLanePairs) {
        for (unsigned int u = 0; u < a.cnt && !hit; ++u) {
            const float4 p = list[a.beg + u];
            for (unsigned int v = 0; v < b.cnt && !hit; ++v)
                hit = touching(p, list[b.beg + v], touch);
        }
        open = false;
    }
    for (unsigned int todo = __ballot_sync(0xffffffffu, open); todo; todo &= todo - 1u) {
        const int src = __ffs(todo) - 1;
        CellInfo q;
        q.beg = __shfl_sync(0xffffffffu, b.beg, src);
        q.cnt = __shfl_sync(0xffffffffu, b.cnt, src);
        const bool swap = a.cnt < q.cnt;  // the larger cell's bodies on the lanes
        const bool any = cells_touch_warp(list, swap ? q : a, swap ? a : q, touch, lane);
        if (lane == src) hit = any;
    }
    // the lanes link together: their attempts on one root collide and
    // are tried again on the root that won
    if (hit && !link(parent, a.leader, b.leader, tries)) atomicExch(err, 1);
}

// One warp per occupied cell.  FAR = false: its 13 forward neighbours that
// share a face, edge or corner; FAR = true: the 49 forward cells beyond them,
// two a lane.
template <bool FAR>
__global__ void __launch_bounds__(128)
cluster_link(const float4 *__restrict__ list, CellTable tab, const CellInfo *__restrict__ info,
             unsigned int mask, float touch, int tries, int *parent,
             const ClusterCounters *__restrict__ ctr, int *__restrict__ err)
{
    launch_wait();
    const int lane = threadIdx.x & 31;
    const unsigned int cells = ctr->cells, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < cells; k += nwarps) {
        const CellInfo a = info[k];
        const int4 c = tab.cell[a.slot];
        for (int round = 0; round < (FAR ? 2 : 1); ++round) {
            // forward half of the 3^3 or 5^3 block around the cell
            constexpr int kSide = FAR ? 5 : 3, kHalf = kSide / 2;
            const int o = kSide * kSide * kSide / 2 + 1 + round * 32 + lane;
            const int ox = o % kSide - kHalf, oy = o / kSide % kSide - kHalf,
                      oz = o / (kSide * kSide) - kHalf;
            bool look = o < kSide * kSide * kSide;
            if (FAR) look = look && (abs(ox) == 2 || abs(oy) == 2 || abs(oz) == 2);
            CellInfo b{0u, 0u, 0, 0};
            if (look) {
                unsigned int s = cluster_hash(c.x + ox, c.y + oy, c.z + oz) & mask;
                for (unsigned int t = 0; t <= mask; ++t, s = (s + 1u) & mask) {
                    if (__ldg(&tab.rep[s]) < 0) break;
                    const int4 d = __ldg(&tab.cell[s]);
                    if (d.x == c.x + ox && d.y == c.y + oy && d.z == c.z + oz) {
                        b = info[d.w];
                        break;
                    }
                }
            }
            link_cells(list, a, b, touch, 0u, tries, parent, err, lane);
        }
    }
}

// The same for many bodies, whose table is larger than L2: there a cell costs its
// chain of dependent loads from memory, and most of a sparse state's cells hold one
// body among empty neighbours.  So the chain is made short and taken once: the
// filter, a byte for each slot's 28, says from L2 which neighbours are empty; all 62
// are looked up before any is linked, two to a lane, their first probes together;
// one or two pairs are tested sooner than two trees are climbed; and a cell of at
// most kFew bodies takes its near and far neighbours in the first launch.  Grouping
// a raw ball of 4M bodies took 14.0 ms with the two launches above (9.1 with one
// thread per body and its 27 cells), now 8.5; of 1M 2.6 (2.2) and 1.6; 200,000 0.50
// and 0.33; 4M settled bodies 5.2 both ways.  Below kSparseMin bodies more lanes
// linking at once collide on the roots: 20,000 settled ones 0.14 and 0.19.
constexpr unsigned int kFew = 2u;
constexpr int kSparseMin = 150000;
template <bool FAR>
__global__ void __launch_bounds__(128)
cluster_link_sparse(const float4 *__restrict__ list, CellTable tab, const CellInfo *__restrict__ info,
                    unsigned int mask, float touch, int tries, int *parent,
                    const ClusterCounters *__restrict__ ctr, int *__restrict__ err)
{
    launch_wait();
    const int lane = threadIdx.x & 31;
    const unsigned int cells = ctr->cells, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < cells; k += nwarps) {
        const CellInfo a = info[k];
        const bool few = a.cnt <= kFew;
        if (FAR && few) continue;
        const int4 c = tab.cell[a.slot];
        int3 at[2];
        unsigned int s[2];
        bool look[2];
        int rep[2];
        int4 d[2];
        CellInfo b[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int o = 63 + r * 32 + lane;  // of the 5^3 block
            const int ox = o % 5 - 2, oy = o / 5 % 5 - 2, oz = o / 25 - 2;
            const bool near = abs(ox) < 2 && abs(oy) < 2 && oz < 2;
            at[r] = make_int3(c.x + ox, c.y + oy, c.z + oz);
            const unsigned int h = cluster_hash(at[r].x, at[r].y, at[r].z), f = filter_bit(h, mask);
            s[r] = h & mask;
            look[r] = o < 125 && (few || near != FAR) && !(__ldg(&tab.absent[f >> 5]) >> (f & 31u) & 1u);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            rep[r] = look[r] ? __ldg(&tab.rep[s[r]]) : -1;
            d[r] = look[r] ? __ldg(&tab.cell[s[r]]) : c;
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            for (unsigned int t = 0; t <= mask && rep[r] >= 0; ++t) {
                if (d[r].x == at[r].x && d[r].y == at[r].y && d[r].z == at[r].z) break;
                s[r] = (s[r] + 1u) & mask;
                rep[r] = __ldg(&tab.rep[s[r]]);
                d[r] = __ldg(&tab.cell[s[r]]);
            }
            b[r] = CellInfo{0u, 0u, 0, 0};
            if (rep[r] >= 0) b[r] = info[d[r].w];
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) link_cells(list, a, b[r], touch, kFew, tries, parent, err, lane);
    }
}

// Bodies without a cell (beyond 1e9 cells, or not finite): one warp each
// against every body.
__global__ void __launch_bounds__(128)
cluster_link_loose(const float4 *__restrict__ pos, int n, const int *__restrict__ loose,
                   float touch, int tries, int *parent, const ClusterCounters *__restrict__ ctr,
                   int *__restrict__ err)
{
    launch_wait();
    const int lane = threadIdx.x & 31;
    const unsigned int total = ctr->loose, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total; w += nwarps) {
        const int i = loose[w];
        const float4 p = pos[i];
        for (int j = lane; j < n; j += 32)
            if (j != i && touching(p, pos[j], touch) && !link(parent, i, j, tries))
                atomicExch(err, 1);
    }
}

// sizes start at -1 (the ~0 fill); one atomic per warp and group.
__global__ void __launch_bounds__(256)
cluster_flatten(int *parent, int n, int *__restrict__ size, int *__restrict__ ngroups)
{
    launch_wait();
    const int lane = threadIdx.x & 31;
    int roots = 0;
    for (int i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        int r = -1;
        if (i < n) {
            r = find_root_ro(parent, i);
            __stcg(&parent[i], r);
            roots += r == i;
        }
        const unsigned int same = __match_any_sync(0xffffffffu, r);
        if (r >= 0 && lane == __ffs(same) - 1) atomicAdd(&size[r], __popc(same));
    }
    for (int o = 16; o > 0; o >>= 1) roots += __shfl_down_sync(0xffffffffu, roots, o);
    if (lane == 0 && roots) atomicAdd(ngroups, roots);
}

__device__ __forceinline__ unsigned long long group_key(int size, int name)
{
    return ((unsigned long long)(unsigned int)size << 32) | (unsigned int)(~(unsigned int)name);
}

__device__ __forceinline__ int key_name(unsigned long long k)
{
    return k ? (int)(~(unsigned int)(k & 0xffffffffull)) : -1;
}

// exclude_key: the Earth's key when picking the Moon, NULL when picking the Earth.
__global__ void __launch_bounds__(256)
cluster_pick(const int *__restrict__ group, const int *__restrict__ size, int n,
             const unsigned long long *exclude_key, unsigned long long *best)
{
    launch_wait();
    const int skip = exclude_key ? key_name(*exclude_key) : -1;
    unsigned long long k = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (group[i] == i && i != skip) k = max(k, group_key(size[i] + 1, i));
    for (int o = 16; o > 0; o >>= 1) k = max(k, __shfl_down_sync(0xffffffffu, k, o));
    if ((threadIdx.x & 31) == 0 && k) atomicMax(best, k);
}

// keys[0] Earth, keys[1] Moon; counts[0..3] Earth, [4..7] Moon by origin.
__global__ void __launch_bounds__(256)
cluster_tag(const int *__restrict__ group, int n, const unsigned long long *__restrict__ keys,
            int b0, int b1, int b2, int *__restrict__ group_out,
            unsigned char *__restrict__ scope_out, int *__restrict__ counts)
{
    launch_wait();
    __shared__ int sc[8];
    if (threadIdx.x < 8) sc[threadIdx.x] = 0;
    __syncthreads();
    const int earth = key_name(keys[0]), moon = key_name(keys[1]);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int g = group[i];
        const unsigned char s = g == earth ? 1 : (g == moon ? 2 : 0);
        if (group_out) group_out[i] = g;
        if (scope_out) scope_out[i] = s;
        if (s) {
            const int c = i < b0 ? 0 : (i < b1 ? 1 : (i < b2 ? 2 : 3));
            atomicAdd(&sc[4 * (s - 1) + c], 1);
        }
    }
    __syncthreads();
    if (threadIdx.x < 8 && sc[threadIdx.x]) atomicAdd(&counts[threadIdx.x], sc[threadIdx.x]);
}

}  // namespace gi

namespace {

struct ClusterResult {
    unsigned long long keys[2];
    int counts[8];
    int ngroups;
    int err;
    gi::ClusterCounters ctr;
    int pad;
};

int cuda_status(cudaError_t e, const char *what)
{
    char buf[256];
    snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    return gi_internal_fail(e == cudaErrorMemoryAllocation ? GI_ERR_OUT_OF_MEMORY : GI_ERR_CUDA, buf);
}

}  // namespace

extern "C" int gi_find_earth_moon(gi_ctx *ctx, const float *pos, int n, float touch,
                                  const int bounds[3], int *group, unsigned char *scope,
                                  gi_earth_moon *out, void *stream)
{
    if (!ctx || !out || !bounds || (n > 0 && !pos) || n < 0)
        return gi_internal_fail(GI_ERR_INVALID_ARG, "gi_find_earth_moon: NULL argument or n < 0");
    if (!(touch > 0.0f) || !(touch < 1.0e30f))
        return gi_internal_fail(GI_ERR_INVALID_ARG, "gi_find_earth_moon: touch must be positive");
    if (reinterpret_cast<uintptr_t>(pos) % 16)
        return gi_internal_fail(GI_ERR_ALIGNMENT, "gi_find_earth_moon: pos not 16-byte aligned");
    std::memset(out, 0, sizeof *out);
    out->earth_label = out->moon_label = -1;
    if (n == 0) return GI_OK;
    const int dev = gi_internal_ctx_device(ctx);
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
    struct Restore {
        int prev, dev;
        ~Restore()
        {
            if (prev != dev && prev >= 0) cudaSetDevice(prev);
        }
    } restore{prev, dev};
    cudaStream_t s = (cudaStream_t)stream;
    unsigned int m = 1024;
    while (m < 2u * (unsigned int)n && m < (1u << 30)) m <<= 1;
    if (m > 1024u * 8192u) return gi_internal_fail(GI_ERR_BAD_SIZE, "gi_find_earth_moon: n too large");
    // One block of the context's workspace: the result, the cell
    // coordinates, the body list and the cell list (16-byte words), then the
    // words that start at ~0 (rep, leader, count, absent, size), then the rest.
    const size_t M = m, N = (size_t)n;
    const size_t head = (sizeof(ClusterResult) + 15) & ~(size_t)15;
    const bool sparse = n >= gi::kSparseMin;
    const size_t F = sparse ? M / 4 : 0;
    const size_t bytes = head + 16 * (M + 2 * N) + 4 * (3 * M + F + N) + 4 * 3 * N;
    void *work = nullptr, *pinned = nullptr;
    if (int st = gi_internal_ctx_workspace(ctx, bytes, &work, &pinned)) return st;
    unsigned char *buf = static_cast<unsigned char *>(work);
    ClusterResult *res = reinterpret_cast<ClusterResult *>(buf);
    gi::CellTable tab;
    tab.cell = reinterpret_cast<int4 *>(buf + head);
    float4 *list = reinterpret_cast<float4 *>(tab.cell + M);
    gi::CellInfo *info = reinterpret_cast<gi::CellInfo *>(list + N);
    tab.rep = reinterpret_cast<int *>(info + N);
    tab.leader = reinterpret_cast<unsigned int *>(tab.rep + M);
    tab.count = tab.leader + M;
    tab.absent = sparse ? tab.count + M : nullptr;
    int *size = reinterpret_cast<int *>(tab.count + M + F);
    int *parent = size + N, *slot_of = parent + N, *loose = slot_of + N;
    ClusterResult &host = *static_cast<ClusterResult *>(pinned);
    // Where the squares of the touch test leave FP32's normal range, cells
    // would not decide as the test does: no body gets one then.
    const bool plain = touch > 1.0e-17f && touch < 1.0e18f;
    const double inv_cell = plain ? std::sqrt(3.0) / ((double)touch * (1.0 - 1.0 / 1024.0)) : HUGE_VAL;
    const float4 *P = reinterpret_cast<const float4 *>(pos);
    const int tries = gi_internal_ctx_cluster_tries(ctx);
    const int gridded = std::min((n + 255) / 256, 4096);
    const int warps = std::min((n + 3) / 4, 16384);  // blocks of four warps, one cell each
    cudaError_t e;
    do {
        if ((e = cudaMemsetAsync(res, 0, sizeof(ClusterResult), s)) != cudaSuccess) break;
        if ((e = cudaMemsetAsync(tab.rep, 0xff, 4 * (3 * M + F + N), s)) != cudaSuccess) break;
        gi::cluster_insert<<<gridded, 256, 0, s>>>(P, n, inv_cell, m - 1, tab, info, slot_of, loose,
                                                   &res->ctr);
        // each launch follows the one before it early
        const auto next = [&](auto kernel, int grid, int threads, auto &&...args) {
            if (e == cudaSuccess) e = gi_launch(kernel, dim3(grid), threads, true, s, args...);
        };
        e = cudaGetLastError();
        next(gi::cluster_ranges, gridded, 256, tab, info, &res->ctr);
        next(gi::cluster_scatter, gridded, 256, P, n, tab, slot_of, list, parent);
        next(sparse ? gi::cluster_link_sparse<false> : gi::cluster_link<false>, warps, 128, list, tab, info,
             m - 1, touch, tries, parent, &res->ctr, &res->err);
        next(sparse ? gi::cluster_link_sparse<true> : gi::cluster_link<true>, warps, 128, list, tab, info,
             m - 1, touch, tries, parent, &res->ctr, &res->err);
        next(gi::cluster_link_loose, std::min(warps, 1024), 128, P, n, loose, touch, tries, parent,
             &res->ctr, &res->err);
        next(gi::cluster_flatten, gridded, 256, parent, n, size, &res->ngroups);
        next(gi::cluster_pick, gridded, 256, parent, size, n, nullptr, &res->keys[0]);
        next(gi::cluster_pick, gridded, 256, parent, size, n, &res->keys[0], &res->keys[1]);
        next(gi::cluster_tag, gridded, 256, parent, n, res->keys, bounds[0], bounds[1], bounds[2], group,
             scope, res->counts);
        if (e != cudaSuccess) break;
        if ((e = cudaMemcpyAsync(&host, res, sizeof host, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
            break;
    } while (false);
    const cudaError_t es = cudaStreamSynchronize(s);  // the workspace is idle again
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) return cuda_status(e, "gi_find_earth_moon");
    if (host.err) return gi_internal_fail(GI_ERR_TIMEOUT, "gi_find_earth_moon: a link did not settle");
    auto name = [](unsigned long long k) { return k ? (int)(~(unsigned int)(k & 0xffffffffull)) : -1; };
    out->earth_label = name(host.keys[0]);
    out->moon_label = name(host.keys[1]);
    out->n_earth = (int)(host.keys[0] >> 32);
    out->n_moon = (int)(host.keys[1] >> 32);
    out->n_groups = host.ngroups;
    for (int c = 0; c < 4; ++c) {
        out->earth_counts[c] = host.counts[c];
        out->moon_counts[c] = host.counts[4 + c];
    }
    return GI_OK;
}

// ------------------------------------------------------------------ disk --

namespace gi {

// Largest distance of an Earth element (scope 1) from the Earth's centre of
// mass, as the bits of a non-negative double (ordered like the value).
__global__ void __launch_bounds__(256)
earth_radius_kernel(const float4 *__restrict__ pos, const unsigned char *__restrict__ scope, int off,
                    int n, double cx, double cy, double cz, unsigned long long *__restrict__ rmax)
{
    double m = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int i = off + k;
        if (scope[i] != 1) continue;
        const float4 p = pos[i];
        const double dx = p.x - cx, dy = p.y - cy, dz = p.z - cz;
        m = fmax(m, sqrt(dx * dx + dy * dy + dz * dz));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(rmax, (unsigned long long)__double_as_longlong(m));
}

// counts: [disk, bound inside, unbound]
__global__ void __launch_bounds__(256)
disk_kernel(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
            unsigned char *__restrict__ scope, int off, int n, double cx, double cy, double cz,
            double ux, double uy, double uz, double gm, const unsigned long long *__restrict__ rmax,
            int *__restrict__ counts)
{
    launch_wait();
    __shared__ int sc[3];
    if (threadIdx.x < 3) sc[threadIdx.x] = 0;
    __syncthreads();
    const double R = __longlong_as_double((long long)*rmax) + 0.5;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int i = off + k;
        const unsigned char s = scope[i];
        if (s == 1 || s == 2) continue;
        const float4 p = pos[i], u = vel[i];
        const double rx = p.x - cx, ry = p.y - cy, rz = p.z - cz;
        const double vx = u.x - ux, vy = u.y - uy, vz = u.z - uz;
        const double r = sqrt(rx * rx + ry * ry + rz * rz);
        const double eps = 0.5 * (vx * vx + vy * vy + vz * vz) - gm / r;
        const double hx = ry * vz - rz * vy, hy = rz * vx - rx * vz, hz = rx * vy - ry * vx;
        const double req = (hx * hx + hy * hy + hz * hz) / gm;
        int c;
        if (eps < 0.0) c = req > R ? 0 : 1;
        else c = 2;
        scope[i] = c == 0 ? 3 : 0;
        atomicAdd(&sc[c], 1);
    }
    __syncthreads();
    if (threadIdx.x < 3 && sc[threadIdx.x]) atomicAdd(&counts[threadIdx.x], sc[threadIdx.x]);
}

}  // namespace gi

extern "C" int gi_find_disk(gi_ctx *ctx, const float *pos, const float *vel, const gi_run *run,
                            const gi_pair_params *params, unsigned char *scope, gi_disk_info *out,
                            void *stream)
{
    if (!ctx || !pos || !vel || !run || !params || !scope || !out)
        return gi_internal_fail(GI_ERR_INVALID_ARG, "gi_find_disk: NULL argument");
    if (run->n < 0 || run->offset < 0)
        return gi_internal_fail(GI_ERR_BAD_SIZE, "gi_find_disk: bad run");
    if (!(params->MassSi > 0.0f) || !(params->GMassSiSi > 0.0f))
        return gi_internal_fail(GI_ERR_PARAMS, "gi_find_disk: masses and gravity must be positive");
    std::memset(out, 0, sizeof *out);
    double earth[15];
    if (int st = gi_diag_fp64(ctx, pos, vel, scope, 2, run, params, earth, stream)) return st;
    out->earth_mass = earth[0];
    if (run->n == 0 || !(earth[0] > 0.0)) return GI_OK;  // no Earth: nothing is bound to it
    const double G = (double)params->GMassSiSi / ((double)params->MassSi * params->MassSi);
    const int dev = gi_internal_ctx_device(ctx);
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
    struct Restore {
        int prev, dev;
        ~Restore()
        {
            if (prev != dev && prev >= 0) cudaSetDevice(prev);
        }
    } restore{prev, dev};
    cudaStream_t s = (cudaStream_t)stream;
    struct Res {
        unsigned long long rmax;
        int counts[3];
        int pad;
    };
    void *work = nullptr, *pinned = nullptr;
    if (int st = gi_internal_ctx_workspace(ctx, sizeof(Res), &work, &pinned)) return st;
    Res *res = static_cast<Res *>(work);
    Res &host = *static_cast<Res *>(pinned);
    cudaError_t e;
    const int blocks = std::min((run->n + 255) / 256, 4096);
    const float4 *P = reinterpret_cast<const float4 *>(pos);
    do {
        if ((e = cudaMemsetAsync(res, 0, sizeof(Res), s)) != cudaSuccess) break;
        gi::earth_radius_kernel<<<blocks, 256, 0, s>>>(P, scope, run->offset, run->n, earth[1], earth[2],
                                                       earth[3], &res->rmax);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        e = gi_launch(gi::disk_kernel, dim3(blocks), 256, true, s, P, reinterpret_cast<const float4 *>(vel),
                      scope, run->offset, run->n, earth[1], earth[2], earth[3], earth[4], earth[5],
                      earth[6], G * earth[0], &res->rmax, res->counts);
        if (e != cudaSuccess) break;
        if ((e = cudaMemcpyAsync(&host, res, sizeof host, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
            break;
    } while (false);
    const cudaError_t es = cudaStreamSynchronize(s);  // the workspace is idle again
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) return cuda_status(e, "gi_find_disk");
    double r = 0.0;
    std::memcpy(&r, &host.rmax, sizeof r);
    out->earth_radius = r + 0.5;
    out->n_disk = host.counts[0];
    out->n_bound_inside = host.counts[1];
    out->n_unbound = host.counts[2];
    return GI_OK;
}
