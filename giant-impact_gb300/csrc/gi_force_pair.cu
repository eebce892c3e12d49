// gi_force_pair.cu -- the far field with every unordered pair evaluated once
// (GI_ACCUM_PAIRED, the default accumulation mode).
//
// The law's far field is symmetric: the clamped gravity of a pair,
// G m_i m_j (x_j - x_i) / max(r, 1)^3, acts on i, and its negative on j
// (the pair law of Code/ImpactCode/impactAddTime.cu:283-370 for r >= 1,
// and the clamped term that gi_grid.cu corrects for r < 1).  The reference
// evaluates every ordered pair, each thread summing the force on its own
// body; here each pair is evaluated once and applied to both bodies, which
// cuts the pair arithmetic on the FMA pipe, the unit that bounds the far
// field, from 22 to 14 lane operations per pair.
//
// Work decomposition.  An i-block is 1024 consecutive bodies of one run; a
// j-chunk is 64 consecutive bodies of the run, two per lane (slots l and
// l + 32).  A work item is (run, i-block a, a range of `cpi` chunks); block a
// takes the chunks from its own first body onwards, so every pair i < j is
// covered exactly once.  An item is taken by independent warps, each a CTA of
// its own: a warp holds 32 ipl of the block's rows in registers (ipl = 8: four
// warps an item) and takes cpt of the item's chunks:
//   - a chunk wholly after the warp's rows: every pair, unmasked;
//   - a chunk inside the warp's rows (the diagonal): only i < j, and no row
//     whose pairs of the chunk are all masked;
//   - a chunk wholly before the warp's rows: skipped (the warp that owns
//     those bodies meets this warp's bodies as its j).
// One-warp CTAs: no barrier, no warp waits for the item's longest one, and
// the hardware hands out the next task per warp.  At N = 66,000 the kernel
// alone takes 1.012 ms; CTAs of an item's four warps, their j-sums merged in
// shared memory, took 1.070.
// ipl and cpt depend on n alone (pair_shape in gi_api.cu): short runs have too
// few items for the GPU's 608 warp schedulers, so theirs are cut finer.
// Items are numbered block-major; block a has ceil((C - 16 a) / cpi) of them
// (C = chunks of the run; cpi divides 16, so this is k0 - a 16 / cpi and the
// items before block a are an arithmetic series, decoded by bisection).  Item
// slot t of a run is item (t * stride) mod items, the stride coprime with the
// item count and about one i-block's items long: warps resident together then
// hold different i-blocks, so their i-side atomics do not queue on the same
// addresses.  Where cpt chunks are no more than a warp's rows (runs below 65,536
// bodies at the default) the i-block is the row group and the item its cpt chunks:
// the same warps, without those that would skip all their chunks.
//
// Inner loop (per warp and chunk): the chunk is staged in shared memory as
// (x_a, x_b, y_a, y_b) and (z_a, z_b, gm_a, gm_b) of slots a = l, b = l + 32,
// so one lane's two j-bodies fill the two halves of an FP32x2 register; each
// i-body is held duplicated in both halves.  Lane l starts with slots
// (l, l + 32); at step s it meets slots ((l + s) mod 32, + 32) and adds the
// 16 pairs to its 8 i-sums (one half per j) and to the two j-sums, which
// then move one lane down (one shuffle per half and component).  After 32
// steps the j-sums have visited every lane and are back on their lanes.  Per
// i-body and step, all packed: 3 FADD2 (dp), FMUL2 + 2 FFMA2 (r2), 2 FMNMX,
// 2 MUFU.RSQ, 2 FMUL2 (r^-3), 3 FFMA2 (i-sums), 3 FFMA2 (j-sums): 14
// FMA-pipe lane operations per pair, with no per-step fold of the j-sums
// (each half is one j's).  What bounds the loop is the register file: an FFMA2
// with three distinct operands issues every 3.2 to 5.3 cycles rather than 2,
// and the six sums are of that kind, so a step of 64 pairs takes 36 cycles a
// scheduler where the FMA pipe alone would take 28.  Scalar instructions for
// any group of the operations were slower (1.05 to 1.20 ms at N = 66,000,
// against 1.012): they need more issue slots and registers than they save.
// The step loop is not unrolled: 8 rows are enough independent work (1.012
// against 1.042 ms unrolled twice).
//
// Masses (gm = sqrt(G) m, so G m_i m_j = gm_i gm_j).  The i-sums gather
// dp r^-3 over a chunk and are scaled by the chunk's gm_j when folded;
// chunks that straddle the Fe/Si boundary, and the diagonal ones, take the
// per-pair gm_j instead.  A warp's 256 rows are of one class except in the
// one warp per run that straddles the boundary: the others scale their
// finished i-sums and every j-sum by their gm_i, and only the straddling
// warp multiplies gm_i into each pair.  The j-sums are scaled by their own
// gm_j and negated.
//
// Accumulation and determinism.  Chunk sums are FP32 (32 terms a half per
// i-body, 32 ipl a half per j-body and warp); a chunk's two halves are folded
// into the i-body's running FP32 sum in shared memory (at most 16 chunks).
// Everything beyond that is 64-bit fixed point with a power-of-two unit chosen
// per run so that no sum of a body's pair terms can overflow it (|F| <=
// n gm_max^2 < 2^62 units), added to one int64 per body and component in
// global memory (a plane per component: a warp's atomics are contiguous).
// Integer addition is associative, so the result does not depend on which
// warp finished first: it depends only on the run's bodies, n and cpi.
// pair_finish_kernel converts the sums, adds the contact corrections and
// stores the force or steps the bodies with the arithmetic of the one-sided
// kernel's epilogue.
#include <algorithm>

#include "gi_contact.cuh"

namespace gi {

__host__ __device__ __forceinline__ long long pair_items_before(long long a, long long k0, long long q)
{
    return a * k0 - q * ((a * (a - 1)) / 2);
}

// One warp, one 64-body chunk, two j-bodies a lane.  cxy[l] = (x_a, x_b,
// y_a, y_b) and czg[l] = (z_a, z_b, gm_a, gm_b) of chunk slots a = l and
// b = l + 32.  di = (warp's first row) - (chunk's first body), relative to
// the run.
//   EDGE: a diagonal chunk (only i < j) or one that straddles the Fe/Si
//         boundary; the i-sums take the per-pair gm_j.
//   IMIX: the warp's rows straddle the Fe/Si boundary; w takes the per-row
//         gm_i.  Every other warp has one i mass, applied after the sums.
// ax[k] (per component) gathers row k's terms, one half per j of the lane.
template <int IPL, bool EDGE, bool IMIX>
__device__ __forceinline__ void pair_chunk(const float4 *__restrict__ cxy,
                                           const float4 *__restrict__ czg, const int lane,
                                           const int di, const float (&nx)[IPL],
                                           const float (&ny)[IPL], const float (&nz)[IPL],
                                           const float (&gi)[IPL], float2 (&ax)[IPL],
                                           float2 (&ay)[IPL], float2 (&az)[IPL], float2 &bx,
                                           float2 &by, float2 &bz)
{
    bx = by = bz = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int s = 0; s < 32; ++s) {
        const int jl = (lane + s) & 31;
        const float4 q = cxy[jl];
        const float4 g = czg[jl];
        const float2 X = make_float2(q.x, q.y), Y = make_float2(q.z, q.w),
                     Z = make_float2(g.x, g.y);
#pragma unroll
        for (int k = 0; k < IPL; ++k) {
            // rows from here on have no j > i in the chunk
            if (EDGE && di + 32 * k >= kPairChunk) break;
            const float2 dx = __fadd2_rn(X, make_float2(nx[k], nx[k]));
            const float2 dy = __fadd2_rn(Y, make_float2(ny[k], ny[k]));
            const float2 dz = __fadd2_rn(Z, make_float2(nz[k], nz[k]));
            // fma(dz, dz, fma(dx, dx, dy*dy)) per lane, as the reference
            float2 r2 = __fmul2_rn(dy, dy);
            r2 = __ffma2_rn(dx, dx, r2);
            r2 = __ffma2_rn(dz, dz, r2);
            const float2 ri = make_float2(rsqrt_mufu(fmaxf(r2.x, 1.0f)),
                                          rsqrt_mufu(fmaxf(r2.y, 1.0f)));
            float2 w = IMIX ? __fmul2_rn(__fmul2_rn(ri, ri),
                                         __fmul2_rn(ri, make_float2(gi[k], gi[k])))
                            : __fmul2_rn(__fmul2_rn(ri, ri), ri);
            float2 wi = w;
            if (EDGE) {
                const int i = di + k * 32 + lane;  // this row, relative to the chunk
                w.x = i < jl ? w.x : 0.0f;
                w.y = i < jl + 32 ? w.y : 0.0f;
                wi = __fmul2_rn(w, make_float2(g.z, g.w));
            }
            ax[k] = __ffma2_rn(wi, dx, ax[k]);
            bx = __ffma2_rn(w, dx, bx);
            ay[k] = __ffma2_rn(wi, dy, ay[k]);
            by = __ffma2_rn(w, dy, by);
            az[k] = __ffma2_rn(wi, dz, az[k]);
            bz = __ffma2_rn(w, dz, bz);
        }
        // the j-sums move to the lane that meets these j next
        bx.x = __shfl_sync(0xffffffffu, bx.x, lane + 1);
        bx.y = __shfl_sync(0xffffffffu, bx.y, lane + 1);
        by.x = __shfl_sync(0xffffffffu, by.x, lane + 1);
        by.y = __shfl_sync(0xffffffffu, by.y, lane + 1);
        bz.x = __shfl_sync(0xffffffffu, bz.x, lane + 1);
        bz.y = __shfl_sync(0xffffffffu, bz.y, lane + 1);
    }
}

// Shared memory of one warp: the staged chunks and its rows' running sums.
struct PairSmem {
    float4 cxy[kPairStage * 32];  // (x_a, x_b, y_a, y_b)
    float4 czg[kPairStage * 32];  // (z_a, z_b, gm_a, gm_b)
    float si[3][kPairWarpRows];
};

// Chunk c of the run (its bodies from pos on) into place `at`.
__device__ __forceinline__ void pair_stage(PairSmem &sm, const float4 *__restrict__ pos,
                                           const RunDev &R, const PairDev &P, int c, int at, int lane)
{
    const int ja = c * kPairChunk + lane, jb = ja + 32;
    float4 pa = make_float4(GI_FAR_J, GI_FAR_J, GI_FAR_J, 0.0f), pb = pa;
    float ga = 0.0f, gb = 0.0f;
    if (ja < R.n) {
        pa = __ldg(&pos[ja]);
        ga = ja < R.nfe ? P.gm_fe : P.gm_si;
    }
    if (jb < R.n) {
        pb = __ldg(&pos[jb]);
        gb = jb < R.nfe ? P.gm_fe : P.gm_si;
    }
    sm.cxy[at * 32 + lane] = make_float4(pa.x, pb.x, pa.y, pb.y);
    sm.czg[at * 32 + lane] = make_float4(pa.z, pb.z, ga, gb);
}

__device__ __forceinline__ void add_fx(long long *p, float v)
{
    atomicAdd(reinterpret_cast<unsigned long long *>(p), (unsigned long long)__float2ll_rn(v));
}

// One warp: rows wi0 .. wi0 + 32 IPL, chunks c0 .. c1 (relative to the run).
// Row r's running i-sum (sm.si[.][r]) gathers sum_chunks gm_j sum_j w dp; each
// chunk's j-sums go, times -gm_j and scale_j, into the global sums.
template <int IPL, bool IMIX>
__device__ __forceinline__ void pair_rows(PairSmem &sm, const ForceArgs &a, const RunDev &R,
                                          const PairDev &P, const int c0, const int c1,
                                          const int wi0, const int lane, const float scale_j,
                                          const float scale_i)
{
    constexpr int kRows = 32 * IPL;
    const int rbeg = R.offset, n = R.n, nfe = R.nfe;
    long long *const out = a.fsum_fx + rbeg;
    const size_t plane = a.fsum_plane;
    // this lane's rows; beyond the run at GI_FAR_I, where r^-3 underflows to 0
    float nx[IPL], ny[IPL], nz[IPL], gi[IPL];
#pragma unroll
    for (int k = 0; k < IPL; ++k) {
        const int i = wi0 + k * 32 + lane;
        float4 p = make_float4(GI_FAR_I, GI_FAR_I, GI_FAR_I, 0.0f);
        float g = 0.0f;
        if (i < n) {
            p = __ldg(&a.pos[rbeg + i]);
            g = i < nfe ? P.gm_fe : P.gm_si;
        }
        nx[k] = -p.x;
        ny[k] = -p.y;
        nz[k] = -p.z;
        gi[k] = g;
#pragma unroll
        for (int d = 0; d < 3; ++d) sm.si[d][k * 32 + lane] = 0.0f;
    }
#pragma unroll 1
    for (int cb = c0; cb < c1; cb += kPairStage) {
        const int ce = min(cb + kPairStage, c1);
        __syncwarp();  // the previous chunks are consumed
        for (int c = cb; c < ce; ++c) pair_stage(sm, a.pos + rbeg, R, P, c, c - cb, lane);
        __syncwarp();
#pragma unroll 1
        for (int c = cb; c < ce; ++c) {
            const float4 *cxy = sm.cxy + (c - cb) * 32, *czg = sm.czg + (c - cb) * 32;
            const int jc0 = c * kPairChunk;
            const bool diag = jc0 < wi0 + kRows;
            const bool straddle = jc0 < nfe && nfe < jc0 + kPairChunk;
            float2 ax[IPL], ay[IPL], az[IPL];
#pragma unroll
            for (int k = 0; k < IPL; ++k) ax[k] = ay[k] = az[k] = make_float2(0.0f, 0.0f);
            float2 bx, by, bz;
            float gc;  // the chunk's gm_j, applied at the fold (1 for EDGE chunks)
            if (diag || straddle) {
                pair_chunk<IPL, true, IMIX>(cxy, czg, lane, wi0 - jc0, nx, ny, nz, gi, ax, ay, az,
                                            bx, by, bz);
                gc = 1.0f;
            } else {
                pair_chunk<IPL, false, IMIX>(cxy, czg, lane, 0, nx, ny, nz, gi, ax, ay, az, bx, by,
                                             bz);
                gc = jc0 < nfe ? P.gm_fe : P.gm_si;
            }
            // j side: lane l holds j = jc0 + l (.x) and jc0 + 32 + l (.y);
            // the force on j is -gm_j times its sum
            const float4 g = czg[lane];
            const float ga = -g.z * scale_j, gb = -g.w * scale_j;
            const int ja = jc0 + lane, jb = ja + 32;
            if (ja < n) {
                add_fx(out + ja, ga * bx.x);
                add_fx(out + plane + ja, ga * by.x);
                add_fx(out + 2 * plane + ja, ga * bz.x);
            }
            if (jb < n) {
                add_fx(out + jb, gb * bx.y);
                add_fx(out + plane + jb, gb * by.y);
                add_fx(out + 2 * plane + jb, gb * bz.y);
            }
            // i side: the two halves, scaled by the chunk's gm_j, into the
            // running sums (each lane owns its rows)
#pragma unroll
            for (int k = 0; k < IPL; ++k) {
                const int r = k * 32 + lane;
                sm.si[0][r] = __fmaf_rn(ax[k].x + ax[k].y, gc, sm.si[0][r]);
                sm.si[1][r] = __fmaf_rn(ay[k].x + ay[k].y, gc, sm.si[1][r]);
                sm.si[2][r] = __fmaf_rn(az[k].x + az[k].y, gc, sm.si[2][r]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < IPL; ++k) {
        const int r = k * 32 + lane, i = wi0 + r;
        if (i >= n) break;
        add_fx(out + i, sm.si[0][r] * scale_i);
        add_fx(out + plane + i, sm.si[1][r] * scale_i);
        add_fx(out + 2 * plane + i, sm.si[2][r] * scale_i);
    }
}

template <int IPL>
__device__ __forceinline__ void pair_task(PairSmem &sm, const ForceArgs &a, const RunDev &R,
                                          const PairDev &P, const int c0, const int c1,
                                          const int wi0, const int lane)
{
    // A warp whose rows are all of one class takes its gm_i out of the pair
    // loop: it scales the j-sums and the finished i-sums instead.
    const float inv = R.far_inv;
    if (wi0 < R.nfe && R.nfe < wi0 + 32 * IPL) {
        pair_rows<IPL, true>(sm, a, R, P, c0, c1, wi0, lane, inv, inv);
    } else {
        const float scale = inv * (wi0 < R.nfe ? P.gm_fe : P.gm_si);
        pair_rows<IPL, false>(sm, a, R, P, c0, c1, wi0, lane, scale, scale);
    }
}

// Warp `part` of item t of run R: its first row wi0 and its chunks [c0, c1) (none
// when they are all before the rows, or there are no rows).
__host__ __device__ __forceinline__ void pair_place(const RunDev &R, long long t, int part, int &wi0,
                                                    int &c0, int &c1)
{
    // (i-block, item of the block), then rows and chunks of the item
    const int rlog = R.pblk + 1 - R.pipl;  // log2 of the row groups of an i-block
    const long long k0 = R.pk0, q = 1 << (R.pblk - R.pcl);
    int lo = 0, hi = R.pnb - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pair_items_before(mid, k0, q) <= t) lo = mid;
        else hi = mid - 1;
    }
    wi0 = (lo << R.pblk) * kPairChunk + ((part & ((1 << rlog) - 1)) << (5 + R.pipl));
    const int cpt = 1 << (R.pcl - (R.ptpi - rlog));  // chunks of this warp
    const int cb = (lo << R.pblk) + ((int)(t - pair_items_before(lo, k0, q)) << R.pcl) +
                   (part >> rlog) * cpt;
    c0 = max(cb, wi0 / kPairChunk);
    c1 = min(cb + cpt, R.pnc);
}

// Task k of the run's items << ptpi, in 64 bits.
__host__ __device__ __forceinline__ unsigned long long pair_items_of(const RunDev &R)
{
    return pair_items_before(R.pnb, R.pk0, 1 << (R.pblk - R.pcl));
}

__host__ __device__ __forceinline__ void pair_task_place(const RunDev &R, unsigned long long k,
                                                         unsigned long long items, int &wi0, int &c0,
                                                         int &c1)
{
    pair_place(R, (long long)(((k >> R.ptpi) * R.pstride) % items), (int)k & ((1 << R.ptpi) - 1), wi0, c0,
               c1);
}

// CTA `cta` of run R, likewise.
__device__ __forceinline__ void pair_decode(const RunDev &R, int cta, int &wi0, int &c0, int &c1)
{
    const int local = cta - R.item_start;
    const int slot = local >> R.ptpi, part = local & ((1 << R.ptpi) - 1);
    pair_place(R, ((long long)slot * R.pstride) % R.pitems, part, wi0, c0, c1);
}

__device__ __forceinline__ void pair_item(PairSmem &sm, const ForceArgs &a, const LaunchTable &tab,
                                          int cta, int lane)
{
    const RunDev &R = tab.runs[find_run(tab, cta)];
    const PairDev &P = tab.params[R.param];
    int wi0, c0, c1;
    pair_decode(R, cta, wi0, c0, c1);
    if (c0 >= c1) return;
    if (R.pipl == 3) pair_task<8>(sm, a, R, P, c0, c1, wi0, lane);
    else if (R.pipl == 2) pair_task<4>(sm, a, R, P, c0, c1, wi0, lane);
    else pair_task<2>(sm, a, R, P, c0, c1, wi0, lane);
}

// The far field and, of small tables, the contact pass's row path
// (gi_contact.cuh) in one launch of one-warp CTAs: the first `rows` CTAs take
// rows, the others far-field tasks.  The two are independent until the
// epilogue, and the row path, which waits on memory, runs in the far field's
// issue gaps.  One launch on one stream: each event between streams costs 2 to
// 5 us, a step of a few thousand bodies 20 to 50.
// 162 registers (no spills): 12 CTAs per SM.  ptxas's allocation moves the
// loop by 5 %: held to 160 it takes 1.073 ms at N = 66,000 (262,144: 16.8),
// at 162 1.012 (15.25), at 168 1.037, with the sums in another order 1.032.  (The
// cap is 168; ptxas takes 162 of its own.)  Code beside the loop moves it too: with
// the row path's row_few in this kernel every run from 66,000 bodies on took 0.3 %
// more, so it is left to contact_row_kernel.
__global__ void __maxnreg__(168)
pair_force_kernel(const ForceArgs a, const GridView g, long long *__restrict__ delta, int rows,
                  const __grid_constant__ LaunchTable tab)
{
    __shared__ union Smem {
        PairSmem pair;
        RowSmem row;
        __device__ Smem() {}
    } sm;
    launch_wait();
    if ((int)blockIdx.x < rows)
        contact_rows<false>(sm.row, a.pos, a.vel, g, delta, tab, blockIdx.x);
    else
        pair_item(sm.pair, a, tab, blockIdx.x - rows, threadIdx.x);
}

// ------------------------------------------------------------- potential --
// U(r) of every unordered pair once (gi_potential_fp64), over the far field's
// work items: the same warps, rows and chunks.  No per-body sums, so the
// chunk's bodies are broadcast from shared memory, two in the halves of a
// packed register, against the lane's 8 rows.  Per pair the one-sided form's
// arithmetic: r2 as in the far field, rsqrt of max(r2, 1) refined by one
// Newton step, rounded, and added with j's mass to the row's FP32 sum of 128
// bodies, which is folded in FP64 with i's mass.  (That product's rounding is
// not even for every mass: 2.6e-8 of the sum for sqrt(G) m = 0.4 and none for
// 1, so the rounding points stay where a sum over ordered pairs has them: 128
// bodies a sum, and of the pairs of two classes half weighted with either
// mass.)  Pairs
// with r2 < 1 are left out of the sum and get the full-K polynomial: a lane
// that met one looks its step's pairs over.  Chunks on the diagonal take every
// pair by itself.
//
// 12 packed operations, 6 selects and 2 MUFU a step of 64 pairs, 9 of the
// packed ones with two distinct operands at most, so the register file holds
// it less than the far field.  A call on 66,000 bodies takes 1.04 to
// 1.18 ms (every ordered pair, unpacked, in blocks of 128: 5.3).

__device__ __forceinline__ float max_nan(float a, float b)  // NaN if a is
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ float rsqrt_refined(float rr)
{
    const float ri = rsqrt_mufu(rr);
    return ri * __fmaf_rn(-0.5f * rr, ri * ri, 1.5f);
}

// hi + lo += x, hi's rounding kept in lo (TwoSum).
__device__ __forceinline__ void add_exact(float &hi, float &lo, float x)
{
    const float s = __fadd_rn(hi, x), b = __fsub_rn(s, hi);
    lo += __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b));
    hi = s;
}

// The contact potential of one pair, r2 < 1.
__device__ __forceinline__ float contact_potential(float G, float K, float r2)
{
    const float r = __fsqrt_rn(r2);
    return -G + G * (r - 1.0f) - K * (r - r * r * r * (1.0f / 3.0f) - 2.0f / 3.0f);
}

// A chunk wholly after the rows: far[k] gathers row k's pairs, weighted with
// j's mass, or with i's (SWAP); the contact potentials go to acc, an FP32 sum for
// each step's 16 pairs (over the lane's 512 pairs, equal terms, as of bodies in one
// point, were off by up to 4e-6).  jfe: Fe bodies of the chunk (its first ones);
// i0: the lane's first row.
template <bool SWAP>
__device__ __forceinline__ void potential_chunk(const float4 *__restrict__ cxy,
                                                const float4 *__restrict__ czg, const PairDev &P,
                                                int jfe, int i0, int nfe,
                                                const float (&nx)[kPairIpl],
                                                const float (&ny)[kPairIpl],
                                                const float (&nz)[kPairIpl],
                                                float2 (&far)[kPairIpl], double &acc)
{
#pragma unroll 1
    for (int s = 0; s < 32; ++s) {
        const float4 q = cxy[s], g = czg[s];
        const float2 X = make_float2(q.x, q.y), Y = make_float2(q.z, q.w), Z = make_float2(g.x, g.y);
        bool close = false;
#pragma unroll
        for (int k = 0; k < kPairIpl; ++k) {
            const float2 dx = __fadd2_rn(X, make_float2(nx[k], nx[k]));
            const float2 dy = __fadd2_rn(Y, make_float2(ny[k], ny[k]));
            const float2 dz = __fadd2_rn(Z, make_float2(nz[k], nz[k]));
            float2 r2 = __fmul2_rn(dy, dy);
            r2 = __ffma2_rn(dx, dx, r2);
            r2 = __ffma2_rn(dz, dz, r2);
            const bool cx = r2.x < 1.0f, cy = r2.y < 1.0f;  // not in the far sum
            close |= cx | cy;
            const float gk = i0 + k * 32 < nfe ? P.gm_fe : P.gm_si;
            const float2 gm = make_float2(cx ? 0.0f : SWAP ? gk : g.z, cy ? 0.0f : SWAP ? gk : g.w);
            const float2 rr = make_float2(max_nan(r2.x, 1.0f), max_nan(r2.y, 1.0f));
            const float2 ri = make_float2(rsqrt_mufu(rr.x), rsqrt_mufu(rr.y));
            const float2 h = __fmul2_rn(rr, make_float2(-0.5f, -0.5f));
            const float2 t = __ffma2_rn(h, __fmul2_rn(ri, ri), make_float2(1.5f, 1.5f));
            far[k] = __ffma2_rn(gm, __fmul2_rn(ri, t), far[k]);
        }
        if (close) {
            float sum = 0.0f;
#pragma unroll
            for (int k = 0; k < kPairIpl; ++k) {
                const float2 dx = __fadd2_rn(X, make_float2(nx[k], nx[k]));
                const float2 dy = __fadd2_rn(Y, make_float2(ny[k], ny[k]));
                const float2 dz = __fadd2_rn(Z, make_float2(nz[k], nz[k]));
                float2 r2 = __fmul2_rn(dy, dy);
                r2 = __ffma2_rn(dx, dx, r2);
                r2 = __ffma2_rn(dz, dz, r2);
                const int ic = i0 + k * 32 < nfe;
                if (r2.x < 1.0f)
                    sum += contact_potential(P.G[ic + (s < jfe)], P.K[ic + (s < jfe)], r2.x);
                if (r2.y < 1.0f)
                    sum += contact_potential(P.G[ic + (s + 32 < jfe)], P.K[ic + (s + 32 < jfe)], r2.y);
            }
            acc += (double)sum;
        }
    }
}

// Short runs (pipl 0): every ordered pair, a lane's body against a tile of 128;
// a run of 2,000 bodies has too few sums of 128 for their rounding to average
// out, so its sums are the same ones whatever the decomposition.  Four warps of
// 32 bodies share the staged tile; each warp has its own partial.  What bounds it
// is latency: one-warp CTAs with the paired path's shared memory held 20 warps an
// SM: 1,085 us a call on 64 runs of 4,000 bodies, 817 this way (118 and 92 on one of
// 9,000).
__global__ void __launch_bounds__(128)
potential_tile_kernel(const float4 *__restrict__ pos, const __grid_constant__ LaunchTable tab,
                      double *__restrict__ partials)
{
    __shared__ float4 tile[128];  // x, y, z, gm
    int lo = 0, hi = tab.nruns - 1;  // the last run whose first block is not after this one
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tab.runs[mid].row_start <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const RunDev &R = tab.runs[lo];
    const PairDev &P = tab.params[R.param];
    const float4 *const run = pos + R.offset;
    const int t = threadIdx.x, tiles = (R.n + 127) / 128, local = (int)blockIdx.x - R.row_start;
    const int ib = local / tiles, jt = local % tiles * 128, i = ib * 128 + t;
    {
        float4 p = make_float4(GI_FAR_J, GI_FAR_J, GI_FAR_J, 0.0f);
        if (jt + t < R.n) {
            p = __ldg(&run[jt + t]);
            p.w = jt + t < R.nfe ? P.gm_fe : P.gm_si;
        }
        tile[t] = p;
    }
    const bool ife = i < R.nfe;
    float4 p = make_float4(GI_FAR_I, GI_FAR_I, GI_FAR_I, 0.0f);
    if (i < R.n) p = __ldg(&run[i]);
    __syncthreads();
    if ((i & ~31) >= R.n) return;  // the warp has no bodies
    float far = 0.0f, near = 0.0f;
#pragma unroll 4
    for (int s = 0; s < 128; ++s) {
        const float4 q = tile[s];
        const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
        const bool c = r2 < 1.0f;  // contact pairs and the body itself: not in the far sum
        far = __fmaf_rn(c ? 0.0f : q.w, rsqrt_refined(c ? 1.0f : r2), far);
        if (c && jt + s != i && i < R.n) {
            const int cls = ife + (jt + s < R.nfe);
            near += contact_potential(P.G[cls], P.K[cls], r2);
        }
    }
    double u = i < R.n ? 0.5 * (-(double)(ife ? P.gm_fe : P.gm_si) * (double)far + (double)near) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u += __shfl_down_sync(0xffffffffu, u, o);
    if ((t & 31) == 0) partials[R.item_start + (i >> 5) * tiles + jt / 128] = u;
}

// What one warp of the far field's decomposition adds to the potential: rows from
// wi0 on, chunks [c0, c1).
__device__ __forceinline__ void potential_task(PairSmem &sm, const float4 *__restrict__ run,
                                               const RunDev &R, const PairDev &P, int wi0, int c0,
                                               int c1, int lane, double &acc)
{
    constexpr int IPL = kPairIpl;
    const int n = R.n, nfe = R.nfe;
    const bool imix = wi0 < nfe && nfe < wi0 + 32 * IPL;
    float nx[IPL], ny[IPL], nz[IPL];
#pragma unroll
    for (int k = 0; k < IPL; ++k) {
        const int i = wi0 + k * 32 + lane;
        float4 p = make_float4(GI_FAR_I, GI_FAR_I, GI_FAR_I, 0.0f);
        if (c0 < c1 && i < n) p = __ldg(&run[i]);
        nx[k] = -p.x;
        ny[k] = -p.y;
        nz[k] = -p.z;
    }
    const auto class_of = [&](int k) { return (int)(wi0 + k * 32 + lane < nfe); };
    float2 far[IPL];  // per row, one sum per half: 128 bodies each, then folded
#pragma unroll
    for (int k = 0; k < IPL; ++k) far[k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int cb = c0; cb < c1; cb += kPairStage) {
        const int ce = min(cb + kPairStage, c1);
        __syncwarp();
        for (int c = cb; c < ce; ++c) pair_stage(sm, run, R, P, c, c - cb, lane);
        __syncwarp();
#pragma unroll 1
        for (int c = cb; c < ce; ++c) {
            const float4 *cxy = sm.cxy + (c - cb) * 32, *czg = sm.czg + (c - cb) * 32;
            const int jc0 = c * kPairChunk;
            // in every other group of four chunks the pairs' roots are weighted
            // with i's mass, and j's is applied at the fold
            const int g0 = jc0 & ~255;  // the group's first body
            // (not in the last, which may have places past the run: their mass is 0)
            const bool swap = (jc0 & 256) && g0 + 256 <= n && !(g0 < nfe && nfe < g0 + 256) &&
                              jc0 >= wi0 + 32 * IPL;
            const bool diag = jc0 < wi0 + 32 * IPL;
            if (diag) {  // each pair by itself
#pragma unroll 1
                for (int s = 0; s < kPairChunk; ++s) {
                    const int j = jc0 + s;
                    if (j >= n) break;
                    const float4 q = cxy[s & 31], g = czg[s & 31];
                    const float X = s < 32 ? q.x : q.y, Y = s < 32 ? q.z : q.w,
                                Z = s < 32 ? g.x : g.y, gmj = s < 32 ? g.z : g.w;
                    float sum = 0.0f;
#pragma unroll
                    for (int k = 0; k < IPL; ++k) {
                        const int i = wi0 + k * 32 + lane;
                        if (i >= j) continue;  // each pair once; no rows past the run
                        const float dx = X + nx[k], dy = Y + ny[k], dz = Z + nz[k];
                        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
                        const int cls = (i < nfe) + (j < nfe);
                        if (r2 < 1.0f) sum += contact_potential(P.G[cls], P.K[cls], r2);
                        else far[k].x = __fmaf_rn(gmj, rsqrt_refined(r2), far[k].x);
                    }
                    if (sum != 0.0f) acc += (double)sum;
                }
            } else if (swap) {
                potential_chunk<true>(cxy, czg, P, nfe - jc0, wi0 + lane, nfe, nx, ny, nz, far, acc);
            } else {
                potential_chunk<false>(cxy, czg, P, nfe - jc0, wi0 + lane, nfe, nx, ny, nz, far, acc);
            }
            if (((c - c0) & (diag ? 1 : 3)) == (diag ? 1 : 3) || c + 1 == c1) {
                // 128 bodies a sum: the rows' sums without rounding (hi + lo);
                // each with its own mass where that differs
                float hi = 0.0f, lo = 0.0f;
#pragma unroll
                for (int k = 0; k < IPL; ++k) {
                    if (imix && !swap) {
                        acc -= (double)(class_of(k) ? P.gm_fe : P.gm_si) *
                               ((double)far[k].x + (double)far[k].y);
                    } else {
                        add_exact(hi, lo, far[k].x);
                        add_exact(hi, lo, far[k].y);
                    }
                    far[k] = make_float2(0.0f, 0.0f);
                }
                const bool fe = swap ? g0 < nfe : wi0 < nfe;
                acc -= (double)(fe ? P.gm_fe : P.gm_si) * ((double)hi + (double)lo);
            }
        }
    }
}

// A run's tasks, a CTA and a partial for each; MANY: for tables with a run of more
// than kPotentialPartials, whose nsplit CTAs take several in turn (the loop and its
// 64-bit item numbers cost runs of short items 1 to 7 %).
template <bool MANY>
__global__ void __launch_bounds__(32)
potential_kernel(const float4 *__restrict__ pos, const __grid_constant__ LaunchTable tab,
                 double *__restrict__ partials)
{
    __shared__ PairSmem sm;
    const int lane = threadIdx.x;
    const RunDev &R = tab.runs[find_run(tab, blockIdx.x)];
    const PairDev &P = tab.params[R.param];
    const float4 *const run = pos + R.offset;
    int wi0, c0, c1;
    double acc = 0.0;
    if (MANY) {
        const unsigned long long items = pair_items_of(R);
        for (unsigned long long k = blockIdx.x - R.item_start; k < items << R.ptpi; k += R.nsplit) {
            pair_task_place(R, k, items, wi0, c0, c1);
            potential_task(sm, run, R, P, wi0, c0, c1, lane, acc);
        }
    } else {
        pair_decode(R, blockIdx.x, wi0, c0, c1);
        potential_task(sm, run, R, P, wi0, c0, c1, lane, acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) partials[blockIdx.x] = acc;
}

// Each run's partials summed in a fixed order: thread t takes t, t + 1024, ...,
// then a fixed shuffle tree and the 32 warps in order.
__global__ void __launch_bounds__(1024)
potential_sum_kernel(const __grid_constant__ LaunchTable tab, const double *__restrict__ partials,
                     double *__restrict__ out)
{
    __shared__ double sh[32];
    const RunDev &R = tab.runs[blockIdx.x];
    const int end = R.item_start + R.nsplit;
    double v = 0.0;
    for (int k = R.item_start + threadIdx.x; k < end; k += 1024) v += partials[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 32; ++w) t += sh[w];
        out[blockIdx.x] = t;
    }
}

// The epilogue: F = fixed-point far field + contact correction, rounded once
// to float, stored (GI_EPI_FORCE) or applied as the kick-drift (GI_EPI_STEP)
// by finish_body, the one-sided kernel's own epilogue arithmetic.  The sums
// and, behind them, the contact pass's counters are left at zero for the next
// call.
template <int EPI>
__global__ void __launch_bounds__(256) pair_finish_kernel(const ForceArgs a,
                                                          const __grid_constant__ LaunchTable tab)
{
    const RunDev &R = tab.runs[blockIdx.y];
    const double unit = tab.params[R.param].fx_unit;
    const double far_unit = R.far_unit;
    launch_wait();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < kCtrWords)
        reinterpret_cast<unsigned int *>(a.fsum_fx + 3 * a.fsum_plane)[threadIdx.x] = 0u;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < R.n; k += gridDim.x * blockDim.x) {
        const int i = R.offset + k;
        long long *q = a.fsum_fx + i;
        const double fd[3] = {(double)__ldcg(q) * far_unit,
                              (double)__ldcg(q + a.fsum_plane) * far_unit,
                              (double)__ldcg(q + 2 * a.fsum_plane) * far_unit};
        finish_body<EPI>(a, R, unit, i, fd);
        q[0] = q[a.fsum_plane] = q[2 * a.fsum_plane] = 0;
    }
}

}  // namespace gi

using namespace gi;

long long gi_pair_task(const RunDev &R, long long task, int *row, int *c0, int *c1)
{
    const unsigned long long items = pair_items_of(R);
    pair_task_place(R, (unsigned long long)task, items, *row, *c0, *c1);
    return (long long)(items << R.ptpi);
}

cudaError_t gi_pair_setup() { return gi_full_carveout(reinterpret_cast<const void *>(pair_force_kernel)); }

cudaError_t gi_launch_pair_force(const ForceArgs &a, const LaunchTable &tab, const GridWork &g,
                                 long long *delta, const unsigned int *ctr, bool with_rows,
                                 bool early, cudaStream_t s)
{
    if (tab.nitems <= 0) return cudaSuccess;
    const int rows = with_rows ? tab.rows : 0;
    return gi_launch(pair_force_kernel, dim3(rows + tab.nitems), 32, early, s, a, g.view(ctr), delta,
                     rows, tab);
}

cudaError_t gi_launch_pair_finish(int epi, const ForceArgs &a, const LaunchTable &tab, int maxn,
                                  int nsm, bool early, cudaStream_t s)
{
    if (tab.nruns <= 0 || maxn <= 0) return cudaSuccess;
    const int bx = std::max(1, std::min((maxn + 255) / 256, 4 * nsm));
    const dim3 grid(bx, tab.nruns);
    if (epi == GI_EPI_FORCE) return gi_launch(pair_finish_kernel<GI_EPI_FORCE>, grid, 256, early, s, a, tab);
    if (epi == GI_EPI_STEP) return gi_launch(pair_finish_kernel<GI_EPI_STEP>, grid, 256, early, s, a, tab);
    return cudaErrorInvalidValue;
}

cudaError_t gi_launch_potential(const float4 *pos, const LaunchTable &tab, double *partials,
                                double *out, cudaStream_t s)
{
    if (tab.nruns <= 0) return cudaSuccess;
    bool many = false;
    for (int r = 0; r < tab.nruns; ++r) many |= tab.runs[r].nsplit == kPotentialPartials;
    if (tab.nitems > 0 && many) potential_kernel<true><<<tab.nitems, 32, 0, s>>>(pos, tab, partials);
    else if (tab.nitems > 0) potential_kernel<false><<<tab.nitems, 32, 0, s>>>(pos, tab, partials);
    if (tab.rows > 0) potential_tile_kernel<<<tab.rows, 128, 0, s>>>(pos, tab, partials);
    potential_sum_kernel<<<tab.nruns, 1024, 0, s>>>(tab, partials, out);
    return cudaGetLastError();
}
