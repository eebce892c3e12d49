// gi_aux.cu -- the memory-bound kernels around the force pass: kick-drift,
// FP64 diagnostic reductions, and the FFMA throughput
// microbenchmark that gives the force kernel its roofline denominator.
#include <algorithm>

#include "gi_internal.h"

namespace gi {

// v += (F - damp v) dt/m ; x += v dt, w carried through.
// Reference: moveBodiesCollisionSingleGPU (Code/ImpactCode/impactAddTime.cu:
// 379-394) and moveBodiesDampedSeperate (Code/GenerateTargetImpactorCode/
// generateTargetImpactor.cu:628-664).  80 B per body (read pos, vel, force;
// write pos, vel).
__global__ void __launch_bounds__(256)
move_kernel(float4 *__restrict__ pos, float4 *__restrict__ vel,
            const float4 *__restrict__ force, const __grid_constant__ LaunchTable tab)
{
    const RunDev &R = tab.runs[blockIdx.y];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= R.n) return;
    const int i = R.offset + k;
    const float dtm = (k < R.nfe) ? R.dtm_fe : R.dtm_si;
    const float4 f = __ldg(&force[i]);
    float4 v = vel[i];
    float4 p = pos[i];
    v.x = __fmaf_rn(__fmaf_rn(-R.damp, v.x, f.x), dtm, v.x);
    v.y = __fmaf_rn(__fmaf_rn(-R.damp, v.y, f.y), dtm, v.y);
    v.z = __fmaf_rn(__fmaf_rn(-R.damp, v.z, f.z), dtm, v.z);
    p.x = __fmaf_rn(v.x, R.dt, p.x);
    p.y = __fmaf_rn(v.y, R.dt, p.y);
    p.z = __fmaf_rn(v.z, R.dt, p.z);
    vel[i] = v;
    pos[i] = p;
}

// ----------------------------------------------------------------- diag --

// Whether a body of label l is in the scope (1: labels 1 and 2, 2: label 1,
// 3: label 2, 4: label 3); scope 0 takes every body and reads no labels.
__device__ __forceinline__ bool label_in_scope(unsigned char l, int scope)
{
    if (scope == 1) return l == 1 || l == 2;
    if (scope == 2) return l == 1;
    if (scope == 3) return l == 2;
    return l == 3;
}

// Calls body(p, u) for the in-scope bodies k, k + stride, k + 2 stride, ...
// below k1 (run-relative; off is the run's first body), in that order.  The
// loop is software-pipelined: the next two bodies' loads (position,
// velocity, label) are issued before the current two bodies' arithmetic, so
// a thread always has loads in flight and the passes stream at the HBM rate
// rather than waiting on each load.
template <class Body>
__device__ __forceinline__ void stream_bodies(const float4 *__restrict__ pos,
                                              const float4 *__restrict__ vel,
                                              const unsigned char *__restrict__ label,
                                              int scope, int off, int k, int k1, int stride,
                                              Body &&body)
{
    const bool lab = label != nullptr && scope != 0;
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 p0 = z, u0 = z, p1 = z, u1 = z;
    unsigned char l0 = 0, l1 = 0;
    bool h0 = k < k1, h1 = k + stride < k1;
    if (h0) {
        p0 = pos[off + k]; u0 = vel[off + k];
        if (lab) l0 = label[off + k];
    }
    if (h1) {
        p1 = pos[off + k + stride]; u1 = vel[off + k + stride];
        if (lab) l1 = label[off + k + stride];
    }
    while (h0) {
        const int kn = k + 2 * stride;
        const bool g0 = kn < k1, g1 = kn + stride < k1;
        float4 q0 = z, w0 = z, q1 = z, w1 = z;
        unsigned char m0 = 0, m1 = 0;
        if (g0) {
            q0 = pos[off + kn]; w0 = vel[off + kn];
            if (lab) m0 = label[off + kn];
        }
        if (g1) {
            q1 = pos[off + kn + stride]; w1 = vel[off + kn + stride];
            if (lab) m1 = label[off + kn + stride];
        }
        if (!lab || label_in_scope(l0, scope)) body(p0, u0);
        if (h1 && (!lab || label_in_scope(l1, scope))) body(p1, u1);
        p0 = q0; u0 = w0; l0 = m0; p1 = q1; u1 = w1; l1 = m1;
        h0 = g0; h1 = g1; k = kn;
    }
}

// The sums of the diagnostics are kept per thread in float-float pairs on
// the FP32 pipe: a value is hi + lo, about 48 significant bits.  TwoSum and
// the FMA form of TwoProd are error-free, and every addition renormalises the
// pair, so a thread's sum of n terms is exact to about n 2^-48 of the terms'
// magnitudes.  (Gathering lo without that is 3 operations of 11 less and 10 to
// 1,000 times further off in the sums that cancel.)  This GPU
// issues FP64 at a small fraction of its FP32 rate: with the per-body work in
// FP64 the sums ran at ~850 GB/s.  FP64 remains for the block partials and
// everything after them.
struct FF {
    float hi, lo;
};

__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// a += xh + xl, renormalised (|lo| <= ulp(hi) / 2).
__device__ __forceinline__ void ff_add(FF &a, float xh, float xl)
{
    float s, e;
    two_sum(a.hi, xh, s, e);
    e = __fadd_rn(e, __fadd_rn(a.lo, xl));
    a.hi = __fadd_rn(s, e);
    a.lo = __fsub_rn(e, __fsub_rn(a.hi, s));
}

// x - c for floats, exactly.
__device__ __forceinline__ FF ff_diff(float x, float c)
{
    FF r;
    two_sum(x, -c, r.hi, r.lo);
    return r;
}

// a += u v - w z for float-float u, v, w, z: each product's high part
// exact, its cross terms to 2^-24 of themselves, the lo * lo terms
// (2^-48 of the product) left out.
__device__ __forceinline__ void ff_add_cross(FF &a, FF u, FF v, FF w, FF z)
{
    const float p1 = __fmul_rn(u.hi, v.hi);
    float e1 = __fmaf_rn(u.hi, v.hi, -p1);
    e1 = __fmaf_rn(u.hi, v.lo, __fmaf_rn(u.lo, v.hi, e1));
    const float p2 = __fmul_rn(w.hi, z.hi);
    float e2 = __fmaf_rn(w.hi, z.hi, -p2);
    e2 = __fmaf_rn(w.hi, z.lo, __fmaf_rn(w.lo, z.hi, e2));
    float s, t;
    two_sum(p1, -p2, s, t);
    ff_add(a, s, __fadd_rn(t, __fsub_rn(e1, e2)));
}

// The sums of a block's bodies, all of one material class.
constexpr int kDiagSums = 10;    // r, w (3 each), v.v, r x w (3)
constexpr int kDiagParts = 12;   // the same times the class mass, r.r's, then the count
constexpr int kDiagLook = 32;    // bodies a thread looks at for the reference

// The body that the sums are taken about: the run's first, or where that one is
// not in scope the first of its first 8,192 that is, if any.  By the whole block.
__device__ __forceinline__ int diag_reference(const unsigned char *__restrict__ label, int scope, int n)
{
    if (label == nullptr || scope == 0 || label_in_scope(label[0], scope)) return 0;
    __shared__ int first;
    if (threadIdx.x == 0) first = n;
    __syncthreads();
    int mine = n;
#pragma unroll 16
    for (int v = kDiagLook - 1; v >= 0; --v) {
        const int k = 256 * v + (int)threadIdx.x;
        if (k < n && label_in_scope(label[k], scope)) mine = k;
    }
    if (mine < n) atomicMin(&first, mine);
    __syncthreads();
    return first < n ? first : 0;
}

// The whole diagnostic in one pass over the state (32 B per body): with r = x
// - x0 and w = v - v0 about a reference body of the scope (exact as float-float
// pairs), the sums of m, m r, m w, m v.v and m r x w give the mass, the centre of
// mass, the momenta, and the angular momentum about the centre of mass relative
// to its velocity, L = sum m r x w - M rc x wc (impactBasicFunctions.h:507-652 in
// double; rc, wc the centre's r and w).  That is as good as sums about the centre
// wherever the scope is and however it moves, while the reference is about as
// near to the centre as the scope's bodies are.  Where it is not (a body that
// escaped or ran away) L would lose digits to the difference, or overflow:
// gi_diag_fp64 sees that from rc, wc and the sum of m r.r, and repeats the pass
// about the centre it found.
// The call, read-back included, takes 110 us on 8.4M bodies and 23 us on 66,000
// (24 where it looks for the reference).  Two passes, the first for the centre,
// took 144 and 65; one about the run's first body whatever the scope 108 and 22,
// but L of a Moon with that body in the Earth was off by 8e-13 of sqrt(sum m r.r
// sum m w.w), with it 1e6 D away by 2e-9 (now 6e-16 and 1e-15).  What bounds the
// pass is the FP32 pipe beside HBM: 219 operations a body.
//
// Each block takes one material class, so the class mass multiplies the
// block's sums once, in FP64: blocks [0, nbfe) the run's Fe bodies [0, nfe),
// the others its Si bodies [nfe, n), each class in a grid-stride loop over its
// own blocks.  Block b's partials are work[16 b ..]; the block that takes the
// last ticket sums them in a fixed order (a warp per value: lane l takes
// blocks l, l + 32, ..., then a fixed shuffle tree), so the result is
// deterministic for a given grid.
// out = [mass, com3, vcom3, L3, ke, p3, count, sum of m r.r (FP32 sums), rc3, wc3].
// Four blocks an SM (64 registers, two words spilled outside the loop); three of
// 75 registers took 135 us.
__global__ void __launch_bounds__(256, 4)
diag_kernel(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
            const unsigned char *__restrict__ label, int scope, int off, int n, int nfe, int nbfe,
            double mfe, double msi, const DiagOrigin origin, double *__restrict__ work,
            int *__restrict__ ticket, double *__restrict__ out)
{
    const bool fe = (int)blockIdx.x < nbfe;
    const int k0 = fe ? 0 : nfe, k1 = fe ? nfe : n;
    const int b = fe ? (int)blockIdx.x : (int)blockIdx.x - nbfe;
    const int nb = fe ? nbfe : (int)gridDim.x - nbfe;
    const double m = fe ? mfe : msi;
    __shared__ float ref[6];  // the reference; a component that is not finite counts as 0
    {
        float x[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) x[d] = origin.x[d];
        if (!origin.given && n > 0) {
            float4 p = pos[off], u = vel[off];
            if (const int k = diag_reference(label ? label + off : nullptr, scope, n)) {
                p = pos[off + k];
                u = vel[off + k];
            }
            x[0] = p.x; x[1] = p.y; x[2] = p.z;
            x[3] = u.x; x[4] = u.y; x[5] = u.z;
        }
#pragma unroll
        for (int d = 0; d < 6; ++d)
            if ((int)threadIdx.x == d) ref[d] = fabsf(x[d]) <= 3.0e38f ? x[d] : 0.0f;
    }
    __syncthreads();
    float x0[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) x0[d] = ref[d];
    FF v[kDiagSums];
#pragma unroll
    for (int c = 0; c < kDiagSums; ++c) v[c] = FF{0.0f, 0.0f};
    int cnt = 0;
    float rr = 0.0f;
    stream_bodies(pos, vel, label, scope, off, k0 + b * blockDim.x + threadIdx.x, k1,
                  nb * blockDim.x, [&](float4 p, float4 u) {
                      const FF r[3] = {ff_diff(p.x, x0[0]), ff_diff(p.y, x0[1]), ff_diff(p.z, x0[2])};
                      const FF w[3] = {ff_diff(u.x, x0[3]), ff_diff(u.y, x0[4]), ff_diff(u.z, x0[5])};
                      const float uu[3] = {u.x, u.y, u.z};
#pragma unroll
                      for (int d = 0; d < 3; ++d) {
                          ff_add(v[d], r[d].hi, r[d].lo);
                          ff_add(v[3 + d], w[d].hi, w[d].lo);
                          rr = __fmaf_rn(r[d].hi, r[d].hi, rr);
                      }
                      float q = __fmul_rn(uu[0], uu[0]), e = __fmaf_rn(uu[0], uu[0], -q);
#pragma unroll
                      for (int d = 1; d < 3; ++d) {
                          const float y = __fmul_rn(uu[d], uu[d]);
                          float t;
                          e = __fadd_rn(e, __fmaf_rn(uu[d], uu[d], -y));
                          two_sum(q, y, q, t);
                          e = __fadd_rn(e, t);
                      }
                      ff_add(v[6], q, e);
                      ff_add_cross(v[7], r[1], w[2], r[2], w[1]);
                      ff_add_cross(v[8], r[2], w[0], r[0], w[2]);
                      ff_add_cross(v[9], r[0], w[1], r[1], w[0]);
                      ++cnt;
                  });
    // the warp's sums to lane 0, then the block's warps in order
    __shared__ double part[kDiagParts][8];
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < kDiagSums; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float h = __shfl_down_sync(0xffffffffu, v[c].hi, o);
            const float l = __shfl_down_sync(0xffffffffu, v[c].lo, o);
            ff_add(v[c], h, l);
        }
        if (lane == 0) part[c][warp] = (double)v[c].hi + (double)v[c].lo;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rr += __shfl_down_sync(0xffffffffu, rr, o);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        part[kDiagSums][warp] = (double)rr;
        part[kDiagSums + 1][warp] = (double)cnt;
    }
    __syncthreads();
    if (threadIdx.x < kDiagParts) {
        double x = 0.0;
        for (int w = 0; w < 8; ++w) x += part[threadIdx.x][w];
        work[16 * blockIdx.x + threadIdx.x] = threadIdx.x <= kDiagSums ? m * x : x;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    __shared__ double sum[kDiagParts + 1];  // the last: Fe bodies
    for (int c = warp; c < kDiagParts + 1; c += 8) {
        const int end = c == kDiagParts ? nbfe : (int)gridDim.x;
        double x = 0.0;
        for (int q = lane; q < end; q += 32) x += __ldcg(work + 16 * q + min(c, kDiagSums + 1));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sum[c] = x;
    }
    __syncthreads();
    if (warp != 0) return;
    if (lane == 0) *ticket = 0;  // for the next call
    const double count = sum[kDiagSums + 1], cfe = sum[kDiagParts];
    const double M = mfe * cfe + msi * (count - cfe);
    // lane c < 6: the centre's position and velocity, one FP64 division each
    const int c = min(lane, 5);
    const double rel = M > 0.0 ? sum[c] / M : 0.0, mean = M > 0.0 ? (double)ref[c] + rel : 0.0;
    // lane d < 3: component d of the angular momentum
    const int d = lane % 3, p = (d + 1) % 3, q = (d + 2) % 3;
    const double rp = __shfl_sync(0xffffffffu, rel, p), rq = __shfl_sync(0xffffffffu, rel, q),
                 wp = __shfl_sync(0xffffffffu, rel, 3 + p), wq = __shfl_sync(0xffffffffu, rel, 3 + q);
    if (lane < 6) {
        out[1 + lane] = mean;
        out[16 + lane] = rel;
        if (lane >= 3) out[8 + lane] = M * (double)ref[c] + sum[lane];
    }
    if (lane < 3) out[7 + lane] = sum[7 + lane] - M * (rp * wq - rq * wp);
    if (lane == 0) {
        out[0] = M;
        out[10] = 0.5 * sum[6];
        out[14] = count;
        out[15] = sum[kDiagSums];
    }
}

// ------------------------------------------------------------ FFMA peak --
// Eight independent FMA chains per thread; 2 flops per FMA.
__global__ void __launch_bounds__(256) ffma_peak_kernel(float *sink, int iters)
{
    float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
    float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
    const float m = 0.9999999f, c = 1e-7f;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            a0 = __fmaf_rn(a0, m, c); a1 = __fmaf_rn(a1, m, c);
            a2 = __fmaf_rn(a2, m, c); a3 = __fmaf_rn(a3, m, c);
            a4 = __fmaf_rn(a4, m, c); a5 = __fmaf_rn(a5, m, c);
            a6 = __fmaf_rn(a6, m, c); a7 = __fmaf_rn(a7, m, c);
        }
    }
    const float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 1234.5f) sink[blockIdx.x] = s;
}

}  // namespace gi

cudaError_t gi_launch_move(float4 *pos, float4 *vel, const float4 *force,
                           const LaunchTable &tab, cudaStream_t s)
{
    int maxn = 0;
    for (int r = 0; r < tab.nruns; ++r) maxn = tab.runs[r].n > maxn ? tab.runs[r].n : maxn;
    if (maxn == 0 || tab.nruns == 0) return cudaSuccess;
    dim3 grid((maxn + 255) / 256, tab.nruns), block(256);
    gi::move_kernel<<<grid, block, 0, s>>>(pos, vel, force, tab);
    return cudaGetLastError();
}

int gi_diag_blocks(int sm_count)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gi::diag_kernel, 256, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    return std::max(2, per_sm * sm_count);
}

cudaError_t gi_launch_diag(const float4 *pos, const float4 *vel,
                           const unsigned char *label, int scope,
                           const RunDev &run, float mass_fe, float mass_si, double *work,
                           const DiagOrigin &origin, int max_blocks, double *out, int *ticket,
                           cudaStream_t s)
{
    if (max_blocks < 2) return cudaErrorInvalidValue;
    // One resident wave (the grid-stride loops give every block the same
    // number of bodies, so there is no partial last wave), but no more blocks
    // than two bodies a thread: a small run's time is the blocks' sums.
    const int nblocks = std::max(2, std::min(max_blocks, (run.n + 511) / 512));
    // blocks for the Fe bodies in proportion to their number (at least one
    // when there are any), the rest for the Si bodies
    int nbfe = run.n > 0 ? (int)((long long)nblocks * run.nfe / run.n) : 0;
    if (run.nfe > 0 && nbfe < 1) nbfe = 1;
    if (nbfe > nblocks - 1) nbfe = nblocks - 1;
    gi::diag_kernel<<<nblocks, 256, 0, s>>>(pos, vel, label, scope, run.offset, run.n, run.nfe, nbfe,
                                            mass_fe, mass_si, origin, work, ticket, out);
    return cudaGetLastError();
}

cudaError_t gi_launch_ffma_peak(float *sink, int blocks, int iters, cudaStream_t s)
{
    gi::ffma_peak_kernel<<<blocks, 256, 0, s>>>(sink, iters);
    return cudaGetLastError();
}
