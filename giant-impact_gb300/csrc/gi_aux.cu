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
// the FMA form of TwoProd are error-free, and every addition renormalises
// the pair, so a thread's sum of n terms is exact to about n 2^-48 of the
// terms' magnitudes.  This GPU issues FP64 at a small fraction of its FP32
// rate: with the per-body work in FP64 the two passes ran at ~850 GB/s, with
// it on the FP32 pipe they are bound by HBM.  FP64 remains for the block
// partials and everything after them.
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
__device__ __forceinline__ void ff_add2(FF &a, float xh, float xl)
{
    float s, e;
    two_sum(a.hi, xh, s, e);
    e = __fadd_rn(e, __fadd_rn(a.lo, xl));
    a.hi = __fadd_rn(s, e);
    a.lo = __fsub_rn(e, __fsub_rn(a.hi, s));
}

__device__ __forceinline__ void ff_add(FF &a, float x) { ff_add2(a, x, 0.0f); }

// a += x * y, the product taken exactly (p + e with e = fma(x, y, -p)).
__device__ __forceinline__ void ff_add_prod(FF &a, float x, float y)
{
    const float p = __fmul_rn(x, y);
    ff_add2(a, p, __fmaf_rn(x, y, -p));
}

// x - c for a float x and a double c given as ch + cl (ch = (float)c):
// TwoSum of x and -ch is exact, cl is folded into the low part.
__device__ __forceinline__ FF ff_sub_d(float x, float ch, float cl)
{
    FF r;
    float e;
    two_sum(x, -ch, r.hi, e);
    r.lo = __fsub_rn(e, cl);
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
    ff_add2(a, s, __fadd_rn(t, __fsub_rn(e1, e2)));
}

__device__ __forceinline__ double ff_value(const FF &a) { return (double)a.hi + (double)a.lo; }

// Sum of the lanes' pairs to lane 0 (float-float), NV of them.
template <int NV>
__device__ __forceinline__ void warp_ff_sum(FF (&v)[NV])
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            const float h = __shfl_down_sync(0xffffffffu, v[c].hi, o);
            const float l = __shfl_down_sync(0xffffffffu, v[c].lo, o);
            ff_add2(v[c], h, l);
        }
    }
}

// Lane 0 of each warp passes its values (FP64); the block's warps are
// added in warp order and thread c < NV writes value c of the block to
// dst.  Then each block takes a ticket: the block that takes the last one
// returns true, after a fence, so every block's partials are visible to it.
template <int NV>
__device__ __forceinline__ bool block_store_last(const double (&v)[NV], double *dst,
                                                 int *ticket)
{
    __shared__ double sh[NV][8];
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) sh[c][warp] = v[c];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double x = 0.0;
        const int nw = blockDim.x >> 5;
        for (int w = 0; w < nw; ++w) x += sh[threadIdx.x][w];
        dst[threadIdx.x] = x;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// Both passes give each block one material class, so the class mass
// multiplies the block's sums once, in FP64: blocks [0, nbfe) take the
// run's Fe bodies [0, nfe), blocks [nbfe, gridDim.x) its Si bodies [nfe, n),
// each class in a grid-stride loop over its own blocks (nbfe in proportion
// to nfe).  Block b's partials are work[16 b ..].
__device__ __forceinline__ void class_range(int nfe, int n, int nbfe, double mfe, double msi,
                                            int &k0, int &k1, int &b, int &nb, double &m)
{
    const bool fe = (int)blockIdx.x < nbfe;
    k0 = fe ? 0 : nfe;
    k1 = fe ? nfe : n;
    b = fe ? (int)blockIdx.x : (int)blockIdx.x - nbfe;
    nb = fe ? nbfe : (int)gridDim.x - nbfe;
    m = fe ? mfe : msi;
}

// The block partials summed in a fixed order, by the block that finished
// last: thread t takes blocks t, t + 256, ... in order (read past L1), then
// a fixed shuffle tree within each warp, then the 8 warps in order.  The
// result is deterministic for a given grid; it is valid in thread 0.
template <int NV>
__device__ __forceinline__ void ordered_sums(const double *work, int nblocks, double (&res)[NV])
{
    __shared__ double sh[NV][8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double v[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) v[c] = 0.0;
    for (int b = t; b < nblocks; b += 256)
#pragma unroll
        for (int c = 0; c < NV; ++c) v[c] += __ldcg(work + 16 * b + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < NV; ++c) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) sh[c][warp] = v[c];
    }
    __syncthreads();
    if (t == 0) {
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            double x = 0.0;
            for (int w = 0; w < 8; ++w) x += sh[c][w];
            res[c] = x;
        }
    }
}

// Pass 1: mass, sum m x, sum m v, kinetic energy, count (9 doubles / block);
// its last block writes out = [mass, com3, vcom3, -, -, -, ke, p3, count].
__global__ void __launch_bounds__(256)
diag_pass1(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
           const unsigned char *__restrict__ label, int scope, int off, int n,
           int nfe, int nbfe, double mfe, double msi, double *__restrict__ work,
           int *__restrict__ ticket, double *__restrict__ out)
{
    int k0, k1, b, nb;
    double m;
    class_range(nfe, n, nbfe, mfe, msi, k0, k1, b, nb, m);
    FF v[7];
#pragma unroll
    for (int c = 0; c < 7; ++c) v[c] = FF{0.0f, 0.0f};
    int cnt = 0;
    stream_bodies(pos, vel, label, scope, off, k0 + b * blockDim.x + threadIdx.x, k1,
                  nb * blockDim.x, [&](float4 p, float4 u) {
                      ff_add(v[0], p.x);
                      ff_add(v[1], p.y);
                      ff_add(v[2], p.z);
                      ff_add(v[3], u.x);
                      ff_add(v[4], u.y);
                      ff_add(v[5], u.z);
                      ff_add_prod(v[6], u.x, u.x);
                      ff_add_prod(v[6], u.y, u.y);
                      ff_add_prod(v[6], u.z, u.z);
                      ++cnt;
                  });
    warp_ff_sum<7>(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    const double d[9] = {m * cnt,
                         m * ff_value(v[0]), m * ff_value(v[1]), m * ff_value(v[2]),
                         m * ff_value(v[3]), m * ff_value(v[4]), m * ff_value(v[5]),
                         0.5 * m * ff_value(v[6]), (double)cnt};
    if (!block_store_last<9>(d, work + 16 * blockIdx.x, ticket)) return;
    double s[9];
    ordered_sums<9>(work, gridDim.x, s);
    if (threadIdx.x != 0) return;
    const double M = s[0];
    out[0] = M;
    for (int c = 0; c < 3; ++c) {
        out[1 + c] = M > 0.0 ? s[1 + c] / M : 0.0;
        out[4 + c] = M > 0.0 ? s[4 + c] / M : 0.0;
        out[11 + c] = s[4 + c];
    }
    out[10] = s[7];
    out[14] = s[8];
}

// Pass 2: angular momentum about the com, relative to the com velocity
// (impactBasicFunctions.h:507-652 in double): r = x - com and w = v - vcom
// as float-float pairs, sum of r x w per class; its last block writes
// out[7..9].
__global__ void __launch_bounds__(256, 4)
diag_pass2(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
           const unsigned char *__restrict__ label, int scope, int off, int n,
           int nfe, int nbfe, double mfe, double msi, double *__restrict__ out,
           double *__restrict__ work, int *__restrict__ ticket)
{
    int k0, k1, b, nb;
    double m;
    class_range(nfe, n, nbfe, mfe, msi, k0, k1, b, nb, m);
    float ch[6], cl[6];  // com xyz, vcom xyz as float pairs
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        const double x = out[1 + c];
        ch[c] = (float)x;
        cl[c] = (float)(x - (double)ch[c]);
    }
    FF L[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) L[c] = FF{0.0f, 0.0f};
    stream_bodies(pos, vel, label, scope, off, k0 + b * blockDim.x + threadIdx.x, k1,
                  nb * blockDim.x, [&](float4 p, float4 u) {
                      const FF rx = ff_sub_d(p.x, ch[0], cl[0]), ry = ff_sub_d(p.y, ch[1], cl[1]),
                               rz = ff_sub_d(p.z, ch[2], cl[2]);
                      const FF wx = ff_sub_d(u.x, ch[3], cl[3]), wy = ff_sub_d(u.y, ch[4], cl[4]),
                               wz = ff_sub_d(u.z, ch[5], cl[5]);
                      ff_add_cross(L[0], ry, wz, rz, wy);
                      ff_add_cross(L[1], rz, wx, rx, wz);
                      ff_add_cross(L[2], rx, wy, ry, wx);
                  });
    warp_ff_sum<3>(L);
    const double d[3] = {m * ff_value(L[0]), m * ff_value(L[1]), m * ff_value(L[2])};
    if (!block_store_last<3>(d, work + 16 * blockIdx.x, ticket)) return;
    double s[3];
    ordered_sums<3>(work, gridDim.x, s);
    if (threadIdx.x != 0) return;
    out[7] = s[0]; out[8] = s[1]; out[9] = s[2];
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

// One resident wave per pass: the grid-stride loops give every block the
// same number of bodies, so a grid of exactly the resident blocks has no
// partial last wave.
int gi_diag_blocks(int pass, int sm_count)
{
    int per_sm = 0;
    const cudaError_t e = pass == 1
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gi::diag_pass1, 256, 0)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gi::diag_pass2, 256, 0);
    if (e != cudaSuccess || per_sm < 1) per_sm = 1;
    return std::max(2, per_sm * sm_count);
}

cudaError_t gi_launch_diag(const float4 *pos, const float4 *vel,
                           const unsigned char *label, int scope,
                           const RunDev &run, float mass_fe, float mass_si, double *work,
                           int nblocks1, int nblocks2, double *out_dev, int *ticket,
                           cudaStream_t s)
{
    if (nblocks1 < 2 || nblocks2 < 2) return cudaErrorInvalidValue;
    // blocks for the Fe bodies in proportion to their number (at least one
    // when there are any), the rest for the Si bodies
    const auto fe_blocks = [&](int nblocks) {
        int nbfe = run.n > 0 ? (int)((long long)nblocks * run.nfe / run.n) : 0;
        if (run.nfe > 0 && nbfe < 1) nbfe = 1;
        if (nbfe > nblocks - 1) nbfe = nblocks - 1;
        return nbfe;
    };
    cudaError_t e = cudaMemsetAsync(ticket, 0, 2 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    gi::diag_pass1<<<nblocks1, 256, 0, s>>>(pos, vel, label, scope, run.offset, run.n, run.nfe,
                                            fe_blocks(nblocks1), mass_fe, mass_si, work, ticket,
                                            out_dev);
    gi::diag_pass2<<<nblocks2, 256, 0, s>>>(pos, vel, label, scope, run.offset, run.n, run.nfe,
                                            fe_blocks(nblocks2), mass_fe, mass_si, out_dev, work,
                                            ticket + 1);
    return cudaGetLastError();
}

cudaError_t gi_launch_ffma_peak(float *sink, int blocks, int iters, cudaStream_t s)
{
    gi::ffma_peak_kernel<<<blocks, 256, 0, s>>>(sink, iters);
    return cudaGetLastError();
}
