// gi_internal.h -- device-side tables and launch plumbing shared by the
// libgi translation units.  Not part of the public ABI (see include/gi_api.h).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/gi_api.h"

// Threads per CTA of the one-sided force kernel (gi_force_impl.cuh); also
// its j-tile staged in shared memory and the granularity of its Kahan fold
// (one fold per 128 j).  The paired far field's shape is kPair* below.
#define GI_NT 128
// Runs and pair tables carried by value in one launch.
#define GI_MAX_RUNS 64
#define GI_MAX_PARAMS 8
// Padding position for j beyond a chunk / i beyond a run: far enough that
// gravity underflows to zero, never within contact range of a real body.
#define GI_FAR_J 1.0e16f
#define GI_FAR_I (-1.0e16f)

#define GI_ACC_PAIRED GI_ACCUM_PAIRED  // gi_force_pair.cu
#define GI_ACC_KAHAN GI_ACCUM_KAHAN    // the one-sided kernel's modes
#define GI_ACC_FP32 GI_ACCUM_FP32
#define GI_ACC_FP64 GI_ACCUM_FP64

#define GI_EPI_FORCE 0  // write force[i].xyz
#define GI_EPI_STEP 1   // fused kick-drift into the other state buffer
#define GI_EPI_SUM 2    // FP64 far-field sums into fsum; gi_launch_finish completes

// Pair constants indexed by the pair class test = (i is Fe) + (j is Fe):
// 0 = Si-Si, 1 = Fe-Si, 2 = Fe-Fe.
struct PairDev {
    double fx_unit;      // fixed-point unit of the contact corrections (force)
    float gm_fe, gm_si;  // sqrt(G) m: G m_i m_j = gm_i gm_j (far-field gravity)
    float G[3];          // G m_i m_j of the class (contact band)
    float K[3];          // full stiffness
    float KRmid[3];      // reduced stiffness, middle shell band (Fe-Si: KRMix)
    float KRin[3];       // reduced stiffness, inner band
    float Tband[3];      // r >= ShellBreak(1)  <=>  r2 >= Tband
    float Tmid[3];       // r >= ShellBreakFeSi2 <=> r2 >= Tmid (= Tband otherwise)
    float inv_unit;      // (float)(1 / fx_unit), the scale of a pair term into fixed point
};

struct RunDev {
    int offset, n, nfe, param;
    int item_start;   // first work item of this run (paired: first CTA)
    int nsplit;       // j-chunks per i-block
    int jchunk;       // bodies per big chunk (GI_NT * 2^lg)
    int nib;          // i-blocks
    int lg;           // log2 of the big chunk in tiles of GI_NT bodies
    int tiles;        // tiles of the run, ceil(n / GI_NT)
    int tick_base;    // first ticket of this run
    long long part_base;  // first double of this run's partial sums
    float dt, dtm_fe, dtm_si, damp;
    int ipt;          // i-bodies per thread this run was planned for
    // GI_ACC_PAIRED decomposition (gi_force_pair.cu)
    int pblk;         // log2 of the chunks (of rows) in an i-block
    int pcl;          // log2 of the j-chunks per work item
    int pnc;          // j-chunks of the run, ceil(n / kPairChunk)
    int pnb;          // i-blocks of the run, ceil(pnc / 2^pblk)
    int pk0;          // work items of i-block 0, ceil(pnc / 2^pcl)
    int pitems;       // work items of the run
    int pstride;      // item slot t of the run is item (t * pstride) mod pitems (coprime)
    int pipl;         // log2 of the rows a lane holds: 32 << pipl rows a warp
    int ptpi;         // log2 of the warps (CTAs) that share an item
    float far_inv;    // 1 / far_unit: scale of a far-field sum into fixed point
    double far_unit;  // fixed-point unit of the far-field sums (a power of two)
    // cell grid of the contact pass (gi_grid_runs)
    int glog;         // log2 of the run's buckets; 0: no grid, every body is a candidate
    int gbase, gslot; // its first bucket and first slot
    int row_start;    // its first row-path CTA
};

struct LaunchTable {
    int nruns;
    int nitems;
    int sep_test;
    int dense_min;  // contact pass: bucket size from which the tiled kernel takes it
    int rows;       // row-path CTAs of all runs
    int gridn;      // bodies of the largest run with a grid (0: none)
    int gridruns;   // runs with a grid
    RunDev runs[GI_MAX_RUNS];
    PairDev params[GI_MAX_PARAMS];
};

struct ForceArgs {
    const float4 *pos;
    const float4 *vel;
    float4 *force;     // GI_EPI_FORCE
    float4 *pos_out;   // GI_EPI_STEP
    float4 *vel_out;   // GI_EPI_STEP
    double *partials;  // split-j partial sums (nullptr when no run splits)
    unsigned int *tickets;
    unsigned int *queue;  // [0] next work item, [1] CTAs finished (zero between launches)
    const long long *delta;  // contact corrections, 3 per body, fixed point (gi_grid.cu)
    double *fsum;            // GI_EPI_SUM: far-field sums, 3 per body
    long long *fsum_fx;      // GI_ACC_PAIRED: far-field sums, fixed point, one plane per
    size_t fsum_plane;       // component, fsum_plane bodies apart
};

// Launchers (gi_force_ipt*.cu).  Return cudaError_t of the launch.
cudaError_t gi_launch_force(int ipt, int acc, int epi, const ForceArgs &a,
                            const LaunchTable &tab, int grid, cudaStream_t s);
cudaError_t gi_launch_force_ipt1(int acc, int epi, const ForceArgs &a, const LaunchTable &tab, int grid, cudaStream_t s);
cudaError_t gi_launch_force_ipt2(int acc, int epi, const ForceArgs &a, const LaunchTable &tab, int grid, cudaStream_t s);
cudaError_t gi_launch_force_ipt4(int acc, int epi, const ForceArgs &a, const LaunchTable &tab, int grid, cudaStream_t s);
cudaError_t gi_launch_force_ipt8(int acc, int epi, const ForceArgs &a, const LaunchTable &tab, int grid, cudaStream_t s);
// Resident CTAs per SM of a force kernel instance (for the planner).
int gi_force_occupancy(int ipt, int acc, int epi);
cudaError_t gi_force_carveout(int ipt, int acc);
// The epilogue of a GI_EPI_SUM launch (epi = GI_EPI_FORCE or GI_EPI_STEP):
// adds the contact corrections and stores or steps, one thread per body.
cudaError_t gi_launch_finish(int epi, const ForceArgs &a, const LaunchTable &tab, int maxn,
                             int nsm, cudaStream_t s);

// gi_force_pair.cu: the far field with each unordered pair evaluated once.
// Its shape is fixed here, where the planner reads it.
namespace gi {
constexpr int kPairIpl = 8;                               // i-bodies per lane, at most
constexpr int kPairWarpRows = 32 * kPairIpl;              // 256 rows per warp, at most
constexpr int kPairRowsLog2 = 10;
constexpr int kPairRows = 1 << kPairRowsLog2;             // 1024: the i-block
constexpr int kPairChunkLog2 = 6;
constexpr int kPairChunk = 1 << kPairChunkLog2;           // 64, the j-chunk: two bodies per lane
constexpr int kPairBlockChunks = kPairRows / kPairChunk;  // 16
constexpr int kPairMaxCpi = 16;                           // j-chunks per work item, at most
constexpr int kPairStage = 8;                             // chunks staged at a time (8 KB)
static_assert(kPairMaxCpi <= kPairBlockChunks && kPairBlockChunks % kPairMaxCpi == 0,
              "chunks per item must divide the chunks of an i-block");
}  // namespace gi
// Far-field sums of every body of the table's runs into a.fsum_fx (which
// must be zero on entry), and with_rows the row path's corrections into delta
// (the grid must be built); then the epilogue, as gi_launch_finish.
struct GridWork;
cudaError_t gi_launch_pair_force(const ForceArgs &a, const LaunchTable &tab, const GridWork &g,
                                 long long *delta, const unsigned int *ctr, bool with_rows,
                                 bool early, cudaStream_t s);
// Pair potentials of the table's runs, one double per run in out, in table order.
// First the runs planned as for gi_launch_pair_force (tab.nitems CTAs), then the
// short ones (pipl 0; tab.rows blocks from row_start on); each run has nsplit
// partials from item_start on (the former a CTA for each).
constexpr int kPotentialPartials = 262144;  // of a run, at most (2 MB)
cudaError_t gi_launch_potential(const float4 *pos, const LaunchTable &tab, double *partials,
                                double *out, cudaStream_t s);
// The kernels' own decode of a task (CTA) of a run planned by gi_internal_pair_run: its
// first row and chunks [c0, c1); returns the run's tasks.
long long gi_pair_task(const RunDev &R, long long task, int *row, int *c0, int *c1);
cudaError_t gi_launch_pair_finish(int epi, const ForceArgs &a, const LaunchTable &tab, int maxn,
                                  int nsm, bool early, cudaStream_t s);

// gi_grid.cu: contact corrections of every body of the table's runs into
// delta (3 x int64 per body) through a cell grid.  Its scratch layout
// is computed here, as constexpr functions, so that gi_noalloc.cu can check
// at compile time that its static array holds the largest run it accepts.
namespace gi {
// A bucket goes through the tiled path only when it holds at least this many
// bodies; that bounds the number of tiled buckets and work items.
constexpr unsigned int kDenseFloor = 32;
// Bodies of a cell from which it goes that way unless gi_options.dense_min says
// otherwise.  A row-path warp with the cells of a body's dense core around it
// (no more than 180 bodies each there) runs 100 us longer than the others; ms a
// step at 64, 128, 192 and 256: the 66,000-body impact settled 1.052, 1.050,
// 1.090, 1.131, after 6,000 steps 1.620, 1.619, 1.630, 1.763.  (48: 1.092.)
constexpr int kDenseMin = 128;
// Cost classes of the tiled path's work items (128-body tiles staged - 1).
constexpr unsigned int kItemClasses = 16;
// Tiled-path counters: items, tiled buckets, queue head, candidate buckets,
// then a count and a fill cursor per cost class, then a bit per run.
constexpr int kCtrWords = 4 + 2 * (int)kItemClasses + GI_MAX_RUNS / 32;
// Runs of at most kDirectMax bodies take no grid (every body of the run is a
// candidate) where all such runs of a table together have at most kDirectCandidates
// candidates, one run of 3,648, whose row CTAs are what the GPU holds at once; in
// fuller tables those of at most kDirectAlways.  The candidates of a full GPU cost
// more than a grid build, whose launches are what a lone short run spends its step
// on.  us a step of settled bodies, without a grid / with one: one run of 2,000 13 /
// 33, 3,000 26 / 30, 3,600 35 / 30 (a remnant 64 / 75), 4,000 40 / 30 (101 / 81); two
// of 3,000 41 / 32; eight of 1,000 28 / 30, 2,000 72 / 52; 24 of 500 27 / 39, 1,000 65
// / 56, 2,000 200 / 102; 64 of 500 60 / 79, 1,000 160 / 95, 4,000 1,757 / 480.  Beside
// the one-sided far field, where the grid-wide kernels build the grid: one of 4,000
// 41 / 66, 24 of 1,000 60 / 78, eight of 2,000 72 / 86, 24 of 2,000 182 / 128.
constexpr int kDirectMax = 4096, kDirectAlways = 512;
constexpr long long kDirectCandidates = 3648 * 3648, kDirectCandidatesOneSided = 40000000;
// Runs below it have their grid built by a cluster of 8 CTAs, larger ones by 16.
constexpr int kClusterSmallMax = 65536;
// Bodies of a row-path CTA (one warp), of a run with a grid and without.
constexpr int kRowBodies = 8, kDirectBodies = 2;
}  // namespace gi

// Buckets of the grid for `bodies` bodies: a power of two >= 2 * bodies.
constexpr unsigned int gi_grid_buckets(long long bodies)
{
    unsigned long long m = 1024;
    while (m < 2ull * (unsigned long long)bodies) m <<= 1;
    return (unsigned int)m;
}

// Tiled-path work items: at most 27 per chunk of 128 bodies of a dense
// bucket, and a dense bucket holds at least kDenseFloor bodies, so at most
// 27 (bodies / 128 + bodies / kDenseFloor + 2).  Tiled buckets: each holds at
// least kDenseFloor bodies.
constexpr size_t gi_dense_item_capacity(long long bodies)
{
    return 27 * ((size_t)bodies / 128 + (size_t)bodies / gi::kDenseFloor + 2);
}
constexpr size_t gi_dense_bucket_capacity(long long bodies)
{
    return (size_t)bodies / gi::kDenseFloor + GI_MAX_RUNS;  // each run rounds up
}

// Words of grid scratch: the slots' positions and velocities, and a second,
// sub-cell ordered copy of the tiled buckets' (16 words per body); items as
// listed and as ordered (4 words each); candidate and tiled buckets (2 words
// each); bucket starts (one word per bucket and one more) and states; block
// sums: 9216; keys and ranks of the grid-wide build (indexed by global body).
constexpr size_t gi_grid_words(long long max_end, long long bodies)
{
    return 16 * (size_t)bodies + 8 * gi_dense_item_capacity(bodies) +
           4 * gi_dense_bucket_capacity(bodies) + 2 * (size_t)gi_grid_buckets(bodies) + 1 + 9216 +
           2 * (size_t)max_end;
}
// What the row path reads of it.
struct GridView {
    const float4 *spos, *svel, *dpos;
    const unsigned int *start, *state, *ctr;
};
// The scratch of one table's contact pass, carved from `work` (16-byte
// aligned): 16-byte words first, then single words (see gi_grid_words).
struct GridWork {
    float4 *spos, *svel, *dpos, *dvel;
    uint4 *raw, *items;
    uint2 *cand, *tiled;
    unsigned int *start, *state, *sums, *keys, *ranks;
    size_t icap, bcap;
    unsigned int buckets;
    GridWork(unsigned int *work, long long bodies, int max_end)
    {
        buckets = gi_grid_buckets(bodies);
        icap = gi_dense_item_capacity(bodies);
        bcap = gi_dense_bucket_capacity(bodies);
        spos = reinterpret_cast<float4 *>(work);
        svel = spos + bodies;
        dpos = svel + bodies;
        dvel = dpos + bodies;
        raw = reinterpret_cast<uint4 *>(dvel + bodies);
        items = raw + icap;
        cand = reinterpret_cast<uint2 *>(items + icap);
        tiled = cand + bcap;
        start = reinterpret_cast<unsigned int *>(tiled + bcap);
        state = start + buckets + 1;
        sums = state + buckets;
        keys = sums + 9216;
        ranks = keys + max_end;
    }
    GridView view(const unsigned int *ctr) const
    {
        return GridView{spos, svel, dpos, start, state, ctr};
    }
};
// Sets the grid and row fields of the table and its runs; candidates: what its runs
// without a grid may have.
void gi_grid_runs(LaunchTable &tab, long long candidates = gi::kDirectCandidates);
// The contact pass, in this order: the grid (with the tiled path's work
// items); the row path, here or in gi_launch_pair_force, and the tiled path.
// delta receives every body's correction.  ctr: gi::kCtrWords words, zero on
// entry of the first.  clusters: CTAs of the largest thread-block cluster that may
// build a run's grid (see grid_cluster_kernel): 8 for runs below 65,536 bodies, 16
// below 131,072 (gi_grid_cluster_ctas), 0 for none.
cudaError_t gi_launch_grid(const float4 *pos, const float4 *vel, const LaunchTable &tab,
                           const GridWork &g, long long *delta, unsigned int *ctr, int nsm,
                           int clusters, cudaStream_t s);
// Asks leave for clusters of 16 CTAs in the current CUDA context, which is where
// that is kept (gone with cudaDeviceReset): 16, or 8 where they are not available.
int gi_grid_cluster_ctas();
cudaError_t gi_launch_rows(const float4 *pos, const float4 *vel, const LaunchTable &tab,
                           const GridWork &g, long long *delta, const unsigned int *ctr,
                           cudaStream_t s);
cudaError_t gi_launch_tiles(const LaunchTable &tab, const GridWork &g, long long *delta,
                            unsigned int *ctr, int nsm, bool early, cudaStream_t s);

// Waits for the kernels this one was launched to follow (see gi_launch).
__device__ __forceinline__ void launch_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a kernel whose blocks begin with launch_wait().  early: its blocks
// may be put on the GPU when the last of the stream's previous kernel have
// left it, before its writes are all in place (what launch_wait waits for).  A
// kernel that depends on the one before it starts 2 us sooner: forces of 1,500
// bodies, two kernels, 14.5 -> 10.9 us; a step of 4,200 settled ones, four,
// 47.8 -> 40.4.  Not for work that shares the GPU with another stream's:
// blocks that wait hold their registers.
template <class... P, class... A>
inline cudaError_t gi_launch(void (*kernel)(P...), dim3 grid, int threads, bool early, cudaStream_t s,
                             A &&...args)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// The largest shared-memory carveout for a kernel, in the current CUDA context.
// Kernels that are to share an SM need the same one: an SM changes its carveout
// only when it is empty.
inline cudaError_t gi_full_carveout(const void *kernel)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared);
}
// That for the paired far field's kernel and for the contact kernels; a gi_ctx does
// it when it is created, and gi_force_carveout and gi_grid_cluster_ctas when a call
// first needs them (it is gone with cudaDeviceReset).
cudaError_t gi_pair_setup();
cudaError_t gi_contact_setup();

// gi_aux.cu
cudaError_t gi_launch_move(float4 *pos, float4 *vel, const float4 *force,
                           const LaunchTable &tab, cudaStream_t s);
// The FP64 diagnostics' resident blocks on sm_count SMs.
int gi_diag_blocks(int sm_count);
// The point that the angular momentum's terms are taken about (position, then
// velocity); not given: a body of the scope.
struct DiagOrigin {
    float x[6];
    bool given;
};
// work holds 16 doubles per block, out kDiagOut doubles (device, or pinned
// host memory), ticket an int that is zero between launches.
constexpr int kDiagOut = 22;
cudaError_t gi_launch_diag(const float4 *pos, const float4 *vel,
                           const unsigned char *label, int scope,
                           const RunDev &run, float mass_fe, float mass_si, double *work,
                           const DiagOrigin &origin, int max_blocks, double *out, int *ticket,
                           cudaStream_t s);
cudaError_t gi_launch_ffma_peak(float *sink, int blocks, int iters, cudaStream_t s);

// gi_api.cu helpers for the library's other translation units: record an
// error for gi_last_error() and return `status`; the device pair table of a
// reference collision struct.
int gi_internal_fail(int status, const char *msg);
int gi_internal_collision_pairdev(const gi_force_collision_consts *c, PairDev *d);
// Device scratch bytes one run of n bodies needs in `ctx` (admission estimate).
long long gi_internal_scratch_bytes(gi_ctx *ctx, int n);
// The paired far field's decomposition of one run of n bodies with 2^pcl
// j-chunks per work item, its CTAs numbered from item_start: fills the run's
// pcl ... far_inv and item_start, returns its CTAs.  ipl: log2 of the rows a
// lane holds (0: the far field's choice).
long long gi_internal_pair_run(RunDev &d, int n, int pcl, const PairDev &p, long long item_start,
                               int ipl = 0);
// log2 of the j-chunks per item of a run of n bodies without a tuning table.
int gi_internal_pair_default_pcl(int n);
// The same of the potential (gi_potential_fp64), all rows eight to a lane.
int gi_internal_potential_pcl(int n);
// Device ordinal of a context (-1 for NULL).
int gi_internal_ctx_device(gi_ctx *ctx);
// The context's workspace of at least `bytes` device bytes (16-byte aligned)
// and a pinned page of kPinnedBytes, for calls that wait for the GPU before
// they return: it is idle between calls, whatever stream they run on.  Kept
// until the context is destroyed; grown, never shared between contexts.
constexpr size_t kPinnedBytes = 4096;
int gi_internal_ctx_workspace(gi_ctx *ctx, size_t bytes, void **dev, void **pinned);
// Attempts one union-find link of gi_find_earth_moon may make (gi_options).
int gi_internal_ctx_cluster_tries(gi_ctx *ctx);
