// fj_internal.h -- launch interface between the C-ABI layer and the kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "fj_device.cuh"

struct fj_ctx;
struct fj_quad_rule;

namespace fj {

struct DeferWork;  // scratch of the mixed form's FP64 pass (below)
constexpr int kMomentBlock = 128;  // threads per block of the phase-space kernel
// Device counters of one call (fj_moment_stats): nodes with H < 0, nodes whose
// action solve still hit a cap (any kind), Poisson integrals that hit theirs,
// nodes whose turning points ran in FP64 (mixed form), the final failures by
// kind (a node can count in several), and mixed-form nodes re-solved by the
// plain FP64 solve because their FP32 solve hit a cap.
enum : int {
    kCntBound = 0, kCntFailed = 1, kCntPoisson = 2, kCntEscalated = 3,
    kCntFailQuad = 4, kCntFailBracket = 5, kCntFailRoot = 6, kCntResolved64 = 7, kNumCounters = 8
};
constexpr int kPlainChunk = 1024;  // most velocity nodes of one point per work item (FP64 form)
// Nodes per work item of a model of npts points, nq3 nodes each: as large as
// possible (a long node list keeps the lanes of a block busy to its end) while
// there are enough items to fill the GPU and balance their uneven cost.  By the
// model's own size alone, so that a batched launch sums in the same order.
constexpr int kPlainItems = 1216;  // 8 per SM of 152 (a constant: the sums keep their order on any device)
// Mixed form: twice the blocks of its kernels (24x8 model: 9.9 ms with 1536 items
// of 512 nodes, 8.1 ms with 3072 of 256; 80x40: 138 ms with 1024-node items, more
// with shorter or longer ones)
constexpr int kMixedItems = 2432;
inline int plain_chunk(long long npts, long long nq3, int most = kPlainChunk, int items = kPlainItems)
{
    int c = most;
    while (c > 128 && npts * ((nq3 + c - 1) / c) < items) c = c / 2 < 128 ? 128 : c / 2;
    return c;
}
// per-thread stack floor: the function attributes do not report the frames of the
// device functions a kernel calls (4.1 KB at most, by ptxas' "cumulative
// stack size")
constexpr size_t kStackBytes = 8192;

// Arguments of the phase-space (moment) kernel.  All pointers are device memory.
struct MomentArgs {
    PotView P;
    const double *Eg, *Dg;
    int ngrid;
    const double *xq, *wq;   // velocity rule [nq]
    int nq;
    GLRule gl;               // momentum-integral rule (n = 0: QAGS)
    DFDev df;
    const double *ci;        // grid mode: ngauss polar GL nodes on (0,1); else NULL
    int ngauss;
    const double *Rz;        // point mode: [npts][2]; else NULL
    int npts;
    int blocks_per_point;
    int plain_chunk;         // FP64 form: nodes per work item (<= kPlainChunk)
    const double2 *trig;     // sines and cosines of the FP64 quadrature angles (launch_trig_table)
    int mixed_chunk;         // mixed form: nodes per block (<= kMixedMaxNodes)
    float *jout;             // mixed form, optional: (Jr, Jz) of every bound node [npts][nq^3][2]
    double *partial;         // [npts][blocks_per_point][6]
    unsigned *defer;         // mixed form: [npts * blocks_per_point][mixed_chunk / 32] bitmaps of the nodes
                             // left to the FP64 pass
    int *defer_count;        // mixed form: [npts * blocks_per_point] how many nodes each block left
    unsigned long long *counters;  // [kNumCounters], the slots below
    double *out6;            // [6][npts]
};

// Work queue and scratch of a persistent FP64 launch (k_moments, k_los,
// k_actions): items 0 .. total-1 from a device counter that the launch zeroes,
// scratch of per_block bytes for each of its blocks
struct PlainWork {
    unsigned *next;
    char *scratch;
    size_t per_block;
    int total, grid;
};
// whether the FP64 kernels stage the radial derivative in shared memory too (16 KB)
FJ_HD bool grad_staged(int nr, int npoly) { return (long long)nr * npoly <= 2048; }
size_t plain_scratch_bytes(int chunk);  // per block, for items of at most chunk points
// Blocks of a kernel that the current device holds at once, with `threads` threads and
// `smem` bytes of dynamic shared memory each; 0 if not one fits.  More than 48 KB (the
// static part included) needs an opt-in, a limit that belongs to the kernel in the
// whole process: it is only ever set to the device's maximum, so that a thread with
// a small model cannot lower it between another's call of this and its launch.
int resident_blocks(const void *kernel, int threads, size_t smem);
int sm_count();  // of the current device; 0 if there is none
int moments_resident(size_t smem);
int los_resident(size_t smem);
int actions_resident(size_t smem);
// the table of MomentArgs::trig, kTrigTableEntries entries
constexpr size_t kTrigTableEntries = 2 * 1024 * 21;
cudaError_t launch_trig_table(double2 *trig, cudaStream_t s);

// Projected density, line profiles and velocity distributions (fj_los.cu):
// n values at Rzv [n][3] (R, z, v) of one kind (FJ_LOS_*), on m's potential,
// focal-distance table, [-1,1] rule and DF, with the 22-point [0,1] table
constexpr int kLos01 = 22;
struct LosArgs {
    MomentArgs m;
    const double *rhl;  // [nr*npoly] density multipoles (SigmaDF)
    int kind;
    const double *Rzv;
    int n;
    double *out;        // [n]
    double x01[kLos01], w01[kLos01];
    int blocks_per_item;  // blocks sharing one value's nodes (kLosChunk nodes each)
    double *partial;      // [n][blocks_per_item] block sums, added in order by k_los_finalize
};
constexpr int kLosChunk = 1024;  // most nodes of one value per work item
size_t los_smem_bytes(const MomentArgs &m);
cudaError_t launch_los(const LosArgs &a, const PlainWork &w, cudaStream_t s);
int los_nodes(int kind, int nq);  // a value's nodes
size_t los_local_bytes();

// Focal-distance tables of n models (fj_delta.cu): one thread per (model,
// energy); pots, Eg, Dg device arrays [n] (tables [ngrid] each), bad device [n]
// (set to 1 where a bracket or root search hit its cap)
cudaError_t launch_tabulate_delta(const PotView *pots, double *const *Eg, double *const *Dg, int n, int ngrid,
                                  int *bad, cudaStream_t s);
size_t delta_local_bytes();

// Several models' phase-space launches in one grid: model m owns blocks
// [block_start[m], block_start[m+1]) and grid points [point_start[m],
// point_start[m+1]) of the batched finalize.  All pointers are device memory;
// n = 0: a single launch described by the kernel's MomentArgs parameter.
struct MomentBatch {
    const MomentArgs *args;
    const int *block_start, *point_start;
    int n;
};

// per-node status tallies of one thread: nodes with any cap, and by kind
struct FailTally {
    unsigned any = 0, quad = 0, bracket = 0, root = 0;
    __device__ __forceinline__ void add(unsigned fail)
    {
        any += fail ? 1u : 0u;
        quad += (fail & kFailQuad) ? 1u : 0u;
        bracket += (fail & kFailBracket) ? 1u : 0u;
        root += (fail & kFailRoot) ? 1u : 0u;
    }
};

// adds a warp's values of v to *ctr (one atomic per warp, none for a zero sum);
// every lane of the warp must call it
__device__ __forceinline__ void warp_count(unsigned long long *ctr, unsigned v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(ctr, (unsigned long long)v);
}

__device__ __forceinline__ void warp_count_fails(unsigned long long *counters, const FailTally &t)
{
    warp_count(&counters[kCntFailed], t.any);
    warp_count(&counters[kCntFailQuad], t.quad);
    warp_count(&counters[kCntFailBracket], t.bracket);
    warp_count(&counters[kCntFailRoot], t.root);
}

// the model of block (or point) `i` of a batch: largest m with start[m] <= i
__device__ __forceinline__ int batch_model(const int *start, int n, int i)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

size_t moment_smem_bytes(const MomentArgs &a);
cudaError_t launch_moments(const MomentArgs &a, const PlainWork &w, cudaStream_t s);
// Work queue and workspace of the mixed form's persistent kernels.  Item i is
// block order[i] (order NULL: block i) of the launch's layout; cost[b] receives
// block b's cycles.  The launch goes through its items in slices of per_slice,
// whose nodes' records fit the workspace.
struct ItemQueue {
    unsigned *next;    // [2] device counters, zeroed by the launch
    const int *order;  // [total] or NULL
    float *cost;       // [total] or NULL
    char *scratch;     // mixed_scratch_bytes() for each of the `grid` blocks
    char *rec;         // [per_slice][stride] node records (mixed_rec_bytes() each)
    double *point;     // [per_slice][4] R, z, Phi, escape speed of the items' points
    int *nbound;       // [per_slice] bound nodes of the items
    int stride;        // most nodes of an item
    int total, per_slice;
    int grid_turn, grid;        // blocks of the two kernels,
    size_t smem_turn, smem;     // their dynamic shared memory
    bool far_turn, far_integrate;  // and whether their tables are in device memory (mixed_place):
    float *far;                    // far_floats for each block
    size_t far_floats;
    int first, count;     // the slice (set per launch)
};
// What a model needs with near and with far tables: dynamic shared memory of the two
// kernels, floats per block in device memory
struct MixedSize {
    size_t turn[2] = {0, 0}, integrate[2] = {0, 0}, far = 0;
    void cover(const MixedSize &o)  // both models in one launch
    {
        for (int p = 0; p < 2; p++) {
            turn[p] = turn[p] > o.turn[p] ? turn[p] : o.turn[p];
            integrate[p] = integrate[p] > o.integrate[p] ? integrate[p] : o.integrate[p];
        }
        far = far > o.far ? far : o.far;
    }
};
MixedSize mixed_size(const MomentArgs &a);
// where the launch's tables go (q.total set), and its grids; false: they do not fit either way
bool mixed_place(int variant, int np, const MixedSize &z, ItemQueue &q);
// a batch: nblocks = items of all models, smem = the largest model's (FP64 form)
cudaError_t launch_moments_batch(const MomentArgs &a0, const MomentBatch &b, int nblocks, size_t smem, bool mixed,
                                 int variant, int np, const DeferWork &dw, const ItemQueue &q, const PlainWork &w,
                                 cudaStream_t s);
cudaError_t launch_moments_finalize_batch(const MomentBatch &b, int npoints, cudaStream_t s);
// dst6[q][idx[t]] = src6[q][t] (moments of n points into a grid of npts)
cudaError_t launch_scatter6(int n, const int *idx, const double *src6, int npts, double *dst6, cudaStream_t s);
// the per-point sums of the block partials (shared by both forms)
cudaError_t launch_moments_finalize(const MomentArgs &a, cudaStream_t s);
// mixed-precision form (FJ_PREC_MIXED, double-power-law DF, QAGS momentum
// integrals); counters[3] gets the nodes whose turning points ran in FP64
constexpr int kMixedBlock = 128;     // threads per block of the mixed kernel
// A mixed-form node whose FP32 solve hits a cap is not re-solved in the block
// (one FP64 solve would hold its warp and block for as long as hundreds of FP32
// ones): its block marks it in a bitmap of its node range, leaves it out of its
// sums and records how many it left.  The FP64 pass (launch_deferred) then lists
// every launch's left nodes compactly, block by block in node order (an
// exclusive scan of the counts gives each block its offset), solves them all in
// parallel, a block of two warps per node, and adds each item's nodes to its
// partial sums in list order: the same sums whatever order the blocks ran in.
struct DeferWork {
    int *count;      // [nblocks] the blocks' counts (the launch's defer_count arrays, in block order)
    int *offset;     // [nblocks] exclusive prefix of the blocks' counts
    int *chunk_sum;  // [nblocks / kScanChunk + 2] scan carries; [nchunks] = the launch's total
    int *node;       // [cap] listed nodes (index within the point's nq^3 rule)
    int *block;      // [cap] global block index of each listed node
    double *mom;     // [cap][6] moment contributions of the listed nodes
    int cap;         // list capacity; nodes beyond it are solved item by item
};
constexpr int kScanChunk = 1024;  // blocks per chunk of the count scan
constexpr int kMixedMaxNodes = 8192; // largest node range of one block (shared-memory list)
FJ_HD int defer_words(int chunk) { return (chunk + 31) / 32; }  // bitmap words of one block
constexpr int kMixedVariants = 8;    // configurations of the mixed kernels (2 turning-point x 4 integral builds)
size_t mixed_rec_bytes();      // per node of a slice
size_t mixed_scratch_bytes();  // per block of the integration kernel
// nodes whose records a workspace holds: 2.2 GB of records at most per context
constexpr long long kMixedSliceNodes = 20ll << 20;
int mixed_blocks_per_point(long long nq3, int chunk);
cudaError_t launch_moments_mixed(const MomentArgs &a, int variant, const DeferWork &dw, const ItemQueue &q,
                                 cudaStream_t s);

// Points per work item of the action batch: whole rounds of two blocks per SM, items of
// a warp at least (20 001 points on 152 SMs: 10.2 ms in items of 32, two rounds of
// which the second is nearly empty; 6.0 ms in one round of items of 66)
constexpr int kActionChunk = 256;
inline int action_chunk(size_t n, int sms)
{
    const size_t blocks = 2 * (size_t)(sms > 0 ? sms : 1), most = blocks * kActionChunk, rounds = (n + most - 1) / most;
    const size_t c = (n + blocks * rounds - 1) / (blocks * rounds);
    return (int)(c < 32 ? 32 : c);
}
size_t actions_smem_bytes(int nr, int npoly, int ngrid);
cudaError_t launch_actions(PotView P, const double *Eg, const double *Dg, int ngrid, GLRule gl, const double2 *trig,
                           const double *pts, size_t n, int chunk, double *out, const PlainWork &w, cudaStream_t s);
cudaError_t launch_potential_eval(PotView P, const double *Rz, size_t n, double *out, cudaStream_t s);

// projection: poly [npoly][ngauss] = 2 P_2l(c_g) w_g
cudaError_t launch_project(int nr, int ngauss, int npoly, const double *ar, const double *poly,
                           const double *grids6, double *coef6, cudaStream_t s);
// Poisson: a warp per radial integral, QAGS interval lists of kPoissonCap entries in
// shared memory (no device workspace)
constexpr int kPoissonCap = 256;
cudaError_t launch_poisson(int nr, int npoly, const double *ar, const double *rhl, double *phil,
                           double *Pr, double *Pr2, unsigned long long *counters, cudaStream_t s);
// Poisson with the radial integrals taken exactly over the linear interpolation
// of the density multipoles (prefix sums, no adaptive quadrature): one block per l
constexpr int kPoissonCumulativeMaxNr = 4096;
cudaError_t launch_poisson_cumulative(int nr, int npoly, const double *ar, const double *rhl, double *phil,
                                      double *Pr, double *Pr2, cudaStream_t s);
cudaError_t launch_sum3(int n, const double *a0, const double *a1, const double *a2, const double *b0,
                        const double *b1, const double *b2, double *o0, double *o1, double *o2, cudaStream_t s);
// o = a + b elementwise (summed component densities)
cudaError_t launch_add(int n, const double *a, const double *b, double *o, cudaStream_t s);
// vir2: ci, wi = ngauss polar nodes/weights on (0,1); out7 device
cudaError_t launch_vir2(PotView P, int ngauss, const double *ci, const double *wi, const double *coef6,
                        double *out7, cudaStream_t s);

// the stream a context orders its work on; the device copies of a grid's polar
// nodes and of a velocity rule
cudaStream_t context_stream(::fj_ctx *ctx);
int context_grid_inputs(::fj_ctx *ctx, int ngauss, const struct ::fj_quad_rule *rule, const double **ci,
                        const double **xq, const double **wq);
// BF16 tensor-core GEMM (fj_mlp.cu): C = A B^T with a fused epilogue
namespace tc { struct Epilogue; }
cudaError_t launch_gemm_tc(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K,
                           int ksplit, const tc::Epilogue &ep, cudaStream_t s);

// largest per-thread local memory (stack) any kernel of the library needs
size_t moments_local_bytes();
size_t moments_mixed_local_bytes();
size_t multipole_local_bytes();
size_t poisson_local_bytes();  // per-thread local memory (stack) of the Poisson kernel

}  // namespace fj
