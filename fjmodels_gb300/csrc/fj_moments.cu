// fj_moments.cu -- the FP64 phase-space kernel: the Staeckel-fudge actions of
// every (meridional point, velocity node), the DF and the six velocity moments;
// plus the batched action and potential kernels.
//
// Work unit: node q = (i, j, k) of the nq^3 tensor rule (integ/GaussQuad.cpp:
// 160-180), velocity V = 1e-6 + Ve*(x_i, x_j, x_k) (integ/Integ.cpp:46-62).
// A work item is a range of at most kPlainChunk consecutive nodes of one point;
// a persistent block compacts its bound ones (H < 0) into a shared list, orders
// it by the cost proxy of fj_order.cuh, solves the list's orbits together
// (fj_solve64.cuh), and thread t sums the moments of entries t, t + 128, .. in
// order.  The per-item sums go to a scratch array and a second kernel adds them
// in a fixed order, so results are deterministic run to run.
#include <algorithm>
#include <cstdint>

#include "fj_internal.h"
#include "fj_order.cuh"
#include "fj_solve64.cuh"

namespace fj {

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

static_assert(kTrigTableEntries == 2 * kTrigPanels * 21, "trig table size");
static_assert(sizeof(SolveShared::vals) >= kPlainChunk * sizeof(float), "the cost keys share the panel values' memory");
static_assert(kMomentBlock == kSolveBlock, "the moment blocks run the orbit solver");

size_t plain_scratch_bytes(int chunk) { return (solve_scratch_bytes(chunk) + 255) / 256 * 256; }

// panels of the bisection trees of [0, pi] (Ju) and [0, pi/2] (Jv): interval
// `heap` by halving from the root, as the quadrature does
__global__ void k_trig_table(double2 *trig)
{
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kTrigTableEntries) return;
    const bool kv = t >= kTrigTableEntries / 2;
    const unsigned heap = (t / 21) % kTrigPanels;
    const int e = t % 21;
    if (heap == 0) { trig[t] = make_double2(0., 0.); return; }
    double a = 0., b = kv ? kPIH : kPI;
    for (int bit = 30 - __clz((int)heap); bit >= 0; bit--) {
        const double m = 0.5 * (a + b);
        if ((heap >> bit) & 1u) a = m; else b = m;
    }
    double sn, cs;
    sincos(gk_abscissa<21>(a, b, e), &sn, &cs);
    trig[t] = make_double2(sn, cs);
}

cudaError_t launch_trig_table(double2 *trig, cudaStream_t s)
{
    k_trig_table<<<(unsigned)((kTrigTableEntries + 127) / 128), 128, 0, s>>>(trig);
    return cudaGetLastError();
}

// shared memory of a model's tables: radii, potential, the integrands' tables,
// interpolation constants, focal distances, velocity and momentum rules, and of
// small models the radial derivative (the second one, which only the
// quasi-isothermal DF reads, stays in device memory)
static size_t table_doubles(int nr, int npoly, int ngrid, int nq, int ngl)
{
    return nr + (size_t)nr * npoly * (grad_staged(nr, npoly) ? 2 : 1) + fast_table_size(nr, npoly) + interp_table_size(nr) +
           2 * ngrid + 2 * nq + 2 * ngl;
}

size_t moment_smem_bytes(const MomentArgs &a)
{
    const size_t nd = table_doubles(a.P.nr, a.P.npoly, a.ngrid, a.nq, a.gl.n);
    return nd * sizeof(double) + 6 * (kMomentBlock / 32) * sizeof(double) + 4 * sizeof(double) + sizeof(SolveShared) +
           kPlainChunk * sizeof(unsigned short) + (kMomentBlock / 32) * sizeof(int) + 16;
}

__global__ void __launch_bounds__(kMomentBlock, 2) k_moments(MomentArgs a0, MomentBatch batch, PlainWork work)
{
    extern __shared__ double sm[];
    __shared__ int s_item;
    int model = -1;  // whose tables are in shared memory
    for (;;) {
        __syncthreads();  // every thread is done with the previous item's shared data
        if (threadIdx.x == 0) s_item = (int)atomicAdd(work.next, 1u);
        __syncthreads();
        int bid = s_item;
        if (bid >= work.total) return;
        int m = 0;
        if (batch.n > 0) {
            m = batch_model(batch.block_start, batch.n, bid);
            bid -= batch.block_start[m];
        }
        const MomentArgs &a = batch.n > 0 ? batch.args[m] : a0;
        const int nr = a.P.nr, npoly = a.P.npoly, nt = nr * npoly;
        const bool grad = grad_staged(nr, npoly);
        double *s_ar = sm, *s_phil = s_ar + nr, *s_Pr = s_phil + nt, *s_fast = grad ? s_Pr + nt : s_Pr,
               *s_it = s_fast + fast_table_size(nr, npoly);
        double *s_Eg = s_it + interp_table_size(nr), *s_Dg = s_Eg + a.ngrid,
               *s_xq = s_Dg + a.ngrid, *s_wq = s_xq + a.nq;
        double *s_glx = s_wq + a.nq, *s_glw = s_glx + a.gl.n, *s_red = s_glw + a.gl.n;
        double *s_pt = s_red + 6 * (kMomentBlock / 32);
        SolveShared *s_solve = (SolveShared *)(s_pt + 4);
        float *s_key = (float *)s_solve->vals;  // until the solves
        unsigned short *s_list = (unsigned short *)(s_solve + 1);
        int *s_wc = (int *)(((uintptr_t)(s_list + kPlainChunk) + 15) & ~(uintptr_t)15);
        if (m != model) {
            model = m;
            for (int i = threadIdx.x; i < nr; i += blockDim.x) s_ar[i] = a.P.ar[i];
            for (int i = threadIdx.x; i < nt; i += blockDim.x) {
                s_phil[i] = a.P.phil[i];
                if (grad) s_Pr[i] = a.P.Pr[i];
            }
            for (int i = threadIdx.x; i < a.ngrid; i += blockDim.x) { s_Eg[i] = a.Eg[i]; s_Dg[i] = a.Dg[i]; }
            for (int i = threadIdx.x; i < a.nq; i += blockDim.x) { s_xq[i] = a.xq[i]; s_wq[i] = a.wq[i]; }
            for (int i = threadIdx.x; i < a.gl.n; i += blockDim.x) { s_glx[i] = a.gl.x01[i]; s_glw[i] = a.gl.w01[i]; }
            __syncthreads();
            interp_table(nr, s_ar, s_it, threadIdx.x, blockDim.x);
            __syncthreads();
            fast_tables(PotView{nr, npoly, s_ar, s_phil, s_Pr, a.P.Pr2, s_it}, s_fast);
            __syncthreads();
        }
        const PotView P{nr, npoly, s_ar, s_phil, grad ? s_Pr : a.P.Pr, a.P.Pr2, s_it};
        const PotFast F{nr, npoly, s_ar, s_phil, s_fast, s_fast + nt, s_it};
        const GLRule gl{a.gl.n, s_glx, s_glw};
        const int B = a.blocks_per_point;
        const int p = bid / B, chunk = bid % B;
        const int nq = a.nq, nq2 = nq * nq, nq3 = nq2 * nq;
        const int n0 = chunk * a.plain_chunk, n1 = min(n0 + a.plain_chunk, nq3);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (threadIdx.x == 0) {  // the point (integ/Integ.cpp:150-151)
            double R, z;
            if (a.Rz) { R = a.Rz[2 * p]; z = a.Rz[2 * p + 1]; }
            else {
                const int n = p / a.ngauss, g = p % a.ngauss;
                const double c = a.ci[g], si = sqrt(1 - c * c);
                R = s_ar[n] * si; z = s_ar[n] * c;
            }
            const double Phi_h = pot_phi(P, R, z), rmax = s_ar[nr - 1];
            s_pt[0] = R; s_pt[1] = z; s_pt[2] = Phi_h;
            s_pt[3] = sqrt(-2 * (Phi_h - pot_phi(P, 10 * rmax, 10 * rmax)));
        }
        __syncthreads();
        const double R = s_pt[0], z = s_pt[1], Phi_h = s_pt[2], Ve = s_pt[3];
        auto velocity = [&](int node, double &V0, double &V1, double &V2) {
            V0 = 1e-6 + Ve * s_xq[node / nq2]; V1 = 1e-6 + Ve * s_xq[(node / nq) % nq]; V2 = 1e-6 + Ve * s_xq[node % nq];
        };
        // bound nodes of [n0, n1) in node order
        int nbound = 0;
        for (int base = n0; base < n1; base += kMomentBlock) {
            const int node = base + threadIdx.x;
            bool b = false;
            if (node < n1) {
                double V0, V1, V2;
                velocity(node, V0, V1, V2);
                b = .5 * (V0 * V0 + V1 * V1 + V2 * V2) + Phi_h < 0;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, b);
            if (lane == 0) s_wc[warp] = __popc(bal);
            __syncthreads();
            int off = nbound, tot = 0;
            for (int w = 0; w < kMomentBlock / 32; w++) {
                if (w < warp) off += s_wc[w];
                tot += s_wc[w];
            }
            if (b) s_list[off + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)(node - n0);
            __syncthreads();
            nbound += tot;
        }
        for (int q = threadIdx.x; q < nbound; q += kMomentBlock) {
            const int node = n0 + s_list[q];
            s_key[q] = node_cost_key((float)s_xq[node / nq2], (float)s_xq[(node / nq) % nq], (float)s_xq[node % nq]);
        }
        sort_list(s_list, s_key, nbound);
        // the orbits of the list
        const SolveScratch S = solve_scratch(work.scratch + blockIdx.x * work.per_block, kPlainChunk);
        solve_orbits64(P, F, gl, a.trig, nbound, S, *s_solve,
                       [&](int q, double &Delta, double &R_, double &z_, double &Phi_, double &V0, double &V1, double &V2) {
                           velocity(n0 + s_list[q], V0, V1, V2);
                           const double H = .5 * (V0 * V0 + V1 * V1 + V2 * V2) + Phi_h;
                           Delta = deltafn(s_Eg, s_Dg, a.ngrid, H);
                           R_ = R; z_ = z; Phi_ = Phi_h;
                       });
        FailTally tally;
        double mm[6] = {0, 0, 0, 0, 0, 0};
        const double jacob = Ve * Ve * Ve;
        for (int q = threadIdx.x; q < nbound; q += kMomentBlock) {
            const int node = n0 + s_list[q];
            double V0, V1, V2;
            velocity(node, V0, V1, V2);
            const OrbitRec &o = S.rec[q];
            unsigned fail = o.status();
            double DF = df_value(a.df, P, R, o.Jr, o.Jz, R * V1, fail);
            if (fail & (kFailBracket | kFailRoot)) DF = 0.;
            tally.add(fail);
            const double w = s_wq[node / nq2] * s_wq[(node / nq) % nq] * s_wq[node % nq];
            const double jd = jacob * DF;
            mm[0] += w * jd;
            mm[1] += w * (jd * V1);
            mm[2] += w * (jd * V0 * V0);
            mm[3] += w * (jd * V1 * V1);
            mm[4] += w * (jd * V2 * V2);
            mm[5] += w * (jd * V0 * V2);
        }
        // block reduction in a fixed order
#pragma unroll
        for (int q = 0; q < 6; q++) {
            const double v = warp_sum(mm[q]);
            if (lane == 0) s_red[warp * 6 + q] = v;
        }
        warp_count_fails(a.counters, tally);
        __syncthreads();
        if (threadIdx.x < 6) {
            double s = 0;
            for (int w = 0; w < kMomentBlock / 32; w++) s += s_red[w * 6 + threadIdx.x];
            a.partial[((size_t)p * B + chunk) * 6 + threadIdx.x] = s;
        }
        if (threadIdx.x == 0 && nbound) atomicAdd(&a.counters[kCntBound], (unsigned long long)nbound);
    }
}

int sm_count()
{
    int dev = 0, nsm = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
                   cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess
               ? nsm
               : 0;
}

int resident_blocks(const void *kernel, int threads, size_t smem)
{
    const int nsm = sm_count();
    int dev = 0, per_sm = 0, optin = 0;
    cudaFuncAttributes at;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
        cudaFuncGetAttributes(&at, kernel) == cudaSuccess && smem + at.sharedSizeBytes <= (size_t)optin &&
        (smem + at.sharedSizeBytes <= 48 * 1024 ||
         cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              optin - (int)at.sharedSizeBytes) == cudaSuccess) &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) == cudaSuccess)
        return per_sm * nsm;
    cudaGetLastError();  // the caller refuses the call; a later launch must not report this
    return 0;
}

int moments_resident(size_t smem) { return resident_blocks((const void *)k_moments, kMomentBlock, smem); }

// sums the per-block partials of each point and normalises as rhofDF does
// (integ/Integ.cpp:160-162)
__device__ __forceinline__ void finalize_point(const double *partial, int npts, int B, double *out6, int p)
{
    double s[6] = {0, 0, 0, 0, 0, 0};
    for (int c = 0; c < B; c++)
#pragma unroll
        for (int q = 0; q < 6; q++) s[q] += partial[((size_t)p * B + c) * 6 + q];
    out6[0 * (size_t)npts + p] = s[0];
    out6[1 * (size_t)npts + p] = s[1] / s[0];
    out6[2 * (size_t)npts + p] = sqrt(s[2] / s[0]);
    out6[3 * (size_t)npts + p] = sqrt(s[3] / s[0]);
    out6[4 * (size_t)npts + p] = sqrt(s[4] / s[0]);
    out6[5 * (size_t)npts + p] = sqrt(fabs(s[5]) / s[0]);
}

__global__ void k_moments_finalize(const double *partial, int npts, int B, double *out6)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < npts) finalize_point(partial, npts, B, out6, p);
}

__global__ void k_moments_finalize_batch(MomentBatch batch, int npoints)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= npoints) return;
    const int m = batch_model(batch.point_start, batch.n, t);
    const MomentArgs &a = batch.args[m];
    finalize_point(a.partial, a.npts, a.blocks_per_point, a.out6, t - batch.point_start[m]);
}

__global__ void k_scatter6(int n, const int *idx, const double *src6, int npts, double *dst6)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    for (int q = 0; q < 6; q++) dst6[(size_t)q * npts + idx[t]] = src6[(size_t)q * n + t];
}

cudaError_t launch_scatter6(int n, const int *idx, const double *src6, int npts, double *dst6, cudaStream_t s)
{
    k_scatter6<<<(n + 127) / 128, 128, 0, s>>>(n, idx, src6, npts, dst6);
    return cudaGetLastError();
}

cudaError_t launch_moments_finalize_batch(const MomentBatch &b, int npoints, cudaStream_t s)
{
    k_moments_finalize_batch<<<(npoints + 127) / 128, 128, 0, s>>>(b, npoints);
    return cudaGetLastError();
}

cudaError_t launch_moments_plain_batch(const MomentArgs &a0, const MomentBatch &b, size_t smem, const PlainWork &w,
                                      cudaStream_t s)
{
    if (w.grid < 1) return cudaErrorInvalidConfiguration;
    const cudaError_t e = cudaMemsetAsync(w.next, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    k_moments<<<(unsigned)w.grid, kMomentBlock, smem, s>>>(a0, b, w);
    return cudaGetLastError();
}

cudaError_t launch_moments(const MomentArgs &a, const PlainWork &w, cudaStream_t s)
{
    const cudaError_t e =
        launch_moments_plain_batch(a, MomentBatch{nullptr, nullptr, nullptr, 0}, moment_smem_bytes(a), w, s);
    return e == cudaSuccess ? launch_moments_finalize(a, s) : e;
}

cudaError_t launch_moments_finalize(const MomentArgs &a, cudaStream_t s)
{
    k_moments_finalize<<<(a.npts + 127) / 128, 128, 0, s>>>(a.partial, a.npts, a.blocks_per_point, a.out6);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- actions
// Work items of `chunk` consecutive points; unbound points (H >= 0) give -1, -1
__global__ void __launch_bounds__(kSolveBlock, 2) k_actions(PotView P0, const double *Eg, const double *Dg, int ngrid,
                                                            GLRule gl0, const double2 *trig, const double *pts,
                                                            size_t n, int chunk, double *out, bool staged,
                                                            PlainWork work)
{
    extern __shared__ double sm[];  // solver | tables (staged: of a size that fits; else read in device memory)
    __shared__ int s_item, s_n;
    __shared__ unsigned short s_list[kActionChunk];
    __shared__ double s_pot[kActionChunk];
    const int nr = P0.nr, npoly = P0.npoly, nt = nr * npoly;
    SolveShared *s_solve = (SolveShared *)sm;
    double *s_ar = (double *)(s_solve + 1), *s_phil = s_ar + nr, *s_Pr = s_phil + nt, *s_it = s_Pr + nt,
           *s_Eg = s_it + interp_table_size(nr), *s_Dg = s_Eg + ngrid, *s_fast = s_Dg + ngrid;
    PotView P = P0;
    PotFast F{nr, npoly, P0.ar, P0.phil, nullptr, nullptr, nullptr};
    if (staged) {
        for (int i = threadIdx.x; i < nr; i += blockDim.x) s_ar[i] = P0.ar[i];
        for (int i = threadIdx.x; i < nt; i += blockDim.x) { s_phil[i] = P0.phil[i]; s_Pr[i] = P0.Pr[i]; }
        for (int i = threadIdx.x; i < ngrid; i += blockDim.x) { s_Eg[i] = Eg[i]; s_Dg[i] = Dg[i]; }
        __syncthreads();
        interp_table(nr, s_ar, s_it, threadIdx.x, blockDim.x);
        __syncthreads();
        P = PotView{nr, npoly, s_ar, s_phil, s_Pr, P0.Pr2, s_it};
        F = fast_tables(P, s_fast);
        Eg = s_Eg; Dg = s_Dg;
    }
    const SolveScratch S = solve_scratch(work.scratch + blockIdx.x * work.per_block, kActionChunk);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) { s_item = (int)atomicAdd(work.next, 1u); s_n = 0; }
        __syncthreads();
        const int item = s_item;
        if (item >= work.total) return;
        const size_t t0 = (size_t)item * chunk;
        const int m = (int)(n - t0 < (size_t)chunk ? n - t0 : (size_t)chunk);
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const double *x = pts + 5 * (t0 + i);
            const double Phi = pot_phi(P, x[0], x[1]);
            if (.5 * (x[2] * x[2] + x[3] * x[3] + x[4] * x[4]) + Phi >= 0) {
                out[2 * (t0 + i)] = -1;
                out[2 * (t0 + i) + 1] = -1;
            } else {
                s_pot[i] = Phi;
                s_list[atomicAdd(&s_n, 1)] = (unsigned short)i;
            }
        }
        __syncthreads();
        solve_orbits64(P, F, gl0, trig, s_n, S, *s_solve,
                       [&](int q, double &Delta, double &R, double &z, double &Phi, double &vR, double &vp, double &vz) {
                           const double *x = pts + 5 * (t0 + s_list[q]);
                           R = x[0]; z = x[1]; vR = x[2]; vp = x[3]; vz = x[4];
                           Phi = s_pot[s_list[q]];
                           Delta = deltafn(Eg, Dg, ngrid, .5 * (vR * vR + vp * vp + vz * vz) + Phi);
                       });
        for (int q = threadIdx.x; q < s_n; q += blockDim.x) {
            const size_t t = t0 + s_list[q];
            out[2 * t] = S.rec[q].Jr;
            out[2 * t + 1] = S.rec[q].Jz;
        }
    }
}

// tables beyond this size stay in device memory (two blocks per SM still fit)
constexpr size_t kStagedTables = 96 * 1024;
static size_t actions_table_bytes(int nr, int npoly, int ngrid)
{
    return (nr + 2 * (size_t)nr * npoly + fast_table_size(nr, npoly) + interp_table_size(nr) + 2 * (size_t)ngrid) *
           sizeof(double);
}
size_t actions_smem_bytes(int nr, int npoly, int ngrid)
{
    const size_t t = actions_table_bytes(nr, npoly, ngrid);
    return sizeof(SolveShared) + (t <= kStagedTables ? t : 0);
}

int actions_resident(size_t smem) { return resident_blocks((const void *)k_actions, kSolveBlock, smem); }

cudaError_t launch_actions(PotView P, const double *Eg, const double *Dg, int ngrid, GLRule gl, const double2 *trig,
                           const double *pts, size_t n, int chunk, double *out, const PlainWork &w, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    if (w.grid < 1 || chunk > kActionChunk) return cudaErrorInvalidConfiguration;
    const cudaError_t e = cudaMemsetAsync(w.next, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    const bool staged = actions_table_bytes(P.nr, P.npoly, ngrid) <= kStagedTables;
    k_actions<<<(unsigned)w.grid, kSolveBlock, actions_smem_bytes(P.nr, P.npoly, ngrid), s>>>(
        P, Eg, Dg, ngrid, gl, trig, pts, n, chunk, out, staged, w);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- potential
// Grid-stride over the points; the tables and interpolation constants staged in
// shared memory once per block where they fit (the FP64 pipe is the bound: ~400
// FP64 instructions per point at l <= 12).  200 003 points, 80 x 7 tables: 367
// us with a division per recurrence step and a bisection search per point, 253
// us with the reciprocals and the interval guess of interp_setup.  Fewer points than
// the threads of the two blocks that an SM holds (94 registers) go to as many blocks, a
// warp of points or more to each: 1000 points 50.6 us at first, 52.3 in whole blocks of
// 256, 35.7 so; 10 000 points 50.8, 53, 38.2.
constexpr int kPotBlock = 256;
constexpr size_t kPotStaged = 40 * 1024;
static size_t potential_smem_bytes(const PotView &P)
{
    return (P.nr + 2 * (size_t)P.nr * P.npoly + interp_table_size(P.nr)) * sizeof(double);
}

__global__ void __launch_bounds__(kPotBlock) k_potential_eval(PotView P, const double *Rz, size_t n, size_t per,
                                                              double *out, bool staged)
{
    extern __shared__ double sm[];
    if (staged) {
        const int nr = P.nr, nt = nr * P.npoly;
        double *s_ar = sm, *s_phil = s_ar + nr, *s_Pr = s_phil + nt, *s_it = s_Pr + nt;
        for (int i = threadIdx.x; i < nr; i += blockDim.x) s_ar[i] = P.ar[i];
        for (int i = threadIdx.x; i < nt; i += blockDim.x) { s_phil[i] = P.phil[i]; s_Pr[i] = P.Pr[i]; }
        __syncthreads();
        interp_table(nr, s_ar, s_it, threadIdx.x, blockDim.x);
        __syncthreads();
        P = PotView{nr, P.npoly, s_ar, s_phil, s_Pr, P.Pr2, s_it};
    }
    // blocks of a small batch take `per` consecutive points each, of a larger one (per = 0) all in strides
    const size_t first = blockIdx.x * (per ? per : (size_t)blockDim.x), end = per && first + per < n ? first + per : n,
                 stride = per ? blockDim.x : (size_t)gridDim.x * blockDim.x;
    for (size_t t = first + threadIdx.x; t < end; t += stride) {
        double phi, dR, dz;
        pot_grad(P, Rz[2 * t], Rz[2 * t + 1], phi, dR, dz);
        out[3 * t] = phi;
        out[3 * t + 1] = dR;
        out[3 * t + 2] = dz;
    }
}

cudaError_t launch_potential_eval(PotView P, const double *Rz, size_t n, double *out, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const size_t tab = potential_smem_bytes(P), sms = std::max(1, sm_count()), held = 2 * sms, wave = 4 * sms;
    const bool staged = tab <= kPotStaged;
    size_t per = 0, blocks = (n + kPotBlock - 1) / kPotBlock;
    if (blocks <= held) {  // a warp or more for each of the blocks that the SMs hold at once
        per = ((n + held - 1) / held + 31) / 32 * 32;
        blocks = (n + per - 1) / per;
    } else if (staged && blocks > wave) {
        blocks = wave;  // each block's tables serve all its points
    }
    k_potential_eval<<<(unsigned)std::min(blocks, (size_t)0x7fffffff), kPotBlock, staged ? tab : 0, s>>>(P, Rz, n, per,
                                                                                                      out, staged);
    return cudaGetLastError();
}

size_t moments_local_bytes()
{
    size_t m = 0;
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, k_moments) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    if (cudaFuncGetAttributes(&at, k_actions) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    if (cudaFuncGetAttributes(&at, k_potential_eval) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    return m;
}

}  // namespace fj
