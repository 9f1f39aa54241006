// fj_moments_mixed.cu -- the mixed-precision phase-space kernel (FJ_PREC_MIXED).
//
// Same decomposition as k_moments (items of a point's node range, fixed-order
// item partials); the per-node arithmetic follows fj_mixed.cuh: FP64 for the
// node's velocity, energy, focal distance and prolate-spheroidal transform,
// FP32 for the turning-point searches, the QAGS momentum integrals and the
// DF, FP64 again for turning points at the u/v limits and for the moments.
// Built with FMA contraction (the plain form is the rounding-faithful one).
#include <algorithm>
#include <cstdint>

#include "fj_group_qags.cuh"
#include "fj_internal.h"
#include "fj_mixed.cuh"
#include "fj_order.cuh"
#include "fj_solve64.cuh"

namespace fj {

// Work layout: an item is one contiguous range of at most a.mixed_chunk nodes
// of one point (mixed_blocks_per_point items per point).  Two persistent kernels
// go through the items of a slice of the launch:
//   k_mixed_turn       compacts an item's bound nodes (H < 0; about 40% of the
//                      cube), sorts them by the cost proxy of fj_order.cuh and
//                      finds their turning points, one node per thread: the FP64
//                      setup, bracket walks and Brent; a node's constants go to a
//                      record in device memory;
//   k_mixed_integrate  kMixedLanes (2) lanes per momentum integral: the first panel of
//                      every Ju and Jv of the item, then the bisections of those
//                      that go on, groups taking the next integral as they finish
//                      (fj_group_qags.cuh); then the DFs and the moment sums.
// With a node's whole solve on one thread (one kernel) the lanes of a warp sat in
// different places of it: the evaluator, 3/4 of the instructions, was entered with
// 13.7 of 32 lanes, and each thread kept its own interval list and call frames in
// local memory.  The same phases in one kernel executed 22 % fewer instructions
// but ran no faster: blocks in different phases pushed each other's code out of
// the instruction caches (4.8 stall cycles per issue waiting for instructions).
// Measured (GB300, 80x40 grid, 22^3 nodes): 270 ms with the fastest of the earlier
// one-kernel builds, 361-371 ms with its initial configuration; 284 ms with the
// phases in one kernel; 171 ms in two with four lanes per integral and the
// multipole loop as it was, 158 ms with it unrolled for the launch's npoly, 144 ms
// with the terms an evaluation does not need left out (dphi_chain), 138 ms with
// two lanes per integral (eight: 237 ms; the list upkeep of an integral is serial,
// so more integrals per warp share it; 24x8 and 33x11 models run 2 % slower with
// two than with four), 131 ms with the capped nodes' pass and the turning points'
// registers as below.  On a 240-point spread of that grid the warp instructions
// fall from 14.8 G (19.3 lanes active) to 3.4 G (17.3) + 4.9 G (25.1).  Interval
// lists kept in shared memory instead of behind L1 were slower (144 -> 162 ms at
// 64 registers: every access selects between the two places).
// (The unrolled range, npoly 3 to 8, is that of the models in use here; what larger ones
// or a batch of differing models would gain from builds of their own is not measured.)
// The integration is built in four register budgets (launch bounds of 4, 5, 6 and
// 8 resident blocks per SM: 128, 96, 80 and 64 registers) and for npoly 3 to 8, the
// turning points in two (10 and 7 blocks: 48 and 72 registers): kMixedVariants
// configurations, all with the same bits.  Turning points at 4, 5, 6, 7, 8 and 10
// blocks, the integration at 8: 141.1, 134.7, 131.8, 130.6, 135.2 and 135.0 ms on
// 80x40, 29.6, 28.5, 27.5, 26.8, 26.9 and 26.7 ms on four iterations of a 33x11 model,
// 53.3, 51.5, 50.6, 50.2, 50.0 and 49.5 ms on six 40x16 ones.  The integration at 6,
// 7, 8, 9 and 10 blocks: 135.3, 131.2, 130.9, 146.2 and 159.2 ms on 80x40.  Which
// configuration, and the item size, is a per-context setting (fj_autotune_mixed).
// Shared memory holds only what the node solves read: the FP32 tables (of a model
// too large for that, device memory: mixed_place), the radii, the focal-distance
// table, the velocity rule and the node list.  The
// FP64 potential tables are read from global memory (the point setup, the
// FP32 table build and the rare FP64 turning-point path).
#ifndef FJ_MIXED_LEAVE_ALL
#define FJ_MIXED_LEAVE_ALL 0  // 1: every bound node goes to the FP64 pass (tests)
#endif
constexpr int kMixedLanes = 2;                            // lanes per momentum integral
constexpr int kMixedGroups = kMixedBlock / kMixedLanes;   // integrals in flight per block
using MixedQags = GroupQags<float, kQagsCapF>;

// What a node's integrals need after its turning points, and its actions
struct alignas(16) MixedRec {
    float Delta, D2, K, EC, C0, Lt, shu2, sv2, swp, svp, sinv, cosv, sinhu, coshu, pvterm, rpt, Phipt, u_f, tb, Dt, wt;
    float Jr, Jz, eu, ev;  // actions; between the passes the first panels' results and errors
    unsigned word;         // kFail* bits of the turning points, kRecJu, kRecJv, node << kRecNode
    unsigned pad[2];
};
enum : unsigned { kRecJu = 8u, kRecJv = 16u, kRecNode = 8u };  // kRecNode: bit position (node within the item)

size_t mixed_rec_bytes() { return sizeof(MixedRec); }
size_t mixed_scratch_bytes() { return kMixedGroups * sizeof(MixedQags::List); }

int mixed_blocks_per_point(long long nq3, int chunk) { return (int)((nq3 + chunk - 1) / chunk); }

// capacity of a block's node list: the next power of two >= the node range (the sort pads to it)
__host__ __device__ static int mixed_list_cap(int chunk)
{
    int c = 1;
    while (c < chunk) c <<= 1;
    return c;
}

// FP32 tables of a model at one grid point.  Near: all in shared memory.  Far: the
// evaluator's table (pd) and the turning points' own copy of the potential and its
// derivative in device memory, one set per block, the rest in shared memory
// (kernels of their own, FAR: the near ones keep their shared-memory loads); the
// same values, so the same bits.  mixed_place chooses.
__host__ __device__ static size_t mixed_table_floats(int nr, int npoly, bool grad, bool far)
{
    return 2 * (size_t)nr + (far ? 0 : (grad ? 4 : 2) * (size_t)nr * npoly) + 4 * kQuadIntervals + npoly +
           2 * kQuadIntervals * npoly;
}
// floats of a block's tables in device memory
static size_t mixed_far_floats(int nr, int npoly) { return 4 * (size_t)nr * npoly; }

struct MixedTables {
    float *ar, *phil, *Pr, *ih, *qc, *pyl, *pd, *pe;
    // carves the tables out of 8-byte aligned memory f and, FAR, the block's set in
    // device memory; returns the first free float of f
    template <bool FAR>
    __device__ float *carve(float *f, int nr, int npoly, bool grad, float *far)
    {
        const int nt = nr * npoly;
        float *&g = FAR ? far : f;
        pd = g; g += 2 * nt;
        phil = Pr = nullptr;
        if (grad) { phil = g; Pr = g + nt; g += 2 * nt; }
        ar = f; f += nr;
        ih = f; f += nr;
        qc = f; f += 4 * kQuadIntervals;
        pyl = f; f += npoly;
        pe = f; f += 2 * kQuadIntervals * npoly;
        return f;
    }
    __device__ PotViewF build(const MomentArgs &a, double Phi_h, double R, double z)
    {
        const int nr = a.P.nr, npoly = a.P.npoly;
        mixed_tables_f(nr, npoly, a.P.ar, a.P.phil, a.P.Pr, Phi_h, R, z, ar, phil, Pr, ih, qc, pyl, threadIdx.x,
                       blockDim.x);
        PotViewF v = mixed_view_f(nr, npoly, a.P.ar, a.P.phil, Phi_h, R, z, ar, phil, Pr, ih, qc, pyl);
        __syncthreads();
        evaluator_tables_f(v, a.P.phil, Phi_h, pd, pe, threadIdx.x, blockDim.x);
        __syncthreads();
        v.pd = pd;
        v.pe = pe;
        return v;
    }
};

static size_t mixed_turn_smem(const MomentArgs &a, bool far)
{
    const size_t cap = mixed_list_cap(a.mixed_chunk);
    return (a.P.nr + 2 * a.ngrid + a.nq + 4) * sizeof(double) +
           (mixed_table_floats(a.P.nr, a.P.npoly, true, far) + 1) * sizeof(float) + (kMixedBlock / 32 + 1) * sizeof(int) +
           cap * (sizeof(float) + sizeof(unsigned short)) + 16;
}

// A block's shared memory of the integrals
struct MixedShared {
    float vals[kMixedGroups][43];  // panel values
    float xk[21];                  // panel abscissas in evaluation order: center + half xk (gk21_abscissa)
    GK21f K;
    int next;
};
enum : unsigned char { kIntNone = 0, kIntNew = 1, kIntMore = 2, kIntFull = 3 };  // state of an integral

static size_t mixed_integrate_smem(const MomentArgs &a, bool far)
{
    return (2 * a.nq + 6 * (kMixedBlock / 32)) * sizeof(double) +
           (mixed_table_floats(a.P.nr, a.P.npoly, false, far) + 1) * sizeof(float) + sizeof(MixedShared) +
           defer_words(a.mixed_chunk) * sizeof(unsigned) + 2 * (size_t)a.mixed_chunk + 16;
}

// the arguments and the model-local index of global block g of a launch
__device__ __forceinline__ const MomentArgs &block_args(const MomentArgs &a0, const MomentBatch &b, int g, int &bid)
{
    bid = g;
    if (b.n == 0) return a0;
    const int m = batch_model(b.block_start, b.n, g);
    bid -= b.block_start[m];
    return b.args[m];
}

// nodes [n0, n1) of item bid of its model
__device__ __forceinline__ void item_range(const MomentArgs &a, int bid, int &n0, int &n1)
{
    const long long nq3 = (long long)a.nq * a.nq * a.nq;
    const int B = a.blocks_per_point, chunk = bid % B;
    n0 = (int)(chunk * nq3 / B);
    n1 = (int)((chunk + 1) * nq3 / B);
}

template <int MINB, bool FAR>
__global__ void __launch_bounds__(kMixedBlock, MINB) k_mixed_turn(MomentArgs a0, MomentBatch batch, ItemQueue q)
{
    extern __shared__ double sm[];
    __shared__ int s_item, s_next;
    for (;;) {
        __syncthreads();  // every thread is done with the previous item's shared data
        if (threadIdx.x == 0) s_item = (int)atomicAdd(q.next, 1u);
        __syncthreads();
        const int slot = s_item;
        if (slot >= q.count) return;
        const int it = q.first + slot, g = q.order ? q.order[it] : it;
        const long long t_start = clock64();
        int bid;
        const MomentArgs &a = block_args(a0, batch, g, bid);
        const int nr = a.P.nr, npoly = a.P.npoly;
        double *s_ar = sm, *s_Eg = s_ar + nr, *s_Dg = s_Eg + a.ngrid, *s_xq = s_Dg + a.ngrid, *s_pt = s_xq + a.nq;
        MixedTables tab;
        int *s_wc = (int *)tab.carve<FAR>((float *)(s_pt + 4), nr, npoly, true, q.far + blockIdx.x * q.far_floats);
        unsigned short *s_list = (unsigned short *)(s_wc + kMixedBlock / 32);
        const int cap = mixed_list_cap(a.mixed_chunk);
        float *s_key = (float *)(((uintptr_t)(s_list + cap) + 15) & ~(uintptr_t)15);
        for (int i = threadIdx.x; i < nr; i += blockDim.x) s_ar[i] = a.P.ar[i];
        for (int i = threadIdx.x; i < a.ngrid; i += blockDim.x) { s_Eg[i] = a.Eg[i]; s_Dg[i] = a.Dg[i]; }
        for (int i = threadIdx.x; i < a.nq; i += blockDim.x) s_xq[i] = a.xq[i];
        const PotView P{nr, npoly, s_ar, a.P.phil, a.P.Pr, a.P.Pr2};
        const int p = bid / a.blocks_per_point;
        __syncthreads();
        if (threadIdx.x == 0) {  // per-point FP64 setup, shared by the block (integ/Integ.cpp:46-62,150-151)
            double R, z;
            if (a.Rz) { R = a.Rz[2 * p]; z = a.Rz[2 * p + 1]; }
            else {
                const int n = p / a.ngauss, gg = p % a.ngauss;
                const double c = a.ci[gg], si = sqrt(1 - c * c);
                R = s_ar[n] * si; z = s_ar[n] * c;
            }
            const double rmax = s_ar[nr - 1];
            const double Phi_h = pot_phi(P, R, z);
            s_pt[0] = R; s_pt[1] = z; s_pt[2] = Phi_h;
            s_pt[3] = sqrt(-2 * (Phi_h - pot_phi(P, 10 * rmax, 10 * rmax)));
        }
        __syncthreads();
        const double R = s_pt[0], z = s_pt[1], Phi_h = s_pt[2], Ve = s_pt[3];
        if (threadIdx.x < 4) q.point[4 * (size_t)slot + threadIdx.x] = s_pt[threadIdx.x];
        const PotViewF PF = tab.build(a, Phi_h, R, z);
        const int nq = a.nq, nq2 = nq * nq;
        int n0, n1;
        item_range(a, bid, n0, n1);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        auto velocity = [&](int node, double &V0, double &V1, double &V2) {
            V0 = 1e-6 + Ve * s_xq[node / nq2]; V1 = 1e-6 + Ve * s_xq[(node / nq) % nq]; V2 = 1e-6 + Ve * s_xq[node % nq];
        };
        // bound nodes of [n0, n1) in node order
        int nbound = 0;
        for (int base = n0; base < n1; base += kMixedBlock) {
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
            for (int w = 0; w < kMixedBlock / 32; w++) {
                if (w < warp) off += s_wc[w];
                tot += s_wc[w];
            }
            if (b) s_list[off + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)(node - n0);
            __syncthreads();
            nbound += tot;
        }
        for (int k = threadIdx.x; k < nbound; k += kMixedBlock) {
            const int node = n0 + s_list[k];
            s_key[k] = node_cost_key((float)s_xq[node / nq2], (float)s_xq[(node / nq) % nq], (float)s_xq[node % nq]);
        }
        if (threadIdx.x == 0) { s_next = kMixedBlock; q.nbound[slot] = nbound; }
        sort_list(s_list, s_key, nbound);
        __syncthreads();
        unsigned esc = 0;
        MixedRec *rec = (MixedRec *)q.rec + (size_t)slot * q.stride;
        for (int k = threadIdx.x; k < nbound;) {  // nodes taken as threads free up
            const int node = s_list[k];
            double V0, V1, V2;
            velocity(n0 + node, V0, V1, V2);
            const double H = .5 * (V0 * V0 + V1 * V1 + V2 * V2) + Phi_h;
            FudgeF o;
            bool ju, jv;
            unsigned fail = 0, e = 0;
            const bool bound = mixed_turning_points(P, PF, deltafn(s_Eg, s_Dg, a.ngrid, H), R, z, Phi_h, V0, V1, V2, o,
                                                    ju, jv, fail, e);
            esc += e;
            MixedRec r;
            r.Delta = o.Delta; r.D2 = o.D2; r.K = o.K; r.EC = o.EC; r.C0 = o.C0; r.Lt = o.Lt; r.shu2 = o.shu2;
            r.sv2 = o.sv2; r.swp = o.swp; r.svp = o.svp; r.sinv = o.sinv; r.cosv = o.cosv; r.sinhu = o.sinhu;
            r.coshu = o.coshu; r.pvterm = o.pvterm; r.rpt = o.rpt; r.Phipt = o.Phipt; r.u_f = o.u_f; r.tb = o.tb;
            r.Dt = o.Dt; r.wt = o.wt;
            r.Jr = r.Jz = bound ? 0.f : 1e31f;
            r.eu = r.ev = 0.f;
            r.word = fail | (ju ? kRecJu : 0u) | (jv ? kRecJv : 0u) | ((unsigned)node << kRecNode);
            r.pad[0] = r.pad[1] = 0;
            rec[k] = r;
            k = atomicAdd(&s_next, 1);
        }
        warp_count(&a.counters[kCntEscalated], esc);
        if (threadIdx.x == 0 && nbound) atomicAdd(&a.counters[kCntBound], (unsigned long long)nbound);
        if (q.cost && threadIdx.x == 0) q.cost[g] = (float)(clock64() - t_start);
    }
}

// The momentum integrals of an item's n nodes, kMixedLanes lanes to one
template <int NP>
__device__ __forceinline__ void mixed_integrals(PotViewF PF, int n, MixedRec *rec, MixedQags::List &L,
                                                unsigned char *state, MixedShared &sh)
{
    if (NP > 0) PF.npoly = NP;
    const int lane = threadIdx.x & 31, g = threadIdx.x / kMixedLanes, gi = threadIdx.x % kMixedLanes;
    const int lead = lane & ~(kMixedLanes - 1);
    const float epsabs = 1e-5f, epsrel = 1e-3f;
    const GK21f &K = sh.K;
    float *vals = sh.vals[g];
    MixedQags st;
    // pass 0: first panels, item = node (Ju), then n + node (Jv), in order;
    // pass 1: the bisections of the items that go on, taken as groups free up
    for (int pass = 0; pass < 2; pass++) {
        int item = pass == 0 ? g - kMixedGroups : -1;
        float a1 = 0.f, b2 = 0.f;
        if (pass == 1) {
            __syncthreads();
            if (threadIdx.x == 0) sh.next = 0;
            __syncthreads();
        }
        for (;;) {
            if (pass == 0) {
                item += kMixedGroups;
                a1 = 0.f; b2 = item < n ? kPIf : kPIHf;
            } else {
                if (gi == 0 && item < 0) {
                    do item = atomicAdd(&sh.next, 1);
                    while (item < 2 * n && state[item] != kIntMore);
                    if (item < 2 * n) {
                        const MixedRec &r = rec[item < n ? item : item - n];
                        a1 = 0.f; b2 = item < n ? kPIf : kPIHf;
                        st.begin(L, a1, b2, item < n ? r.Jr : r.Jz, item < n ? r.eu : r.ev);
                    }
                }
                item = __shfl_sync(0xffffffffu, item, lead);
                a1 = __shfl_sync(0xffffffffu, a1, lead);
                b2 = __shfl_sync(0xffffffffu, b2, lead);
            }
            if (!__any_sync(0xffffffffu, item < 2 * n)) break;
            const bool kv = item >= n;
            const bool on = item < 2 * n && (pass == 1 || state[item] == kIntNew);
            const int q = kv ? item - n : item;
            const float b1 = 0.5f * (a1 + b2);
            if (on) {
                const MixedRec &r = rec[q];
                FudgeF o;
                o.Delta = r.Delta; o.D2 = r.D2; o.K = r.K; o.EC = r.EC; o.C0 = r.C0; o.Lt = r.Lt; o.shu2 = r.shu2;
                o.sv2 = r.sv2; o.swp = r.swp; o.svp = r.svp; o.sinv = r.sinv; o.cosv = r.cosv; o.sinhu = r.sinhu;
                o.coshu = r.coshu; o.pvterm = r.pvterm; o.rpt = r.rpt; o.Phipt = r.Phipt; o.u_f = r.u_f; o.tb = r.tb;
                o.Dt = r.Dt; o.wt = r.wt;
                // the panels' centres and half-lengths, as gk21_abscissa forms them
                const float hi = pass == 0 ? b2 : b1;
                const float ce1 = mul_rn(0.5f, add_rn(a1, hi)), ha1 = mul_rn(0.5f, add_rn(hi, -a1)),
                            ce2 = mul_rn(0.5f, add_rn(b1, b2)), ha2 = mul_rn(0.5f, add_rn(b2, -b1));
                const int npts = pass == 0 ? 21 : 42;
                for (int e = gi; e < npts; e += kMixedLanes) {
                    const bool second = e >= 21;
                    const float x = add_rn(second ? ce2 : ce1, mul_rn(second ? ha2 : ha1, sh.xk[second ? e - 21 : e]));
                    FGeo G;
                    const int mode = kv ? kEvJv : kEvJu;
                    fudge_geom(o, mode, x, G);
                    vals[e] = fudge_finish(mode, G, pot_dphi_f<NP>(PF, G.R, G.z, o.rpt, G.dr2, G.dc2, o.Phipt));
                }
            }
            __syncwarp();
            // the panels' sums on two of the group's lanes
            float res = 0.f, err = 0.f, ra = 0.f, rc = 0.f;
            if (on && (gi == 0 || (gi == kMixedLanes / 2 && pass == 1)))
                gk21_sum(K, gi ? b1 : a1, pass == 0 || gi ? b2 : b1, vals + (gi ? 21 : 0), res, err, ra, rc);
            const int lane2 = lead + kMixedLanes / 2;
            const float res2 = __shfl_sync(0xffffffffu, res, lane2), err2 = __shfl_sync(0xffffffffu, err, lane2),
                        rc2 = __shfl_sync(0xffffffffu, rc, lane2);
            if (on && gi == 0) {
                bool done, full = false;
                float r = res;
                MixedRec &c = rec[q];
                if (pass == 0) {  // the early exits of QAGS
                    const float tol = fmaxf(epsabs, epsrel * fabsf(res));
                    done = (err <= 100 * FLT_EPSILON * ra && err > tol) || (err <= tol && err != rc) || err == 0.0f;
                    if (!done) {
                        if (kv) { c.Jz = res; c.ev = err; } else { c.Jr = res; c.eu = err; }
                        state[item] = kIntMore;
                    }
                } else {
                    done = st.update(L, res, err, rc, res2, err2, rc2, epsabs, epsrel, r, full);
                    if (!done) { a1 = L.iv[st.maxerr].a; b2 = L.iv[st.maxerr].b; }
                }
                if (done) {
                    if (kv) c.Jz = mixed_jz(c.Delta, c.wt, r); else c.Jr = mixed_jr(c.Delta, c.Dt, r);
                    state[item] = full ? kIntFull : kIntNone;
                    if (pass == 1) item = -1;
                }
            }
            __syncwarp();
        }
    }
}

template <int MINB, int NP, bool FAR>
__global__ void __launch_bounds__(kMixedBlock, MINB) k_mixed_integrate(MomentArgs a0, MomentBatch batch, ItemQueue q)
{
    extern __shared__ double sm[];
    __shared__ int s_item, s_nleft;
    MixedQags::List &L = ((MixedQags::List *)q.scratch)[blockIdx.x * kMixedGroups + threadIdx.x / kMixedLanes];
    for (;;) {
        __syncthreads();  // every thread is done with the previous item's shared data
        if (threadIdx.x == 0) { s_item = (int)atomicAdd(q.next + 1, 1u); s_nleft = 0; }
        __syncthreads();
        const int slot = s_item;
        if (slot >= q.count) return;
        const int it = q.first + slot, g = q.order ? q.order[it] : it;
        const long long t_start = clock64();
        int bid;
        const MomentArgs &a = block_args(a0, batch, g, bid);
        const int nr = a.P.nr, npoly = a.P.npoly;
        double *s_xq = sm, *s_wq = s_xq + a.nq, *s_red = s_wq + a.nq;
        MixedTables tab;
        float *const free = tab.carve<FAR>((float *)(s_red + 6 * (kMixedBlock / 32)), nr, npoly, false,
                                           q.far + blockIdx.x * q.far_floats);
        MixedShared &sh = *(MixedShared *)(((uintptr_t)free + 15) & ~(uintptr_t)15);
        unsigned *s_bits = (unsigned *)(&sh + 1);  // nodes left to the FP64 pass
        const int nw = defer_words(a.mixed_chunk);
        unsigned char *state = (unsigned char *)(s_bits + nw);
        const double R = q.point[4 * (size_t)slot], z = q.point[4 * (size_t)slot + 1],
                     Phi_h = q.point[4 * (size_t)slot + 2], Ve = q.point[4 * (size_t)slot + 3];
        const int n = q.nbound[slot];
        MixedRec *rec = (MixedRec *)q.rec + (size_t)slot * q.stride;
        for (int i = threadIdx.x; i < a.nq; i += blockDim.x) { s_xq[i] = a.xq[i]; s_wq[i] = a.wq[i]; }
        for (int i = threadIdx.x; i < nw; i += blockDim.x) s_bits[i] = 0u;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const unsigned w = rec[i].word;
            state[i] = w & kRecJu ? kIntNew : kIntNone;
            state[n + i] = w & kRecJv ? kIntNew : kIntNone;
        }
        if (threadIdx.x < 11) {
            sh.K.xgk[threadIdx.x] = (float)fj_xgk21_d[threadIdx.x];
            sh.K.wgk[threadIdx.x] = (float)fj_wgk21_d[threadIdx.x];
            if (threadIdx.x < 5) sh.K.wg[threadIdx.x] = (float)fj_wg10_d[threadIdx.x];
        }
        if (threadIdx.x < 21) {
            const int e = threadIdx.x, jj = e <= 10 ? 2 * ((e - 1) >> 1) + 1 : 2 * ((e - 11) >> 1);
            const float x = e ? (float)fj_xgk21_d[jj] : 0.f;
            sh.xk[e] = ((e - 1) & 1) ? x : -x;
        }
        const PotViewF PF = tab.build(a, Phi_h, R, z);
        mixed_integrals<NP>(PF, n, rec, L, state, sh);
        __syncthreads();
        // The DFs and the moments: thread t sums nodes t, t + 128, .. of the sorted
        // list.  A node whose FP32 solve hit a cap (a full QAGS list, a bracket walk
        // or Brent at its step limit) is marked in the item's bitmap and counts 0
        // here: the FP64 pass solves it again with the plain form's FP64 solve (QAGS
        // lists of kQagsCap intervals) and adds it to this item's sums.  Only what
        // that solve still caps is a failure, with the plain form's policy (a capped
        // bracket or root: DF 0; a full QAGS list: the estimate so far, as QUADPACK
        // returns it).
        const int nq = a.nq, nq2 = nq * nq, p = bid / a.blocks_per_point;
        const long long nq3 = (long long)nq2 * nq;
        int n0, n1;
        item_range(a, bid, n0, n1);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const double jacob = Ve * Ve * Ve;
        double m[6] = {0, 0, 0, 0, 0, 0};
        FailTally tally;
        for (int k = threadIdx.x; k < n; k += kMixedBlock) {
            const MixedRec &r = rec[k];
            const int local = (int)(r.word >> kRecNode), node = n0 + local;
            const int i = node / nq2, j = (node / nq) % nq, l = node % nq;
            const double V0 = 1e-6 + Ve * s_xq[i], V1 = 1e-6 + Ve * s_xq[j], V2 = 1e-6 + Ve * s_xq[l];
            const unsigned fail =
                (FJ_MIXED_LEAVE_ALL ? kFailQuad : 0u) | (r.word & 7u) | (state[k] == kIntFull || state[n + k] == kIntFull ? kFailQuad : 0u);
            float f = 0.f;
            if (fail && a.defer) {
                atomicOr(&s_bits[local >> 5], 1u << (local & 31));
                atomicAdd(&s_nleft, 1);
            } else {
                if (a.jout) {
                    float *jo = a.jout + ((size_t)p * nq3 + node) * 2;
                    jo[0] = r.Jr;
                    jo[1] = r.Jz;
                }
                tally.add(fail);
                if (!(fail & (kFailBracket | kFailRoot))) f = mixed_df(a.df, R * V1, r.Jr, r.Jz);
            }
            const double jd = (s_wq[i] * s_wq[j] * s_wq[l]) * (jacob * (double)f);
            m[0] += jd;
            m[1] += jd * V1;
            m[2] += jd * V0 * V0;
            m[3] += jd * V1 * V1;
            m[4] += jd * V2 * V2;
            m[5] += jd * V0 * V2;
        }
#pragma unroll
        for (int c = 0; c < 6; c++) {
            double v = m[c];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == 0) s_red[warp * 6 + c] = v;
        }
        warp_count_fails(a.counters, tally);
        __syncthreads();
        if (threadIdx.x < 6) {
            double s = 0;
            for (int w = 0; w < kMixedBlock / 32; w++) s += s_red[w * 6 + threadIdx.x];
            a.partial[(size_t)bid * 6 + threadIdx.x] = s;
        }
        if (a.defer) {  // the item's bitmap of deferred nodes and their number
            for (int i = threadIdx.x; i < nw; i += blockDim.x) a.defer[(size_t)bid * nw + i] = s_bits[i];
            if (threadIdx.x == 0) a.defer_count[bid] = s_nleft;
        }
        if (q.cost && threadIdx.x == 0) q.cost[g] += (float)(clock64() - t_start);
    }
}

// ------------------------------------------------------ the FP64 pass
// Over the nodes the mixed kernels left (launch_deferred): a scan of the items'
// counts, the compact list, a block of two warps per listed node, a warp per item
// adding its nodes in list order.
//
// The pass lasts as long as its slowest nodes (tens to a few thousand nodes, whose
// FP32 lists were full; in FP64 their integrals take up to some 30 bisections), so a
// node's solve is built for latency: a bracket walk evaluates its next 32 positions
// at once (warp_walk; walks were two thirds of a node's time), the two warps take
// the u and the v turning points and then the Ju and the Jv integral side by side,
// the two u roots are two lanes', a panel's values go over the lanes and its two
// sums over two of them, and the integrands are those of fj_solve64.cuh (tables in
// shared memory, one
// exponential, tabulated angles).  Measured (GB300): 0.72 ms for a 24x8 model's
// launch (16^3 nodes), 2.0 ms for one of six 40x16 models; 1.5 and 4.1 ms with the
// walks a step at a time, 2.2 and 5.5 ms with one warp per node, its integrals one
// after the other in the reference's expressions.

constexpr int kDeferBlock = 64;
// FP64 tables of a model staged in shared memory: 80 radii with 8 multipoles fit;
// a block of 32 KB leaves room for seven per SM.  A larger model's potential is
// read from global memory and its integrands are the reference's expressions.
constexpr int kDeferTable = 2560;

struct DeferShared {
    double tab[kDeferTable];
    OrbitQags::List list[2];
    double vals[2][43];
    double pt[4];  // R, z, Phi, escape speed
    OrbitRec rec;
};

// the potential of item arguments a: staged unless cur is a's already (all threads)
__device__ void defer_model(const MomentArgs &a, DeferShared &s, const MomentArgs *&cur, PotView &P, PotFast &F)
{
    if (cur == &a) return;
    cur = &a;
    const int nr = a.P.nr, npoly = a.P.npoly, nt = nr * npoly;
    P = PotView{nr, npoly, a.P.ar, a.P.phil, a.P.Pr, a.P.Pr2, nullptr};
    F = PotFast{nr, npoly, P.ar, P.phil, nullptr, nullptr, nullptr};
    if (nr + 2 * nt + fast_table_size(nr, npoly) + interp_table_size(nr) > kDeferTable) return;
    double *s_ar = s.tab, *s_phil = s_ar + nr, *s_Pr = s_phil + nt, *s_fast = s_Pr + nt,
           *s_it = s_fast + fast_table_size(nr, npoly);
    __syncthreads();
    for (int i = threadIdx.x; i < nr; i += kDeferBlock) s_ar[i] = a.P.ar[i];
    for (int i = threadIdx.x; i < nt; i += kDeferBlock) { s_phil[i] = a.P.phil[i]; s_Pr[i] = a.P.Pr[i]; }
    __syncthreads();
    interp_table(nr, s_ar, s_it, threadIdx.x, kDeferBlock);
    __syncthreads();
    P = PotView{nr, npoly, s_ar, s_phil, s_Pr, a.P.Pr2, s_it};
    F = fast_tables(P, s_fast);
    __syncthreads();
}

// QAGS of r's Ju or Jv integrand by a warp (all lanes; valid on lane 0)
__device__ double warp_orbit_integral(const PotView &P, const PotFast &F, const OrbitRec &r, bool kv, const double2 *trig,
                                      OrbitQags::List &L, double *vals, bool &full)
{
    const int lane = threadIdx.x & 31;
    const double epsabs = 1e-5, epsrel = 1e-3;  // wrp_GSLinteg, include/Utils.h:173-185
    double a1 = 0., b2 = kv ? kPIH : kPI, result = 0;
    unsigned heap = 1;
    bool run = false;
    OrbitQags st;
    if (lane < 21) {
        double sn, cs;
        panel_sincos(trig, kv, 1u, a1, b2, lane, sn, cs);
        vals[lane] = orbit_integrand(P, F, r, kv, sn, cs);
    }
    __syncwarp();
    if (lane == 0) {
        double res, err, ra, rc, ae;
        gk_sum<21>(a1, b2, vals, res, err, ra, rc);
        run = qags_head(res, err, ra, rc, epsabs, epsrel, 1000, result, ae) < 0;
        if (run) st.begin(L, a1, b2, res, err);
    }
    for (;;) {
        if (!__shfl_sync(0xffffffffu, run ? 1 : 0, 0)) return result;
        a1 = __shfl_sync(0xffffffffu, a1, 0);
        b2 = __shfl_sync(0xffffffffu, b2, 0);
        heap = __shfl_sync(0xffffffffu, heap, 0);
        const double b1 = 0.5 * (a1 + b2);
        const unsigned h1 = heap < (1u << 30) ? 2 * heap : 0u, h2 = h1 ? h1 + 1u : 0u;
        for (int e = lane; e < 42; e += 32) {
            const bool second = e >= 21;
            double sn, cs;
            panel_sincos(trig, kv, second ? h2 : h1, second ? b1 : a1, second ? b2 : b1, second ? e - 21 : e, sn, cs);
            vals[e] = orbit_integrand(P, F, r, kv, sn, cs);
        }
        __syncwarp();
        double res = 0, err = 0, ra, rc = 0;
        if (lane < 2) gk_sum<21>(lane ? b1 : a1, lane ? b2 : b1, vals + 21 * lane, res, err, ra, rc);
        const double res2 = __shfl_sync(0xffffffffu, res, 1), err2 = __shfl_sync(0xffffffffu, err, 1),
                     rc2 = __shfl_sync(0xffffffffu, rc, 1);
        if (lane == 0) {
            if (st.update(L, res, err, rc, res2, err2, rc2, epsabs, epsrel, result, full)) run = false;
            else {
                a1 = L.iv[st.maxerr].a;
                b2 = L.iv[st.maxerr].b;
                heap = L.heap[st.maxerr];
            }
        }
        __syncwarp();
    }
}

// A bracket walk by a warp: the positions x, next(x), next(next(x)), .. one per
// lane, each reached by the walk's own steps, up to the first where stop holds.
// x becomes that position, kept the one before it (unchanged if there is none), at
// the lane that holds it; it counts the steps.  False beyond kLoopCap steps.
template <class Next, class Stop>
__device__ bool warp_walk(double &x, double &kept, int &at, int &it, Next next, Stop stop)
{
    const int lane = threadIdx.x & 31;
    for (;;) {
        double p = x;
        for (int i = 0; i < lane; i++) p = next(p);
        const unsigned m = __ballot_sync(0xffffffffu, stop(p));
        if (m) {
            at = __ffs((int)m) - 1;
            if (at > 0) kept = __shfl_sync(0xffffffffu, p, at - 1);
            x = __shfl_sync(0xffffffffu, p, at);
            it += at;
            return it <= kLoopCap;
        }
        kept = __shfl_sync(0xffffffffu, p, 31);
        x = next(kept);
        it += 32;
        if (it > kLoopCap) return false;
    }
}

// U0Walk by a warp: the bracket [ui, uo] of u0; false beyond kLoopCap steps
__device__ bool warp_u0_bracket(const Fudge &o, double &ui, double &uo)
{
    double x = kUmidStart, dut;
    int at, it = 0;
    ui = uo = x;
    bool ok = warp_walk(x, uo, at, it, [](double p) { return p * .8; },
                        [&](double p) { dut = o.duturnfn(p); return !(dut < 0); });
    ui = x;
    if (it == 0 && __shfl_sync(0xffffffffu, dut, 0) > 0) {
        ok = warp_walk(x, ui, at, it, [](double p) { return p * 1.2; },
                       [&](double p) { return !(o.duturnfn(p) > 0); });
        uo = x;
    }
    return ok;
}

// UWalk by a warp (its results; fails beyond kLoopCap steps)
struct UBrackets {
    double u1, u2, uin, uout;
    bool degenerate, capped;
};
__device__ UBrackets warp_u_brackets(const Fudge &o)
{
    UBrackets w{1., 1., 1., 1., false, false};
    double x = 1., ut = o.uturnfn(x), dut = ut < 0 ? o.duturnfn(x) : 0.;
    int at, it = 0;
    auto out = [](double p) { return p * 1.1; };
    auto in = [](double p) { return p * .9; };
    auto positive_ends = [&](double p) { return !(o.uturnfn(p) > 0); };
    bool ok = true;
    if (ut < 0) {
        const bool climb = dut > 0;
        double eps = .1;
        for (;;) {
            const double f = 1 + eps;
            if (climb)
                ok = warp_walk(x, w.uin, at, it, [=](double p) { return p * f; },
                               [&](double p) {
                                   ut = o.uturnfn(p);
                                   return !(ut < 0 && o.duturnfn(p) > 0);
                               });
            else
                ok = warp_walk(x, w.uout, at, it, [=](double p) { return p / f; },
                               [&](double p) {
                                   ut = o.uturnfn(p);
                                   return !(ut < 0 && o.duturnfn(p) < 0);
                               });
            if (!ok || __shfl_sync(0xffffffffu, ut, at) >= 0) break;
            x = climb ? x / f : x * f;
            eps *= .2;
            if (eps < kTINY) {
                w.uin = w.uout = x;
                w.degenerate = true;
                return w;
            }
            x = climb ? x * (1 + eps) : x / (1 + eps);
        }
        if (ok && climb) {
            w.u1 = x;
            ok = warp_walk(x, w.u2, at, it, out, positive_ends);
            w.uout = x;
        } else if (ok) {
            w.u2 = x;
            ok = warp_walk(x, w.u1, at, it, in, positive_ends);
            w.uin = x;
        }
    } else {
        const double fu1 = ut;
        ok = warp_walk(x, w.u2, at, it, out, positive_ends);
        w.uout = x;
        if (ok && fu1 > 0) {
            w.u1 = x;
            x *= .9;
            ok = warp_walk(x, w.u1, at, it, in, positive_ends);
        }
        w.uin = x;
    }
    if (!ok) {
        w.uin = w.uout = x;
        w.degenerate = w.capped = true;
    }
    return w;
}

// VWalk by a warp: the bracket [lo, hi] of the v root, or true with the turning
// point at a limit in lo
__device__ bool warp_v_bracket(const Fudge &o, double &lo, double &hi, bool &capped)
{
    double x = .5 * kPIH, f;
    int at, it = 0;
    lo = hi = x;
    bool ok = warp_walk(x, hi, at, it, [](double p) { return .5 * (kPIH + p); },
                        [&](double p) { f = o.vturnfn(p); return kPIH - p < kTINY || !(f < 0); });
    if (it > 0) {
        if (!ok || kPIH - x < kTINY) { capped = !ok; lo = kPIH; return true; }
        lo = .5 * kPIH; hi = x;
        return false;
    }
    x = .5 * kPIH;
    ok = warp_walk(x, lo, at, it, [](double p) { return p * .5; },
                   [&](double p) { return p < kTINY || !(o.vturnfn(p) > 0); });
    if (!ok || x < kTINY) { capped = !ok; lo = 0; return true; }
    lo = x; hi = .5 * kPIH;
    return false;
}

// one left node's FP64 solve (the turning points of the plain form, QAGS lists of
// kQagsCap intervals, df_value) by the block: its six moment contributions and
// status on thread 0
__device__ void defer_solve(const MomentArgs &a, int bid, int node, const PotView &P, const PotFast &F, DeferShared &s,
                            double *c6, FailTally &tally)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = bid / a.blocks_per_point;
    OrbitRec &rec = s.rec;
    __syncthreads();  // the previous node's record is free
    if (warp == 0) {
        double R, z;  // the point, as the mixed kernels' setup
        if (a.Rz) { R = a.Rz[2 * p]; z = a.Rz[2 * p + 1]; }
        else {
            const int n = p / a.ngauss, gg = p % a.ngauss;
            const double c = a.ci[gg], si = sqrt(1 - c * c);
            R = P.ar[n] * si; z = P.ar[n] * c;
        }
        const double far = 10 * P.ar[P.nr - 1];
        const double phi = pot_phi(P, lane == 1 ? far : R, lane == 1 ? far : z);
        const double Phi_h = __shfl_sync(0xffffffffu, phi, 0), Ve = sqrt(-2 * (Phi_h - __shfl_sync(0xffffffffu, phi, 1)));
        if (lane == 0) { s.pt[0] = R; s.pt[1] = z; s.pt[2] = Phi_h; s.pt[3] = Ve; }
    }
    __syncthreads();
    const double R = s.pt[0], z = s.pt[1], Phi_h = s.pt[2], Ve = s.pt[3];
    const int nq = a.nq, nq2 = nq * nq;
    const int i = node / nq2, j = (node / nq) % nq, l = node % nq;
    const double V0 = 1e-6 + Ve * a.xq[i], V1 = 1e-6 + Ve * a.xq[j], V2 = 1e-6 + Ve * a.xq[l];
    if (warp == 0) {  // the constants of its equations
        Fudge o;
        double pu2, pv2;
        const double H = .5 * (V0 * V0 + V1 * V1 + V2 * V2) + Phi_h;
        const bool bound = fudge_point(P, deltafn(a.Eg, a.Dg, a.ngrid, H), R, z, Phi_h, V0, V1, V2, o, pu2, pv2);
        if (bound) {
            double ui, uo;
            if (!warp_u0_bracket(o, ui, uo)) o.fail |= kFailBracket;
            BrentState b;
            b.begin(ui, uo);
            while (!b.feed(o.duturnfn(b.x))) {}
            o.umid = b.root;
            o.fail |= b.fail;
            fudge_constants(o, pu2, pv2);
        }
        if (lane == 0) {
            rec.o = o;
            rec.todo = bound ? kOrbitBound : 0u;
            rec.Jr = rec.Jz = bound ? 0. : 1e31;
            rec.rootfail[0] = rec.rootfail[1] = rec.rootfail[2] = 0;
            rec.full[0] = rec.full[1] = 0;
        }
    }
    __syncthreads();
    if (rec.todo & kOrbitBound) {
        {
            const Fudge o = rec.o;
            __syncthreads();  // the turning points below go to the record
            if (warp == 0) {
                const UBrackets w = warp_u_brackets(o);
                double root = w.uin;
                unsigned fail = w.capped ? kFailBracket : 0u;
                if (!w.degenerate) {  // the inner root on even lanes, the outer one on odd lanes
                    BrentState b;
                    b.begin(lane & 1 ? w.u2 : w.uin, lane & 1 ? w.uout : w.u1);
                    while (!b.feed(o.uturnfn(b.x))) {}
                    root = b.root;
                    fail |= b.fail;
                }
                __syncwarp();
                const double outer = __shfl_sync(0xffffffffu, root, 1);
                fail |= __shfl_sync(0xffffffffu, fail, 1);
                if (lane == 0) {
                    Fudge &c = rec.o;
                    c.uinner = root; c.uouter = outer;
                    c.ubar = .5 * (root + outer);
                    c.Deltau = .5 * (outer - root);
                    rec.fju = fudge_ju_factor(c);
                    rec.rootfail[0] = fail;
                }
            } else {
                double vt, hi;
                bool capped = false;
                const bool limit = warp_v_bracket(o, vt, hi, capped);
                unsigned fail = capped ? kFailBracket : 0u;
                if (!limit) {
                    BrentState b;
                    b.begin(vt, hi);
                    while (!b.feed(o.vturnfn(b.x))) {}
                    vt = b.root;
                    fail |= b.fail;
                }
                if (lane == 0) {
                    rec.o.vturn = vt;
                    rec.w = kPIH - vt;
                    rec.fjv = fudge_jv_factor(rec.o);
                    rec.rootfail[2] = fail;
                }
            }
        }
        __syncwarp();  // a warp's integral needs its own turning points only
        const bool kv = warp != 0;
        if (!(kv ? fudge_jv_zero(rec.o) : fudge_ju_zero(rec.o))) {
            bool full = false;
            const double r = warp_orbit_integral(P, F, rec, kv, a.trig, s.list[warp], s.vals[warp], full);
            if (lane == 0) {
                if (kv) rec.Jz = rec.fjv * r / kPI; else rec.Jr = rec.fju * r / kPI;
                if (full) rec.full[warp] = 1;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x > 0) return;
    const double Jr = rec.Jr, Jz = rec.Jz;
    unsigned fail = rec.todo & kOrbitBound ? rec.status() : 0u;
    double DF = df_value(a.df, P, R, Jr, Jz, R * V1, fail);
    if (fail & (kFailBracket | kFailRoot)) DF = 0.;
    tally.add(fail);
    if (a.jout) {
        float *jo = a.jout + ((size_t)p * nq2 * nq + node) * 2;
        jo[0] = (float)Jr;
        jo[1] = (float)Jz;
    }
    const double jd = (a.wq[i] * a.wq[j] * a.wq[l]) * (Ve * Ve * Ve * DF);
    c6[0] = jd; c6[1] = jd * V1; c6[2] = jd * V0 * V0;
    c6[3] = jd * V1 * V1; c6[4] = jd * V2 * V2; c6[5] = jd * V0 * V2;
}

__device__ void add_tally(unsigned long long *counters, const FailTally &t, unsigned solved)
{
    if (solved) atomicAdd(&counters[kCntResolved64], (unsigned long long)solved);
    if (!t.any) return;
    atomicAdd(&counters[kCntFailed], (unsigned long long)t.any);
    if (t.quad) atomicAdd(&counters[kCntFailQuad], (unsigned long long)t.quad);
    if (t.bracket) atomicAdd(&counters[kCntFailBracket], (unsigned long long)t.bracket);
    if (t.root) atomicAdd(&counters[kCntFailRoot], (unsigned long long)t.root);
}

// exclusive scan of the counts: per chunk of kScanChunk blocks, then the chunk
// carries (one CTA; chunk_sum[nchunks] = the total), then the carries added
__device__ __forceinline__ int block_exclusive_scan(int v, int *s_warp, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nwarp ? s_warp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nwarp) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[nwarp - 1];
    const int res = x - v + (warp ? s_warp[warp - 1] : 0);
    __syncthreads();
    return res;
}

__global__ void __launch_bounds__(kScanChunk) k_defer_scan_chunks(DeferWork dw, int nblocks)
{
    __shared__ int s_warp[32];
    const int i = blockIdx.x * kScanChunk + threadIdx.x;
    int total;
    const int ex = block_exclusive_scan(i < nblocks ? dw.count[i] : 0, s_warp, total);
    if (i < nblocks) dw.offset[i] = ex;
    if (threadIdx.x == 0) dw.chunk_sum[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanChunk) k_defer_scan_carries(DeferWork dw, int nchunks)
{
    __shared__ int s_warp[32];
    int carry = 0;
    for (int base = 0; base < nchunks; base += kScanChunk) {
        const int i = base + threadIdx.x;
        const int v = i < nchunks ? dw.chunk_sum[i] : 0;
        int total;
        const int ex = block_exclusive_scan(v, s_warp, total);
        if (i < nchunks) dw.chunk_sum[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) dw.chunk_sum[nchunks] = carry;
}

// adds the carries and lists each block's left nodes in node order (a warp per block)
constexpr int kListWarps = 4;
__global__ void __launch_bounds__(32 * kListWarps) k_defer_list(MomentArgs a0, MomentBatch batch, DeferWork dw,
                                                                 int nblocks)
{
    const int lane = threadIdx.x & 31;
    const int g = blockIdx.x * kListWarps + (threadIdx.x >> 5);
    if (g >= nblocks) return;  // the whole warp
    const int off = dw.offset[g] + dw.chunk_sum[g / kScanChunk];
    __syncwarp();
    if (lane == 0) dw.offset[g] = off;
    const int cnt = dw.count[g];
    if (cnt == 0) return;
    int bid;
    const MomentArgs &a = block_args(a0, batch, g, bid);
    const int nw = defer_words(a.mixed_chunk), B = a.blocks_per_point, chunk = bid % B;
    const long long nq3 = (long long)a.nq * a.nq * a.nq;
    const int n0 = (int)(chunk * nq3 / B);
    const unsigned *bits = a.defer + (size_t)bid * nw;
    int rank = 0;
    for (int w = 0; w < nw && rank < cnt; w++) {
        const unsigned word = bits[w];  // the same word on every lane
        if ((word >> lane) & 1u) {
            const int e = off + rank + __popc(word & ((1u << lane) - 1u));
            if (e < dw.cap) { dw.node[e] = n0 + w * 32 + lane; dw.block[e] = g; }
        }
        rank += __popc(word);
    }
}

// a block per listed node (grid-stride over the launch's total); nodes beyond the
// list's capacity by their item, in node order, into its partial sums
__global__ void __launch_bounds__(kDeferBlock) k_defer_solve(MomentArgs a0, MomentBatch batch, DeferWork dw, int nblocks,
                                                             int nchunks)
{
    __shared__ __align__(128) unsigned char raw[sizeof(DeferShared)];
    DeferShared &s = *(DeferShared *)raw;
    const int total = dw.chunk_sum[nchunks], listed = min(total, dw.cap);
    const MomentArgs *cur = nullptr;
    PotView P;
    PotFast F;
    FailTally tally;
    unsigned solved = 0;
    unsigned long long *counters = a0.counters;
    for (int e = blockIdx.x; e < listed; e += gridDim.x) {
        int bid;
        const MomentArgs &a = block_args(a0, batch, dw.block[e], bid);
        counters = a.counters;
        defer_model(a, s, cur, P, F);
        double c6[6];
        defer_solve(a, bid, dw.node[e], P, F, s, c6, tally);
        if (threadIdx.x == 0) {
            for (int q = 0; q < 6; q++) dw.mom[(size_t)e * 6 + q] = c6[q];
            solved++;
        }
    }
    for (int g = blockIdx.x; total > dw.cap && g < nblocks; g += gridDim.x) {
        const int cnt = dw.count[g], off = dw.offset[g];
        if (off + cnt <= dw.cap) continue;
        int bid;
        const MomentArgs &a = block_args(a0, batch, g, bid);
        counters = a.counters;
        defer_model(a, s, cur, P, F);
        const long long nq3 = (long long)a.nq * a.nq * a.nq;
        const int n0 = (int)((bid % a.blocks_per_point) * nq3 / a.blocks_per_point);
        const unsigned *bits = a.defer + (size_t)bid * defer_words(a.mixed_chunk);
        double msum[6] = {0, 0, 0, 0, 0, 0};
        for (int k = max(0, dw.cap - off); k < cnt; k++) {  // the item's k-th left node, from its bitmap
            int r = k, wd = 0;
            while (r >= __popc(bits[wd])) r -= __popc(bits[wd++]);
            unsigned word = bits[wd];
            for (int t = 0; t < r; t++) word &= word - 1;
            double c6[6];
            defer_solve(a, bid, n0 + wd * 32 + (__ffs((int)word) - 1), P, F, s, c6, tally);
            if (threadIdx.x == 0) {
                for (int q = 0; q < 6; q++) msum[q] += c6[q];
                solved++;
            }
        }
        if (threadIdx.x == 0)
            for (int q = 0; q < 6; q++) a.partial[(size_t)bid * 6 + q] += msum[q];
    }
    if (threadIdx.x == 0) add_tally(counters, tally, solved);
}

// a warp per item: its listed nodes added in list order, a moment per lane
constexpr int kAddWarps = 4;
__global__ void __launch_bounds__(32 * kAddWarps) k_defer_add(MomentArgs a0, MomentBatch batch, DeferWork dw,
                                                               int nblocks)
{
    const int lane = threadIdx.x & 31;
    const int g = blockIdx.x * kAddWarps + (threadIdx.x >> 5);
    if (g >= nblocks) return;
    const int cnt = dw.count[g];
    if (cnt == 0 || lane >= 6) return;
    int bid;
    const MomentArgs &a = block_args(a0, batch, g, bid);
    const int off = dw.offset[g], last = min(off + cnt, dw.cap);
    double msum = 0;
    for (int e = off; e < last; e++) msum += dw.mom[(size_t)e * 6 + lane];
    a.partial[(size_t)bid * 6 + lane] += msum;
}

static cudaError_t launch_deferred(const MomentArgs &a, const MomentBatch &b, long long nblocks, const DeferWork &dw,
                                   cudaStream_t s)
{
    if (!dw.count) return cudaSuccess;
    const int nb = (int)nblocks, nchunks = (nb + kScanChunk - 1) / kScanChunk;
    k_defer_scan_chunks<<<nchunks, kScanChunk, 0, s>>>(dw, nb);
    k_defer_scan_carries<<<1, kScanChunk, 0, s>>>(dw, nchunks);
    k_defer_list<<<(nb + kListWarps - 1) / kListWarps, 32 * kListWarps, 0, s>>>(a, b, dw, nb);
    k_defer_solve<<<16 * std::max(1, sm_count()), kDeferBlock, 0, s>>>(a, b, dw, nb, nchunks);
    k_defer_add<<<(nb + kAddWarps - 1) / kAddWarps, 32 * kAddWarps, 0, s>>>(a, b, dw, nb);
    return cudaGetLastError();
}

namespace {
const void *turn_kernel(int variant, bool far)
{
    if (far) return (const void *)k_mixed_turn<7, true>;
    return variant < 4 ? (const void *)k_mixed_turn<10, false> : (const void *)k_mixed_turn<7, false>;
}

template <int MINB>
const void *integrate_kernel_np(int np)
{
    switch (np) {
    case 3: return (const void *)k_mixed_integrate<MINB, 3, false>;
    case 4: return (const void *)k_mixed_integrate<MINB, 4, false>;
    case 5: return (const void *)k_mixed_integrate<MINB, 5, false>;
    case 6: return (const void *)k_mixed_integrate<MINB, 6, false>;
    case 7: return (const void *)k_mixed_integrate<MINB, 7, false>;
    case 8: return (const void *)k_mixed_integrate<MINB, 8, false>;
    default: return (const void *)k_mixed_integrate<MINB, 0, false>;
    }
}

// np: the launch's multipoles per model (0: they differ)
const void *integrate_kernel(int variant, int np, bool far)
{
    if (far) return (const void *)k_mixed_integrate<8, 0, true>;
    switch (variant & 3) {
    case 0: return integrate_kernel_np<4>(np);
    case 1: return integrate_kernel_np<5>(np);
    case 2: return integrate_kernel_np<6>(np);
    default: return integrate_kernel_np<8>(np);
    }
}

// the launch's items, a slice of q.per_slice at a time through both kernels
cudaError_t launch_mixed_any(const MomentArgs &a, const MomentBatch &b, const ItemQueue &q0, int variant, int np,
                             cudaStream_t s)
{
    if (variant < 0 || variant >= kMixedVariants || q0.grid < 1 || q0.grid_turn < 1) return cudaErrorInvalidValue;
    for (int first = 0; first < q0.total; first += q0.per_slice) {
        ItemQueue q = q0;
        q.first = first;
        q.count = q0.total - first < q0.per_slice ? q0.total - first : q0.per_slice;
        cudaError_t e = cudaMemsetAsync(q.next, 0, 2 * sizeof(unsigned), s);
        if (e != cudaSuccess) return e;
        void *args[] = {(void *)&a, (void *)&b, (void *)&q};
        const unsigned gt = (unsigned)(q.count < q.grid_turn ? q.count : q.grid_turn),
                       gi = (unsigned)(q.count < q.grid ? q.count : q.grid);
        if ((e = cudaLaunchKernel(turn_kernel(variant, q.far_turn), dim3(gt), dim3(kMixedBlock), args, q.smem_turn, s)) != cudaSuccess ||
            (e = cudaLaunchKernel(integrate_kernel(variant, np, q.far_integrate), dim3(gi), dim3(kMixedBlock), args, q.smem, s)) !=
                cudaSuccess)
            return e;
    }
    return cudaGetLastError();
}
}  // namespace

// The line between near and far tables, by the blocks that an SM holds: a launch
// that near tables hold below the far kernel's residency runs faster from device
// memory (the tables stay in L1 and L2), the turning points with any block less, the
// integrals, which read little else, with a third less.  1500 points, 14^3 nodes (ms,
// near / turning points far / integrals far; one kernel with everything near before
// these two): 40x24 40.4 / 38.9 / 43.0, before 89; 80x24 39.1 / 33.5 / 40.0, 89; 100x24
// 36.2 / 31.6 / 35.9, 81; 130x24 37.6 / 29.9 / 36.0, 69; 250x24 49.1 / 27.9 / 44.5, 62;
// 500x24 83.2 / 41.0 / 65.4, 70; 80x7 15.3 / 15.5 / 16.9, 38; 400x7 15.4 / 11.5 / 15.3,
// 23; 1000x7 34.7 / 15.5 / 33.1, 36.  As chosen: 33.5, 28.7 (130x24), 23.6, 23.3 (500x24),
// 11.4 and 13.9 (1000x7).  Models beyond the near tables' limit (13 000 to 14 000
// entries) have the far ones only: 700x24 24.6 (one kernel before: 52 for 1000 points).  Few
// items take the near tables where these fit and hold every item at once.
bool mixed_place(int variant, int np, const MixedSize &z, ItemQueue &q)
{
    const int nt = resident_blocks(turn_kernel(variant, false), kMixedBlock, z.turn[0]),
              ni = resident_blocks(integrate_kernel(variant, np, false), kMixedBlock, z.integrate[0]),
              ft = resident_blocks(turn_kernel(variant, true), kMixedBlock, z.turn[1]),
              fi = resident_blocks(integrate_kernel(variant, np, true), kMixedBlock, z.integrate[1]);
    q.far_turn = ft > nt && q.total > nt;
    q.far_integrate = 2 * fi >= 3 * ni && q.total > ni;
    q.smem_turn = z.turn[q.far_turn];
    q.smem = z.integrate[q.far_integrate];
    q.grid_turn = std::min(q.total, q.far_turn ? ft : nt);
    q.grid = std::min(q.total, q.far_integrate ? fi : ni);
    q.far_floats = q.far_turn || q.far_integrate ? z.far : 0;
    return q.grid_turn > 0 && q.grid > 0;
}

MixedSize mixed_size(const MomentArgs &a)
{
    return MixedSize{{mixed_turn_smem(a, false), mixed_turn_smem(a, true)},
                     {mixed_integrate_smem(a, false), mixed_integrate_smem(a, true)},
                     mixed_far_floats(a.P.nr, a.P.npoly)};
}

cudaError_t launch_moments_mixed(const MomentArgs &a, int variant, const DeferWork &dw, const ItemQueue &q,
                                 cudaStream_t s)
{
    if (a.mixed_chunk < kMixedBlock || a.mixed_chunk > kMixedMaxNodes) return cudaErrorInvalidValue;
    const MomentBatch none{nullptr, nullptr, nullptr, 0};
    const long long nblocks = (long long)a.npts * a.blocks_per_point;
    if (q.total != nblocks) return cudaErrorInvalidValue;
    cudaError_t e = launch_mixed_any(a, none, q, variant, a.P.npoly, s);
    if (e == cudaSuccess) e = launch_deferred(a, none, nblocks, dw, s);
    if (e != cudaSuccess) return e;
    return launch_moments_finalize(a, s);
}

cudaError_t launch_moments_plain_batch(const MomentArgs &a0, const MomentBatch &b, size_t smem, const PlainWork &w,
                                      cudaStream_t s);

cudaError_t launch_moments_batch(const MomentArgs &a0, const MomentBatch &b, int nblocks, size_t smem,
                                 bool mixed, int variant, int np, const DeferWork &dw, const ItemQueue &q,
                                 const PlainWork &w, cudaStream_t s)
{
    if (!mixed) return launch_moments_plain_batch(a0, b, smem, w, s);
    if (q.total != nblocks) return cudaErrorInvalidValue;
    const cudaError_t e = launch_mixed_any(a0, b, q, variant, np, s);
    return e == cudaSuccess ? launch_deferred(a0, b, nblocks, dw, s) : e;
}

size_t moments_mixed_local_bytes()
{
    size_t m = 0;
    cudaFuncAttributes at;
    for (int v = 0; v < kMixedVariants; v++)
        for (const void *k : {turn_kernel(v, false), integrate_kernel(v, 0, false), integrate_kernel(v, 7, false)})
            if (cudaFuncGetAttributes(&at, k) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    for (const void *k : {turn_kernel(0, true), integrate_kernel(0, 0, true), (const void *)k_defer_solve,
                          (const void *)k_defer_add})
        if (cudaFuncGetAttributes(&at, k) == cudaSuccess && at.localSizeBytes > m) m = at.localSizeBytes;
    return m;
}

}  // namespace fj
