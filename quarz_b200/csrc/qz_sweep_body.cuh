// qz_sweep_body.cuh -- the quasi-static xi sweep of one time step by ONE CTA (sm_100a, FP64).
//
// Replaces the per-slice kernel chain of Simulation::step_fields (src/Simulation.cpp:636-795):
//   zero_sources -> PlasmaSpecies::deposit -> combine_sources -> solve_slice_fields
//   (psi, E_z, W+, B_z, deposit_S, B+) -> store_slice -> PlasmaSpecies::push
// for azimuthal mode m = 0.
//
// Layout. The radial arrays of a slice (sources, fields, grid, stencils, operator rows) live in shared
// memory (the constant ones fall back to global memory for very large grids). With at most 512
// plasma particles, thread p owns particle p and keeps its state -- position, momentum, Delta,
// weight and the Adams-Bashforth history -- in registers for the whole sweep; larger plasmas keep
// the state in a global scratch buffer.
//
// Tridiagonal solves. Each system is solved by a group of warps of its own, a thread owning a few
// consecutive rows (l0_solve, bplus_solve): the three Thomas recurrences -- pivots u_i = b_i - a_i c_{i-1} /
// u_{i-1}, forward y_i = (d_i - a_i y_{i-1}) / u_i, backward x_i = y_i - (c_i / u_i) x_{i+1} -- run along a
// thread's rows and as scans over the group's threads: pivots as normalised prefix products of 2x2
// matrices, the substitutions as scans of affine maps. The psi, E_z and B_z systems share the constant
// operator L0, whose substitutions are plain sums.
//
// Slice schedule (barriers of the CTA between the phases, of a system's group inside the solves):
//   P2  psi, E_z, B_z and W+; sources of slice k+1 = beam + background
//   P3  S+ deposit by the particles
//   P4  B_r, B_theta
//   P5  store slice k; push k -> k+1 and deposit into the sources of slice k+1
#pragma once
#include "qz_device.cuh"
#include "qz_internal.h"

namespace qzb {

namespace sweep_detail {

constexpr int kThreads = kSweepThreads;
constexpr int kW = kThreads / 32;
constexpr unsigned FULL = 0xffffffffu;

// Gate of a stand-alone sweep: no other CTA to wait for or to inform.
struct NoGate {
    static constexpr bool kActive = false;
    __device__ bool before_rows(int) { return true; }       // warp 0: beam-source rows <= row are final
    __device__ void slice_done_all(int, int = 0, int = 1) {} // every thread, after its stores of slice k (its CTA's
                                                             // rank in, and the size of, the team that sweeps)
    __device__ bool slice_done(int) { return true; }         // thread 0, after the barrier: publish slice k
    // this sweep's buffers
    __device__ const double* bsrc(const SweepArgs& A) const { return A.bsrc; }
    __device__ double* fld(const SweepArgs& A) const { return A.fld; }
    __device__ double* diag(const SweepArgs& A) const { return A.diag; }
    __device__ double* ps(const SweepArgs& A) const { return A.ps; }
    __device__ double* srcs(const SweepArgs& A) const { return A.srcs; }
    __device__ double* bgs(const SweepArgs& A) const { return A.bgs; }
    __device__ double* traj(const SweepArgs& A) const { return A.traj; }
    __device__ double* wrec(const SweepArgs& A) const { return A.wrec; }
};

// ---------------------------------------------------------------- block scans
// Block-wide scans of one row per thread (the smoothing filter and the adjoint's reverse sweep). Shared
// scratch for the warp totals of one scan: 8 x kW doubles; two of them alternate.

// exact power-of-two rescaling of a 2x2 matrix (its largest entry into [1, 2)), by the exponent fields
__device__ __forceinline__ void renorm(double& m00, double& m01, double& m10, double& m11) {
    const int e = max(max(__double2hiint(m00) & 0x7ff00000, __double2hiint(m01) & 0x7ff00000),
                      max(__double2hiint(m10) & 0x7ff00000, __double2hiint(m11) & 0x7ff00000));
    const double s = __hiloint2double(max(0x7fe00000 - e, 0x00100000), 0);
    m00 *= s; m01 *= s; m10 *= s; m11 *= s;
}

// Exclusive forward scan of the affine maps y -> a y + b (thread order = row order), applied to
// y_{-1} = 0: yb[r] is y just before this thread's rows.
template <int NR>
__device__ __forceinline__ void scan_fwd(double a, const double (&b)[NR], double (&yb)[NR], double* tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double A = a, B[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) B[r] = b[r];
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        const double Ap = __shfl_up_sync(FULL, A, st);
        double Bp[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) Bp[r] = __shfl_up_sync(FULL, B[r], st);
        if (lane >= st) {
#pragma unroll
            for (int r = 0; r < NR; ++r) B[r] = fma(A, Bp[r], B[r]);
            A *= Ap;
        }
    }
    if (lane == 31) {
        tot[warp] = A;
#pragma unroll
        for (int r = 0; r < NR; ++r) tot[kW * (1 + r) + warp] = B[r];
    }
    double eA = __shfl_up_sync(FULL, A, 1), eB[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) eB[r] = __shfl_up_sync(FULL, B[r], 1);
    if (lane == 0) {
        eA = 1.0;
#pragma unroll
        for (int r = 0; r < NR; ++r) eB[r] = 0.0;
    }
    __syncthreads();
    double ta = lane < kW ? tot[lane] : 1.0, tb[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) tb[r] = lane < kW ? tot[kW * (1 + r) + lane] : 0.0;
#pragma unroll
    for (int st = 1; st < kW; st <<= 1) {
        const double ap = __shfl_up_sync(FULL, ta, st);
        double bp[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) bp[r] = __shfl_up_sync(FULL, tb[r], st);
        if (lane >= st) {
#pragma unroll
            for (int r = 0; r < NR; ++r) tb[r] = fma(ta, bp[r], tb[r]);
            ta *= ap;
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const double cw = __shfl_sync(FULL, tb[r], (warp + 31) & 31);
        yb[r] = fma(eA, warp > 0 ? cw : 0.0, eB[r]);
    }
}

// Exclusive backward scan of x -> a x + b applied to x_{end} = 0: xa[r] is x just after this
// thread's rows.
template <int NR>
__device__ __forceinline__ void scan_bwd(double a, const double (&b)[NR], double (&xa)[NR], double* tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double A = a, B[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) B[r] = b[r];
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        const double An = __shfl_down_sync(FULL, A, st);
        double Bn[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) Bn[r] = __shfl_down_sync(FULL, B[r], st);
        if (lane + st < 32) {
#pragma unroll
            for (int r = 0; r < NR; ++r) B[r] = fma(A, Bn[r], B[r]);
            A *= An;
        }
    }
    if (lane == 0) {
        tot[warp] = A;
#pragma unroll
        for (int r = 0; r < NR; ++r) tot[kW * (1 + r) + warp] = B[r];
    }
    double eA = __shfl_down_sync(FULL, A, 1), eB[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) eB[r] = __shfl_down_sync(FULL, B[r], 1);
    if (lane == 31) {
        eA = 1.0;
#pragma unroll
        for (int r = 0; r < NR; ++r) eB[r] = 0.0;
    }
    __syncthreads();
    double ta = lane < kW ? tot[lane] : 1.0, tb[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) tb[r] = lane < kW ? tot[kW * (1 + r) + lane] : 0.0;
#pragma unroll
    for (int st = 1; st < kW; st <<= 1) {
        const double an = __shfl_down_sync(FULL, ta, st);
        double bn[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) bn[r] = __shfl_down_sync(FULL, tb[r], st);
        if (lane + st < kW) {
#pragma unroll
            for (int r = 0; r < NR; ++r) tb[r] = fma(ta, bn[r], tb[r]);
            ta *= an;
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const double cw = __shfl_sync(FULL, tb[r], (warp + 1) & 31);
        xa[r] = fma(eA, warp < kW - 1 ? cw : 0.0, eB[r]);
    }
}

// The same two scans for NS independent systems, each with its own map y -> a[s] y + b[s].
template <int NS>
__device__ __forceinline__ void scan_fwd_n(const double (&a)[NS], const double (&b)[NS], double (&yb)[NS],
                                           double* tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double A[NS], B[NS];
#pragma unroll
    for (int r = 0; r < NS; ++r) { A[r] = a[r]; B[r] = b[r]; }
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        double Ap[NS], Bp[NS];
#pragma unroll
        for (int r = 0; r < NS; ++r) { Ap[r] = __shfl_up_sync(FULL, A[r], st); Bp[r] = __shfl_up_sync(FULL, B[r], st); }
        if (lane >= st)
#pragma unroll
            for (int r = 0; r < NS; ++r) { B[r] = fma(A[r], Bp[r], B[r]); A[r] *= Ap[r]; }
    }
    if (lane == 31)
#pragma unroll
        for (int r = 0; r < NS; ++r) { tot[kW * (2 * r) + warp] = A[r]; tot[kW * (2 * r + 1) + warp] = B[r]; }
    double eA[NS], eB[NS];
#pragma unroll
    for (int r = 0; r < NS; ++r) {
        eA[r] = __shfl_up_sync(FULL, A[r], 1);
        eB[r] = __shfl_up_sync(FULL, B[r], 1);
        if (lane == 0) { eA[r] = 1.0; eB[r] = 0.0; }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NS; ++r) {
        double ta = lane < kW ? tot[kW * (2 * r) + lane] : 1.0, tb = lane < kW ? tot[kW * (2 * r + 1) + lane] : 0.0;
#pragma unroll
        for (int st = 1; st < kW; st <<= 1) {
            const double ap = __shfl_up_sync(FULL, ta, st), bp = __shfl_up_sync(FULL, tb, st);
            if (lane >= st) { tb = fma(ta, bp, tb); ta *= ap; }
        }
        const double cw = __shfl_sync(FULL, tb, (warp + 31) & 31);
        yb[r] = fma(eA[r], warp > 0 ? cw : 0.0, eB[r]);
    }
}

template <int NS>
__device__ __forceinline__ void scan_bwd_n(const double (&a)[NS], const double (&b)[NS], double (&xa)[NS],
                                           double* tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double A[NS], B[NS];
#pragma unroll
    for (int r = 0; r < NS; ++r) { A[r] = a[r]; B[r] = b[r]; }
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        double An[NS], Bn[NS];
#pragma unroll
        for (int r = 0; r < NS; ++r) { An[r] = __shfl_down_sync(FULL, A[r], st); Bn[r] = __shfl_down_sync(FULL, B[r], st); }
        if (lane + st < 32)
#pragma unroll
            for (int r = 0; r < NS; ++r) { B[r] = fma(A[r], Bn[r], B[r]); A[r] *= An[r]; }
    }
    if (lane == 0)
#pragma unroll
        for (int r = 0; r < NS; ++r) { tot[kW * (2 * r) + warp] = A[r]; tot[kW * (2 * r + 1) + warp] = B[r]; }
    double eA[NS], eB[NS];
#pragma unroll
    for (int r = 0; r < NS; ++r) {
        eA[r] = __shfl_down_sync(FULL, A[r], 1);
        eB[r] = __shfl_down_sync(FULL, B[r], 1);
        if (lane == 31) { eA[r] = 1.0; eB[r] = 0.0; }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NS; ++r) {
        double ta = lane < kW ? tot[kW * (2 * r) + lane] : 1.0, tb = lane < kW ? tot[kW * (2 * r + 1) + lane] : 0.0;
#pragma unroll
        for (int st = 1; st < kW; st <<= 1) {
            const double an = __shfl_down_sync(FULL, ta, st), bn = __shfl_down_sync(FULL, tb, st);
            if (lane + st < kW) { tb = fma(ta, bn, tb); ta *= an; }
        }
        const double cw = __shfl_sync(FULL, tb, (warp + 1) & 31);
        xa[r] = fma(eA[r], warp < kW - 1 ? cw : 0.0, eB[r]);
    }
}

// Exclusive scan of 2x2 matrix products (later rows on the left) for NS systems: on return
// (p[s], q[s]) = first column of the product of all matrices before this thread's rows.
template <int NS>
__device__ __forceinline__ void scan_pivots(double (&m)[NS][4], double (&p)[NS], double (&q)[NS], double* tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // The thread's matrices must come renormalised (largest entry in [1, 2)); a product of at most 32 such
    // matrices stays below 2^63 and the products of the 16 renormalised warp totals below 2^31, so the
    // scan renormalises once per lane after the warp stage instead of at every level. Renormalising
    // scales by powers of two, which is exact, and the pivots use only ratios of p and q: the results
    // are the same bits either way.
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double p00 = __shfl_up_sync(FULL, m[s][0], st), p01 = __shfl_up_sync(FULL, m[s][1], st);
            const double p10 = __shfl_up_sync(FULL, m[s][2], st), p11 = __shfl_up_sync(FULL, m[s][3], st);
            if (lane >= st) {
                const double n00 = m[s][0] * p00 + m[s][1] * p10, n01 = m[s][0] * p01 + m[s][1] * p11;
                const double n10 = m[s][2] * p00 + m[s][3] * p10, n11 = m[s][2] * p01 + m[s][3] * p11;
                m[s][0] = n00; m[s][1] = n01; m[s][2] = n10; m[s][3] = n11;
            }
        }
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) renorm(m[s][0], m[s][1], m[s][2], m[s][3]);
    if (lane == 31)
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e) tot[kW * (4 * s + e) + warp] = m[s][e];
    double ex[NS][4];
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int e = 0; e < 4; ++e) ex[s][e] = __shfl_up_sync(FULL, m[s][e], 1);
    if (lane == 0)
#pragma unroll
        for (int s = 0; s < NS; ++s) { ex[s][0] = 1.0; ex[s][1] = 0.0; ex[s][2] = 0.0; ex[s][3] = 1.0; }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        double t00 = lane < kW ? tot[kW * (4 * s) + lane] : 1.0, t01 = lane < kW ? tot[kW * (4 * s + 1) + lane] : 0.0;
        double t10 = lane < kW ? tot[kW * (4 * s + 2) + lane] : 0.0, t11 = lane < kW ? tot[kW * (4 * s + 3) + lane] : 1.0;
#pragma unroll
        for (int st = 1; st < kW; st <<= 1) {
            const double p00 = __shfl_up_sync(FULL, t00, st), p01 = __shfl_up_sync(FULL, t01, st);
            const double p10 = __shfl_up_sync(FULL, t10, st), p11 = __shfl_up_sync(FULL, t11, st);
            if (lane >= st) {
                const double n00 = t00 * p00 + t01 * p10, n01 = t00 * p01 + t01 * p11;
                const double n10 = t10 * p00 + t11 * p10, n11 = t10 * p01 + t11 * p11;
                t00 = n00; t01 = n01; t10 = n10; t11 = n11;
            }
        }
        const int src = (warp + 31) & 31;
        double c00 = __shfl_sync(FULL, t00, src), c10 = __shfl_sync(FULL, t10, src);
        if (warp == 0) { c00 = 1.0; c10 = 0.0; }
        // column 0 of (within-warp exclusive product) x (carry of the earlier warps)
        p[s] = ex[s][0] * c00 + ex[s][1] * c10;
        q[s] = ex[s][2] * c00 + ex[s][3] * c10;
    }
}

// ---------------------------------------------------------------- batched shared-memory adds
// All NA updates of one thread are issued together (independent compare-and-swap rounds) instead
// of one serialised atomic loop per address. Lock-free: every round at least one contender of
// each address succeeds, so the loop ends after at most one round per contender.
template <int NA>
__device__ __forceinline__ void add_multi(double* const (&p)[NA], const double (&v)[NA]) {
    unsigned long long old[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) old[i] = __double_as_longlong(*reinterpret_cast<volatile double*>(p[i]));
    unsigned pend = (1u << NA) - 1u;
    for (int round = 0; pend && round < 4 * kThreads; ++round) {
#pragma unroll
        for (int i = 0; i < NA; ++i)
            if (pend & (1u << i)) {
                const unsigned long long nv = __double_as_longlong(__longlong_as_double(old[i]) + v[i]);
                const unsigned long long got = atomicCAS(reinterpret_cast<unsigned long long*>(p[i]), old[i], nv);
                if (got == old[i]) pend &= ~(1u << i); else old[i] = got;
            }
    }
}

// Warp aggregation of deposits: lanes holding contributions to the same cell form runs of equal
// keys in lane order (plasma particles stay close to their radial loading order); a segmented
// warp-shuffle scan sums each run, and only the last lane of a run updates shared memory. Runs
// split by reordering only cost extra updates, never correctness. Blowout piles tens of particles
// into a few sheath or axis cells, where per-particle updates of the same word would serialise.
template <int NV>
__device__ __forceinline__ bool warp_runs_sum(int key, double (&v)[NV]) {
    const int lane = threadIdx.x & 31;
    const int kprev = __shfl_up_sync(FULL, key, 1);
    const bool head = (lane == 0) || (kprev != key);
    const unsigned heads = __ballot_sync(FULL, head);
    if (heads == FULL) return true;                   // no shared cell in this warp
    const unsigned le = heads & (0xffffffffu >> (31 - lane));     // run heads at or below this lane
    const int seg = __popc(le);
    // the scan levels the longest run of the warp needs: a level of stride st adds only within runs
    // longer than st, so stopping after them leaves every sum as the full scan gives it, bit for bit
    const int maxoff = (int)__reduce_max_sync(FULL, (unsigned)(lane - (31 - __clz(le))));
#pragma unroll 1
    for (int st = 1; st <= maxoff; st <<= 1) {
        const int sp = __shfl_up_sync(FULL, seg, st);
        double vp[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) vp[i] = __shfl_up_sync(FULL, v[i], st);
        if (lane >= st && sp == seg)
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] += vp[i];
    }
    const int knext = __shfl_down_sync(FULL, key, 1);
    return (lane == 31) || (knext != key);
}

// ---------------------------------------------------------------- exact, order-independent deposits
// The contributions of a deposit to a node array are summed as 64-bit integers in units of a power-
// of-two quantum q, so the sum is the same whatever order the warps add in: every deposit, and with
// it the whole sweep, is reproducible bit for bit. q is chosen per deposit and per array from the
// largest contribution (its binary exponent: a block-wide maximum taken before the adds) and from
// the most contributions one node can receive (2^bits; every partial sum stays below 2^63 quanta).
// Relative to the largest contribution of the deposit the quantum is 2^(bits - 62): about one unit
// in the last place of FP64 for the 511 plasma particles of a slice. A non-finite contribution makes
// its array's values of that deposit NaN.
__device__ __forceinline__ int fx_bexp(double v) {         // biased exponent: 0 for 0, 2047 for Inf / NaN
    return (int)((__double_as_longlong(v) >> 52) & 0x7ff);
}
// 1 / quantum and the quantum of a block maximum e, as powers of two by their exponent fields: quantum
// 2^(e - 1085 + bits) (the largest contribution below 2^(e - 1022), |sum| < 2^63 quanta), not below 2^-1022
__device__ __forceinline__ double fx_scale(int e, int bits) {
    return __hiloint2double(min(2108 - bits - e, 2045) << 20, 0);
}
__device__ __forceinline__ double fx_quantum(int e, int bits) { return __hiloint2double(max(e - 62 + bits, 1) << 20, 0); }
// p[i] += round(v[i] scale[i]) for NA accumulators in shared memory. A 64-bit shared-memory add is a
// compare-and-swap loop the thread waits for (104 cycles each, one after the other); two 32-bit adds, the
// low words first and then the high words with the carries, are native and overlap (12 values of a full warp:
// 1,254 cycles as 64-bit adds). Sums of integers modulo 2^64: the order of the adds does not matter.
template <int NA>
__device__ __forceinline__ void fx_add(double* const (&p)[NA], const double (&v)[NA], const double (&scale)[NA]) {
    unsigned lo[NA], hi[NA], old[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        const unsigned long long q = (unsigned long long)__double2ll_rn(v[i] * scale[i]);
        lo[i] = (unsigned)q;
        hi[i] = (unsigned)(q >> 32);
    }
#pragma unroll
    for (int i = 0; i < NA; ++i) old[i] = atomicAdd(reinterpret_cast<unsigned*>(p[i]), lo[i]);
#pragma unroll
    for (int i = 0; i < NA; ++i)
        atomicAdd(reinterpret_cast<unsigned*>(p[i]) + 1, hi[i] + (old[i] + lo[i] < lo[i] ? 1u : 0u));
}
// the value of an accumulator (its 64 bits as stored in the double slot p); e == 2047: a non-finite
// contribution was seen
__device__ __forceinline__ double fx_value(const double* p, int e, double quantum) {
    if (e == 2047) return __longlong_as_double(0x7ff8000000000000LL);
    return (double)__double_as_longlong(*p) * quantum;
}
// warp-wide: E[c] = max(E[c], the largest e[c] of the warp's lanes) (shared-memory block maxima); lane c
// holds the maximum of e[c], so one atomic instruction updates all of them
template <int NC>
__device__ __forceinline__ void fx_max(const int (&e)[NC], int* E) {
    const int lane = threadIdx.x & 31;
    unsigned mine = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const unsigned m = __reduce_max_sync(FULL, (unsigned)e[c]);
        if (lane == c) mine = m;
    }
    if (lane < NC && mine) atomicMax(E + lane, (int)mine);
}
// Whether a deposit's maxima E differ from those the one before it had (Ep). With the plasma in global memory a deposit
// adds in the quanta of Ep while it takes its own maxima, which saves a second pass over the particles (1000 cells:
// S deposit 10,900 -> 8,300 cycles per slice, push and deposit 36,500 -> 27,700; with one particle per thread, whose
// values are at hand after the barrier, it gains nothing). A maximum's exponent seldom changes from a slice to the next; when one does, the accumulators are
// cleared and the adds repeated in the quanta of E, so that the quanta always are the slice's own.
template <int NC>
__device__ __forceinline__ bool fx_moved(const int* E, const int* Ep) {
    int d = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) d |= E[c] ^ Ep[c];
    return d != 0;
}
// headroom bits for n contributions per node: 2^bits > 2 n
__device__ __forceinline__ int fx_bits(int n) { return 34 - __clz(n > 1 ? n : 1); }

// ---------------------------------------------------------------- solves by groups of warps
// A slice has three systems with L0 (psi, E_z, B_z) and two with the shifted L1D and L1F (B_r, B_theta). A
// block-wide scan of one row per thread needs 10 (L0) to 16 (pivots) 64-bit shuffles per level and lane for
// all of them, and an SM executes one shuffle per cycle: the five scans took 1,800 to 3,600 cycles each. Here
// every system has its own warps and a thread owns several of its rows: the recurrences run along
// a thread's rows in registers (9 cycles per step), and the shuffles per system drop by the number of rows.
// The psi / E_z / B_z phase went from 9,800 to 7,000 cycles per slice and B+ from 10,800 to 6,900 (512 nodes).
// The row count is odd, so that the lanes' rows lie in different shared-memory banks.
constexpr int kG2 = 5, kG4 = 8;                           // warps per system: 3 x 5 and 2 x 8
constexpr int kTot = 192;                                 // S.tot: 24 + 24 (L0), 64 + 64 + 32 + 32 (B+); block scans 128 + 64
// The words from Smem::lost on; 256 are used. With kTot 2,128 bytes beside the arrays: the largest grid is the
// 1439 nodes (160 bytes each; 1180 with the smoothing filter) that fill a CTA's 227 KB to the last node
constexpr int kMiscBytes = 2128 - 8 * kTot;
__device__ __forceinline__ int group_rows(int M, int warps) { return ((M + 32 * warps - 1) / (32 * warps)) | 1; }
__device__ __forceinline__ void group_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// exclusive sum over a group's threads in thread order (up) or reverse order (!up); tot: one double per warp
template <bool kUp, int kWarps>
__device__ __forceinline__ double group_sum(double v, int wl, double* tot, int id) {
    const int lane = threadIdx.x & 31;
    double s = v;
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        const double t = kUp ? __shfl_up_sync(FULL, s, st) : __shfl_down_sync(FULL, s, st);
        if (kUp ? lane >= st : lane + st < 32) s += t;
    }
    if (lane == (kUp ? 31 : 0)) tot[wl] = s;
    double e = kUp ? __shfl_up_sync(FULL, s, 1) : __shfl_down_sync(FULL, s, 1);
    if (lane == (kUp ? 0 : 31)) e = 0.0;
    group_sync(id, 32 * kWarps);
    double t[kWarps], c = 0.0;                             // (loads first: one shared-memory latency for all)
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t[w] = tot[w];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const int o = kUp ? w : kWarps - 1 - w;
        c += (kUp ? o < wl : o > wl) ? t[o] : 0.0;
    }
    return c + e;
}

// exclusive scan of the affine maps y -> a y + b in thread order (up) or reverse order: y before this
// thread's rows (0 at the start); tot: 2 doubles per warp
template <bool kUp, int kWarps>
__device__ __forceinline__ double group_affine(double a, double b, int wl, double* tot, int id) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        const double ap = kUp ? __shfl_up_sync(FULL, a, st) : __shfl_down_sync(FULL, a, st);
        const double bp = kUp ? __shfl_up_sync(FULL, b, st) : __shfl_down_sync(FULL, b, st);
        if (kUp ? lane >= st : lane + st < 32) { b = fma(a, bp, b); a *= ap; }
    }
    if (lane == (kUp ? 31 : 0)) { tot[2 * wl] = a; tot[2 * wl + 1] = b; }
    double ea = kUp ? __shfl_up_sync(FULL, a, 1) : __shfl_down_sync(FULL, a, 1);
    double eb = kUp ? __shfl_up_sync(FULL, b, 1) : __shfl_down_sync(FULL, b, 1);
    if (lane == (kUp ? 0 : 31)) { ea = 1.0; eb = 0.0; }
    group_sync(id, 32 * kWarps);
    double ta[kWarps], tb[kWarps], c = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        ta[w] = tot[2 * w];
        tb[w] = tot[2 * w + 1];
    }
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const int o = kUp ? w : kWarps - 1 - w;
        const double n = fma(ta[o], c, tb[o]);
        c = (kUp ? o < wl : o > wl) ? n : c;
    }
    return fma(ea, c, eb);
}

// exclusive product (later rows on the left) of the threads' 2x2 matrices, its first column (p, q) up to a
// power of two. The matrices come renormalised (largest entry in [1, 2)): a product of 32 of them stays
// below 2^63, and the column of kWarps renormalised totals below 2^(2 kWarps). tot: 4 doubles per warp
template <int kWarps>
__device__ __forceinline__ void group_pivots(double (&m)[4], double& p, double& q, int wl, double* tot, int id) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
        const double p00 = __shfl_up_sync(FULL, m[0], st), p01 = __shfl_up_sync(FULL, m[1], st);
        const double p10 = __shfl_up_sync(FULL, m[2], st), p11 = __shfl_up_sync(FULL, m[3], st);
        if (lane >= st) {
            const double n00 = m[0] * p00 + m[1] * p10, n01 = m[0] * p01 + m[1] * p11;
            const double n10 = m[2] * p00 + m[3] * p10, n11 = m[2] * p01 + m[3] * p11;
            m[0] = n00; m[1] = n01; m[2] = n10; m[3] = n11;
        }
    }
    renorm(m[0], m[1], m[2], m[3]);
    if (lane == 31)
#pragma unroll
        for (int e = 0; e < 4; ++e) tot[4 * wl + e] = m[e];
    double ex[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) ex[e] = __shfl_up_sync(FULL, m[e], 1);
    if (lane == 0) { ex[0] = 1.0; ex[1] = 0.0; ex[2] = 0.0; ex[3] = 1.0; }
    group_sync(id, 32 * kWarps);
    double c0 = 1.0, c1 = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps - 1; ++w) {
        const double n0 = tot[4 * w] * c0 + tot[4 * w + 1] * c1, n1 = tot[4 * w + 2] * c0 + tot[4 * w + 3] * c1;
        c0 = w < wl ? n0 : c0;
        c1 = w < wl ? n1 : c1;
    }
    p = ex[0] * c0 + ex[1] * c1;
    q = ex[2] * c0 + ex[3] * c1;
}

// (p, q) scaled by the power of two that brings |p| into [1, 2); exact
__device__ __forceinline__ void pivot_scale(double& p, double& q) {
    const int e = (__double2hiint(p) >> 20) & 0x7ff;
    const double s = __hiloint2double((e > 2045 ? 1 : 2046 - e) << 20, 0);
    p *= s;
    q *= s;
}

// q / p for |p| in [1, 2): Newton's iteration for 1/p from a single-precision reciprocal (22 bits, doubled
// twice), then the quotient with one residual correction (Markstein, as Recip). No branch, so the quotients
// of a thread's rows overlap.
__device__ __forceinline__ double pivot_quot(double q, double p) {
    double y = (double)__fdividef(1.0f, (float)p);
    y = fma(y, fma(-p, y, 1.0), y);
    y = fma(y, fma(-p, y, 1.0), y);
    const double r = q * y;
    return fma(fma(-p, r, q), y, r);
}

// doubles per thread of the history kept in shared memory by the sweep variant (0: kept in registers)
constexpr int hist_doubles(int ord, bool reg, int max_r, bool ext) {
    return reg && max_r == 1 && !ext && ord <= 3 ? 5 * ord : 0;
}

// ---------------------------------------------------------------- shared-memory layout
struct Src {                                              // plasma + beam sources of one slice
    double *rhot, *drho, *jz, *chi, *ne, *ni, *jpi1, *S1r, *S1i;
};

struct Smem {
    double *r, *iv, *ih;                                  // grid
    const double *gm, *g0, *gp, *ir;                      // gradient stencils, 1/r
    const double *vw, *gw;                                // L0 in flux form: V / 2 pi, h / r_mid (l0_solve)
    const double *l0r, *l0f, *l0b;                        // L0 Thomas: 1/u, -a/u, -c/u (l0_block)
    const double *l1a, *l1b, *l1c;                        // L1D rows; L1F's differ in row N only (lfa, lfb, c = 0)
    double lfa, lfb;
    double* src0;                                         // sources: 9 arrays, twice when A.dbuf
    double *bgt, *bgr;                                    // neutralising background
    double *psi, *ez, *bz, *wr1, *bpr, *bpi;              // fields of the slice (wr1 = -psi')
    double* tot;                                          // scan scratch of the solves, kTot doubles
    double* hist;                                         // Adams-Bashforth history: slot, component, thread (hist_at)
    double* stage;                                        // A.filter: beam + background part of the next slice (4 x M)
    double* ftot;                                         // A.filter: scan scratch of the filter, 2 x 14 x kW
    int* lost;
    int* flag;                                            // gate result broadcast
    // block maxima of the deposits' exponents: [0, 7) the plasma deposit (rho - J_z, d/dxi, J_z, chi,
    // n_e, n_i, J_theta), [7, 9) the S deposit, [9, 11) the background and neutralising deposits; then
    // counters: [11] extra sub-slices, [12] particles removed as trapped, [13] non-finite deposits
    int* fx;
    int* fxp;                                             // the maxima [0, 9) of the deposits before these
    unsigned long long* cmax;                             // most cells crossed (sub-slicing), as double bits
    long long* tmark;                                     // clock marks of the phase counters: [0] phases, [1] parts
    double* absl;                                         // sub-slicing: xi of the last pushes, twice 8 (AbState)
    // A.pcache > 0 (plasma in global memory, np = A.pcache): a copy of every particle's x y px py Delta w
    // (pc, 6 x np) and its radial cell (pj), written through with the global state whenever a particle
    // moves; the passes that only read the particles take them from here, without a cell search
    double* pc;
    int* pj;
};

// kCS: the constants are in shared memory whatever A says; kHist > 0: sources single-buffered whatever A says, and
// the kHist doubles per thread of the particles' Adams-Bashforth history
template <bool kCS, int kHist>
__device__ __forceinline__ Smem carve(double* base, const SweepArgs& A) {
    // distance between arrays: with the history (M <= kThreads) a constant, so that an element's address is one
    // register and an immediate, and the 29 array pointers take no registers
    const int M = kHist ? kThreads : A.M;
    Smem S;
    double* p = base;
    S.r = p; p += M; S.iv = p; p += M; S.ih = p; p += M;
    // the arrays the sweep reads, behind one another as in A.consts0
    const double* q = p;
    if constexpr (!kCS)
        if (!A.const_smem) q = A.consts0;
    S.gm = q; S.g0 = q + M; S.gp = q + 2 * M; S.ir = q + 3 * M;
    S.l1a = q + 4 * M; S.l1b = q + 5 * M; S.l1c = q + 6 * M;
    S.vw = q + 7 * M; S.gw = q + 8 * M;                   // up to kThreads nodes
    S.l0r = q + 7 * M; S.l0f = q + 8 * M; S.l0b = q + 9 * M;   // more
    S.lfa = A.lfa_N; S.lfb = A.lfb_N;
    if (kCS || A.const_smem) p += (size_t)consts0_arrays(A.M) * M;
    S.src0 = p;
    p += (!kHist && A.dbuf ? 18 : 9) * (size_t)M;
    S.bgt = p; p += M; S.bgr = p; p += M;
    S.psi = p; p += M; S.ez = p; p += M; S.bz = p; p += M; S.wr1 = p; p += M; S.bpr = p; p += M; S.bpi = p; p += M;
    S.tot = p; p += kTot;
    S.hist = p; p += kHist * kThreads;
    S.stage = S.ftot = nullptr;
    if (A.filter) { S.stage = p; p += 4 * (size_t)M; S.ftot = p; p += 2 * 14 * kW; }
    S.lost = reinterpret_cast<int*>(p);
    S.flag = S.lost + 1;
    S.fx = S.lost + 2;
    S.cmax = reinterpret_cast<unsigned long long*>(S.lost + 16);
    S.fxp = S.lost + 18;
    S.tmark = reinterpret_cast<long long*>(S.lost + 28);
    S.absl = reinterpret_cast<double*>(S.lost + 32);
    S.pc = A.pcache ? reinterpret_cast<double*>(reinterpret_cast<char*>(S.lost) + kMiscBytes) : nullptr;
    S.pj = A.pcache ? reinterpret_cast<int*>(S.pc + 6 * (size_t)A.pcache) : nullptr;
    return S;
}

__device__ __forceinline__ Src src_of(const Smem& S, int M, int b) {
    double* p = S.src0 + (size_t)b * 9 * M;
    Src s;
    s.rhot = p; s.drho = p + M; s.jz = p + 2 * M; s.chi = p + 3 * M; s.ne = p + 4 * M;
    s.ni = p + 5 * M; s.jpi1 = p + 6 * M; s.S1r = p + 7 * M; s.S1i = p + 8 * M;
    return s;
}

// beam source values of slice k at node j needed by the m = 0 sweep (src/Simulation.cpp:420-441):
// rho - J_z, its xi-derivative (central / one-sided, or backward for ngp), J_z, J_theta
struct BeamRow { double rt, drt, jz, jt; };

template <bool kL2>                       // kL2: the rows were written by other SMs, read them from L2
__device__ __forceinline__ double ldb(const double* p) { return kL2 ? __ldcg(p) : *p; }

// one beam-source value at p (inside bsrc; NC values per node): the pushed beams' deposit plus, in kernels built
// for it (kStat), the static (analytic) sources when present
template <bool kL2, bool kStat>
__device__ __forceinline__ double ldbs(const SweepArgs& A, const double* bsrc, const double* p) {
    const double v = ldb<kL2>(p);
    if constexpr (kStat) return A.bstat ? v + __ldg(A.bstat + (p - bsrc)) : v;
    return v;
}

// component c of node j of the guard row (the slice ahead of a later slab's first one): doubles, or two
// limbs (the high row, then the low row M B_NC0 values further) when bsrc has the exact format
__device__ __forceinline__ double guard_at(const SweepArgs& A, int j, int c) {
    if (!A.bguard) return 0.0;
    const double* g = A.bguard + (size_t)j * B_NC0 + c;
    return A.bq ? beam_fx_value(g[0], g[(size_t)A.M * B_NC0], A.bq[j], A.bfx_2s) : g[0];
}

template <bool kL2, bool kStat = false>
__device__ __forceinline__ BeamRow beam_row(const SweepArgs& A, const double* bsrc, int k, int j) {
    const size_t st = (size_t)A.M * A.bcs;
    const double* const bj = bsrc + (size_t)j * A.bcs;
    // component c (in place o of a node) of row kk: a double, or the exact two-limb accumulator (A.bq) turned
    // into its value
    const double qj = A.bq ? A.bq[j] : 0.0;
    auto ld = [&](int kk, int o, int c) -> double {
        const double* p = bj + (size_t)kk * st + o;
        double v = ldb<kL2>(p);
        if (A.bq) v = beam_fx_value(v, ldb<kL2>(p + A.bfx_lo), qj, A.bfx_2s);
        if constexpr (kStat) return A.bstat ? v + __ldg(A.bstat + ((size_t)kk * A.M + j) * B_NC0 + c) : v;
        return v;
    };
    auto rt = [&](int kk) { return ld(kk, B_RT0, B_RT0); };
    BeamRow r;
    r.rt = rt(k);
    r.jz = ld(k, B_JZ0, B_JZ0);
    r.jt = ld(k, A.bjt, B_JP1I);
    const int K = A.K;
    // the slice ahead of slice 0: none at the box head, the guard row in a later slab of a staged run
    const double guard = guard_at(A, j, B_RT0);
    if (A.ngp) {
        r.drt = (r.rt - (k > 0 ? rt(k - 1) : guard)) * A.idxi;
    } else if (K == 1) {
        r.drt = 0.0;
    } else if (k == 0) {
        r.drt = A.bguard ? 0.5 * (rt(1) - guard) * A.idxi : (rt(1) - r.rt) * A.idxi;
    } else if (k == K - 1) {
        r.drt = (r.rt - rt(k - 1)) * A.idxi;
    } else {
        r.drt = 0.5 * (rt(k + 1) - rt(k - 1)) * A.idxi;
    }
    return r;
}

// the values beam_row needs, loaded and not yet used: rho - J_z, J_z, J_theta of row k and rho - J_z of the
// rows ahead of and behind it (w: their low limbs in the exact format)
struct BeamRaw { double v[5], w[5]; };
template <bool kL2>
__device__ __forceinline__ void raw_load(const SweepArgs& A, const double* bsrc, int k, int j, BeamRaw& b) {
    const size_t st = (size_t)A.M * A.bcs;
    const double* const bk = bsrc + (size_t)k * st + (size_t)j * A.bcs;
    const double* const p[5] = {bk + B_RT0, bk + B_JZ0, bk + A.bjt, k > 0 ? bk + B_RT0 - (ptrdiff_t)st : bk + B_RT0,
                                k + 1 < A.K ? bk + st + B_RT0 : bk + B_RT0};
#pragma unroll
    for (int c = 0; c < 5; ++c) b.v[c] = ldb<kL2>(p[c]);
    if (A.bq)
#pragma unroll
        for (int c = 0; c < 5; ++c) b.w[c] = ldb<kL2>(p[c] + A.bfx_lo);
}
// beam_row of slice k > 0 from its loaded values; with static sources (which raw_load leaves out) beam_row itself
template <bool kL2, bool kStat>
__device__ __forceinline__ BeamRow raw_row(const SweepArgs& A, const double* bsrc, int k, int j, const BeamRaw& b) {
    if constexpr (kStat)
        if (A.bstat) return beam_row<kL2, kStat>(A, bsrc, k, j);
    double v[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) v[c] = A.bq ? beam_fx_value(b.v[c], b.w[c], A.bq[j], A.bfx_2s) : b.v[c];
    BeamRow r;
    r.rt = v[0];
    r.jz = v[1];
    r.jt = v[2];
    if (A.ngp || k == A.K - 1) r.drt = (v[0] - v[3]) * A.idxi;
    else r.drt = 0.5 * (v[4] - v[3]) * A.idxi;
    return r;
}

// initial source values of a slice: background + beam; the plasma deposit is added on top. With the
// smoothing filter (kernels built with kExt only) the plasma deposit starts from zero and the beam +
// background part is staged, to be added after the filter (filter_sources).
template <bool kExt>
__device__ __forceinline__ void init_sources(const Src& s, const Smem& S, int j, const BeamRow& br, int M) {
    if (kExt && S.stage) {
        S.stage[j] = S.bgt[j] + br.rt;
        S.stage[M + j] = br.drt;
        S.stage[2 * M + j] = br.jz;
        S.stage[3 * M + j] = br.jt;
        s.rhot[j] = 0.0;
        s.drho[j] = 0.0;
        s.jz[j] = 0.0;
        s.jpi1[j] = 0.0;
        s.ni[j] = 0.0;
    } else {
        s.rhot[j] = S.bgt[j] + br.rt;
        s.drho[j] = br.drt;
        s.jz[j] = br.jz;
        s.jpi1[j] = br.jt;
        s.ni[j] = S.bgr[j] > 0.0 ? S.bgr[j] : 0.0;
    }
    s.chi[j] = 0.0;
    s.ne[j] = 0.0;
    s.S1r[j] = 0.0;
    s.S1i[j] = 0.0;
}

// the values a slice's 7 deposit arrays start from at node j (init_sources' values, for deposits
// whose accumulators cannot hold them); with the smoothing filter the beam + background part goes to
// the stage and the arrays start from zero
template <bool kExt>
__device__ __forceinline__ void init_base(const Smem& S, int j, const BeamRow& br, int M, double (&base)[7]) {
    if (kExt && S.stage) {
        S.stage[j] = S.bgt[j] + br.rt;
        S.stage[M + j] = br.drt;
        S.stage[2 * M + j] = br.jz;
        S.stage[3 * M + j] = br.jt;
#pragma unroll
        for (int c = 0; c < 7; ++c) base[c] = 0.0;
    } else {
        base[0] = S.bgt[j] + br.rt;
        base[1] = br.drt;
        base[2] = br.jz;
        base[3] = 0.0;
        base[4] = 0.0;
        base[5] = S.bgr[j] > 0.0 ? S.bgr[j] : 0.0;
        base[6] = br.jt;
    }
}

// The radial smoothing filter f <- F_n^{-1} f (FieldSolver::filter, src/FieldSolver.cpp:148-161) of NS
// shared-memory arrays in place, each with F0 (op 0) or F1 (op 1): Thomas with the host-factored pivots
// A.fconsts, its two substitutions as block scans over the thread's rows [row0, row0 + Rw). Every thread
// reads and writes only its own rows; the caller puts a barrier before (the arrays are complete) and, when
// other threads read them next, after. Only the kernel variants for filtered decks (EXT) contain it.
template <int NS>
struct FilterSet { double* f[NS]; int op[NS]; };

template <int NS, int kMaxR>
__device__ __forceinline__ void filter_rows(const FilterSet<NS> fs, const double* __restrict__ fc, int M, int Rw,
                                         double* tot) {
    const int row0 = threadIdx.x * Rw;
    double a[NS], b[NS], d[kMaxR][NS];
#pragma unroll
    for (int e = 0; e < NS; ++e) { a[e] = 1.0; b[e] = 0.0; }
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
#pragma unroll
        for (int e = 0; e < NS; ++e) {
            d[u][e] = 0.0;
            if (u >= Rw || i >= M) continue;
            const double* F = fc + (size_t)fs.op[e] * 3 * M;
            d[u][e] = fs.f[e][i];
            const double rr = F[i], af = F[M + i];
            b[e] = fma(af, b[e], rr * d[u][e]);
            a[e] *= af;
        }
    }
    double y[NS];
    scan_fwd_n<NS>(a, b, y, tot);
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
#pragma unroll
        for (int e = 0; e < NS; ++e) {
            if (u >= Rw || i >= M) continue;
            const double* F = fc + (size_t)fs.op[e] * 3 * M;
            y[e] = fma(F[M + i], y[e], F[i] * d[u][e]);
            d[u][e] = y[e];
        }
    }
#pragma unroll
    for (int e = 0; e < NS; ++e) { a[e] = 1.0; b[e] = 0.0; }
#pragma unroll
    for (int u = kMaxR - 1; u >= 0; --u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
#pragma unroll
        for (int e = 0; e < NS; ++e) {
            const double ab = fc[(size_t)fs.op[e] * 3 * M + 2 * M + i];
            b[e] = fma(ab, b[e], d[u][e]);
            a[e] *= ab;
        }
    }
    double x[NS];
    scan_bwd_n<NS>(a, b, x, tot + 2 * NS * kW);
#pragma unroll
    for (int u = kMaxR - 1; u >= 0; --u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
#pragma unroll
        for (int e = 0; e < NS; ++e) {
            x[e] = fma(fc[(size_t)fs.op[e] * 3 * M + 2 * M + i], x[e], d[u][e]);
            fs.f[e][i] = x[e];
        }
    }
}

// Simulation::filter_plasma_sources (src/Simulation.cpp:823-835, m = 0) on the plasma deposit of a slice,
// then the staged beam + background part added as combine_sources does (src/Simulation.cpp:430-437):
// rho - J_z, its xi-derivative, J_z, chi, n_e, n_i with F0 and J_theta with F1. Ends with a barrier.
template <int kMaxR>
__device__ __forceinline__ void filter_sources(const Src& s, const Smem& S, const SweepArgs& A, int Rw) {
    FilterSet<7> fs;
    double* arr[7] = {s.rhot, s.drho, s.jz, s.chi, s.ne, s.ni, s.jpi1};
#pragma unroll
    for (int e = 0; e < 7; ++e) { fs.f[e] = arr[e]; fs.op[e] = e == 6 ? 1 : 0; }
    filter_rows<7, kMaxR>(fs, A.fconsts, A.M, Rw, S.ftot);
    const int M = A.M, row0 = threadIdx.x * Rw;
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
        s.rhot[i] += S.stage[i];
        s.drho[i] += S.stage[M + i];
        s.jz[i] += S.stage[2 * M + i];
        s.jpi1[i] += S.stage[3 * M + i];
        if (S.bgr[i] > 0.0) s.ni[i] += S.bgr[i];
    }
    __syncthreads();
}

// 3-point non-uniform gradient at node i (src/FieldSolver.cpp:193-211); odd: axis value f1/r1
__device__ __forceinline__ double grad_at(const Smem& S, int N, const double* f, int i, bool odd) {
    if (i == 0) return odd ? f[1] * S.ir[0] : 0.0;
    if (i == N) return S.g0[N] * f[N] + S.gm[N] * f[N - 1] + S.gp[N] * f[N - 2];
    return S.gm[i] * f[i - 1] + S.g0[i] * f[i] + S.gp[i] * f[i + 1];
}

// cell of x starting from a guess (the previous cell): walks for small moves, bisects otherwise;
// the same cell as locate() (src/RadialGrid.hpp:35-44) for every x
__device__ __forceinline__ int locate_from(const double* __restrict__ r, int N, double R, double x, int j) {
    if (x <= 0.0) return 0;
    if (x >= R) return N - 1;
    j = j < 0 ? 0 : (j > N - 1 ? N - 1 : j);
#pragma unroll 1
    for (int step = 0; step < 3; ++step) {
        if (r[j] > x) { if (j == 0) break; --j; continue; }
        if (r[j + 1] <= x) { if (j == N - 1) break; ++j; continue; }
        return j;
    }
    if (r[j] <= x && x < r[j + 1]) return j;
    return locate(r, N, R, x);
}

// two neighbouring doubles: one 16-byte store when v16 (p on a 16-byte boundary)
__device__ __forceinline__ void put2(double* p, double a, double b, bool v16) {
    if (v16) {
        *reinterpret_cast<double2*>(p) = make_double2(a, b);
    } else {
        p[0] = a;
        p[1] = b;
    }
}

// ---------------------------------------------------------------- one plasma particle
// history h[m] holds the force m pushes ago (h[0] newest): the reference's ring buffer
// (src/PlasmaSpecies.cpp:621-632) with the slot rotation done by moving values.
template <int ORD>
struct PState {
    double x, y, px, py, dl, w;
    double h[ORD][5];
    double q, qm;
};

template <int ORD>
__device__ __forceinline__ void pload(PState<ORD>& P, const double* __restrict__ ps, int npad, int p) {
    P.x = ps[p]; P.y = ps[npad + p]; P.px = ps[2 * (size_t)npad + p]; P.py = ps[3 * (size_t)npad + p];
    P.dl = ps[4 * (size_t)npad + p]; P.w = ps[5 * (size_t)npad + p];
#pragma unroll
    for (int m = 0; m < ORD; ++m)
#pragma unroll
        for (int v = 0; v < 5; ++v) P.h[m][v] = ps[(6 + (size_t)m * 5 + v) * npad + p];
}

template <int ORD>
__device__ __forceinline__ void pstore(const PState<ORD>& P, double* __restrict__ ps, int npad, int p) {
    ps[p] = P.x; ps[npad + p] = P.y; ps[2 * (size_t)npad + p] = P.px; ps[3 * (size_t)npad + p] = P.py;
    ps[4 * (size_t)npad + p] = P.dl; ps[5 * (size_t)npad + p] = P.w;
#pragma unroll
    for (int m = 0; m < ORD; ++m)
#pragma unroll
        for (int v = 0; v < 5; ++v) ps[(6 + (size_t)m * 5 + v) * npad + p] = P.h[m][v];
}

// history m pushes ago of thread tid's particle in the shared ring whose newest slot is hs
template <int ORD>
__device__ __forceinline__ double* hist_at(const Smem& S, int hs, int m) {
    const int slot = hs - m < 0 ? hs - m + ORD : hs - m;
    return S.hist + (size_t)slot * 5 * kThreads + threadIdx.x;
}
template <int ORD>
__device__ __forceinline__ void hist_get(PState<ORD>& P, const Smem& S, int hs) {
#pragma unroll
    for (int m = 0; m < ORD; ++m) {
        const double* h = hist_at<ORD>(S, hs, m);
#pragma unroll
        for (int v = 0; v < 5; ++v) P.h[m][v] = h[v * kThreads];
    }
}
template <int ORD>
__device__ __forceinline__ void hist_put(const PState<ORD>& P, const Smem& S, int hs, bool all) {
#pragma unroll
    for (int m = 0; m < ORD; ++m) {
        if (m > 0 && !all) break;
        double* h = hist_at<ORD>(S, hs, m);
#pragma unroll
        for (int v = 0; v < 5; ++v) h[v * kThreads] = P.h[m][v];
    }
}

// x y px py Delta w of particle p: from the shared copy (A.pcache) or from the global state
template <int ORD>
__device__ __forceinline__ void pbase(PState<ORD>& P, const Smem& S, const SweepArgs& A, const double* __restrict__ ps,
                                      int npad, int p) {
    if (A.pcache) {
        const size_t n = (size_t)A.pcache;
        P.x = S.pc[p]; P.y = S.pc[n + p]; P.px = S.pc[2 * n + p]; P.py = S.pc[3 * n + p];
        P.dl = S.pc[4 * n + p]; P.w = S.pc[5 * n + p];
    } else {
        P.x = ps[p]; P.y = ps[npad + p]; P.px = ps[2 * (size_t)npad + p]; P.py = ps[3 * (size_t)npad + p];
        P.dl = ps[4 * (size_t)npad + p]; P.w = ps[5 * (size_t)npad + p];
    }
}
template <int ORD>
__device__ __forceinline__ void pbase_put(const PState<ORD>& P, const Smem& S, const SweepArgs& A, int p) {
    if (!A.pcache) return;
    const size_t n = (size_t)A.pcache;
    S.pc[p] = P.x; S.pc[n + p] = P.y; S.pc[2 * n + p] = P.px; S.pc[3 * n + p] = P.py;
    S.pc[4 * n + p] = P.dl; S.pc[5 * n + p] = P.w;
}
// AB history of particle p from the global state
template <int ORD>
__device__ __forceinline__ void phist(PState<ORD>& P, const double* __restrict__ ps, int npad, int p) {
#pragma unroll
    for (int m = 0; m < ORD; ++m)
#pragma unroll
        for (int v = 0; v < 5; ++v) P.h[m][v] = ps[(6 + (size_t)m * 5 + v) * npad + p];
}

// the geometry of particle p at (x, y): from its kept cell (A.pcache; the cell locate() would find) or by
// the search
__device__ __forceinline__ PGeo pgeo(const Smem& S, const SweepArgs& A, int N, double R, int p, double x, double y) {
    return A.pcache ? geometry_in(S.r, S.ih, x, y, S.pj[p]) : geometry(S.r, S.ih, N, R, x, y);
}

__device__ __forceinline__ void species_params(const SweepArgs& A, int p, double& q, double& qm) {
    int s = 0;
    while (s + 1 < A.nsp && p >= A.sp_off[s + 1]) ++s;
    q = A.sp_q[s];
    qm = A.sp_qm[s];
}

// gamma = (1 + p_perp^2 + Delta^2) / 2 Delta and 1 / Delta of a particle
struct PKin { double gam, invd; };
__device__ __forceinline__ PKin kin_of(double px, double py, double d) {
    const Recip q(d);
    PKin k;
    k.invd = q.y;
    k.gam = 0.5 * q(1.0 + px * px + py * py + d * d);
    return k;
}
// the same from the particle's state, where nothing is kept from phase to phase (plasma in global memory; with plain
// divisions: sharing reciprocals gained 2 % there)
struct KinNone {};
__device__ __forceinline__ void kin_get(const PKin& k, double, double, double, double& gam, double& invd) {
    gam = k.gam;
    invd = k.invd;
}
__device__ __forceinline__ void kin_get(KinNone, double px, double py, double d, double& gam, double& invd) {
    gam = (1.0 + px * px + py * py + d * d) / (2.0 * d);
    invd = 1.0 / d;
}
__device__ __forceinline__ double kin_next(PKin& k, double px, double py, double d) { return (k = kin_of(px, py, d)).gam; }
__device__ __forceinline__ double kin_next(KinNone&, double px, double py, double d) {
    return (1.0 + px * px + py * py + d * d) / (2.0 * d);
}
// What the phases of a slice need of a particle whose state is kept in registers, computed once per push: its
// polar position and kinematics (a square root and two reciprocals)
struct PKeep {
    double rp, ir, c, s;
    PKin k;
};
__device__ __forceinline__ PGeo keep_geo(const Smem& S, const PKeep& K, int j) {
    return geometry_at(S.r, S.ih, j, K.rp, K.ir, K.c, K.s);
}

// W+ mode 1 at the particle: lin(w1), w1 = -psi' (src/Simulation.cpp:477-498)
__device__ __forceinline__ double w1_at(const Smem& S, int N, const PGeo& g) { return lin(S.wr1, g); }

// src/PlasmaSpecies.cpp:409-478, m = 0 (plasma rho and J_r feed nothing on this path: not deposited).
// Contributions of one particle to nodes j (v[0..5]) and j+1 (v[6..11]): rho - J_z, d/dxi, J_z, chi,
// density, J_theta.
template <int ORD, class Kin>
__device__ __forceinline__ void deposit_values(const PState<ORD>& P, const PGeo& g, const Kin& kin, const Smem& S,
                                               double (&v)[12]) {
    const double PX = P.px, PY = P.py, D = P.dl, w = P.w;
    double gam, invd;
    kin_get(kin, PX, PY, D, gam, invd);
    const double pz = gam - D;
    const double ux = PX * invd, uy = PY * invd;
    const double ur = g.c * ux + g.s * uy, uth = g.c * uy - g.s * ux;
    const double wq = w * P.q;
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
        const int jj = g.j + cc;
        const double iv = S.iv[jj];
        const double Wc = cc ? g.W1 : g.W0;
        const double dWc = cc ? g.ih : -g.ih;
        const double a = wq * Wc * iv;
        const double dr = wq * ur * dWc * iv;
        const double vjz = a * pz * invd, vchi = a * P.qm * invd;
        const double vn = w * Wc * iv * gam * invd;
        v[6 * cc + 0] = a;
        v[6 * cc + 1] = dr;
        v[6 * cc + 2] = vjz;
        v[6 * cc + 3] = vchi;
        v[6 * cc + 4] = vn;
        v[6 * cc + 5] = a * uth;
    }
}

// The plasma deposit of a slice, exact (see fx_add): phase A sums each warp's runs of equal
// (cell, species sign) and takes the block maxima of the run sums' exponents; phase B adds the quantised run sums
// into the accumulator arrays (at once in the quanta of the deposit before, again after a barrier when the maxima
// moved: fx_moved); after another barrier deposit_finish turns the accumulators into values. The 7 arrays in this order: rho - J_z, d/dxi, J_z, chi, n_e, n_i,
// J_theta (n_e takes the negative species, n_i the positive ones).
__device__ __forceinline__ double* dep_arr(const Src& s, int c) {
    switch (c) {
        case 0: return s.rhot;
        case 1: return s.drho;
        case 2: return s.jz;
        case 3: return s.chi;
        case 4: return s.ne;
        case 5: return s.ni;
        default: return s.jpi1;
    }
}

// warp-wide phase A: every lane calls it (active = the lane has a particle); key = 2 j + (positive
// species). Returns whether the lane holds a run sum to add; kExp: also take the exponent maxima
// into E (a deposit that recomputes its values for phase B calls it again without)
template <bool kExp>
__device__ __forceinline__ bool deposit_runs(bool active, int j, bool neg, double (&v)[12], int* E) {
    const int lane = threadIdx.x & 31;
    if (!active)
#pragma unroll
        for (int i = 0; i < 12; ++i) v[i] = 0.0;
    const int key = active ? 2 * j + (neg ? 0 : 1) : -1 - lane;
    const bool tail = warp_runs_sum<12>(key, v) && active;
    if constexpr (kExp) {
        int e[7] = {0, 0, 0, 0, 0, 0, 0};
        if (tail) {
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const int ec = max(fx_bexp(v[c]), fx_bexp(v[6 + c]));
                if (c < 4) e[c] = ec;
                else if (c == 4) e[neg ? 4 : 5] = ec;
                else e[6] = ec;
            }
        }
        fx_max<7>(e, E);
    }
    return tail;
}

// phase B: the run sum of a tail lane into the accumulators of nodes j and j + 1
__device__ __forceinline__ void deposit_add(bool tail, int j, bool neg, const double (&v)[12], const Src& acc,
                                            const int* E, int bits) {
    if (!tail) return;
    const double s0 = fx_scale(E[0], bits), s1 = fx_scale(E[1], bits), s2 = fx_scale(E[2], bits);
    const double s3 = fx_scale(E[3], bits), s4 = fx_scale(E[neg ? 4 : 5], bits), s6 = fx_scale(E[6], bits);
    double* const dens = neg ? acc.ne : acc.ni;
    double* const adr[12] = {acc.rhot + j, acc.drho + j, acc.jz + j, acc.chi + j, dens + j, acc.jpi1 + j,
                             acc.rhot + j + 1, acc.drho + j + 1, acc.jz + j + 1, acc.chi + j + 1, dens + j + 1,
                             acc.jpi1 + j + 1};
    const double sc[12] = {s0, s1, s2, s3, s4, s6, s0, s1, s2, s3, s4, s6};
    fx_add<12>(adr, v, sc);
}

__device__ __forceinline__ void deposit_clear(const Src& acc, int M) {
    for (int j = threadIdx.x; j < M; j += kThreads)
#pragma unroll
        for (int c = 0; c < 7; ++c) dep_arr(acc, c)[j] = 0.0;
}

// the values of node j: dst = base + accumulated deposit (acc and dst may be the same arrays)
__device__ __forceinline__ void deposit_finish(const Src& dst, const Src& acc, int j, const double (&base)[7],
                                               const int* E, int bits) {
#pragma unroll
    for (int c = 0; c < 7; ++c)
        dep_arr(dst, c)[j] = base[c] + fx_value(dep_arr(acc, c) + j, E[c], fx_quantum(E[c], bits));
}

// src/PlasmaSpecies.cpp:508-559, m = 0: S+ contributions to nodes j (v[0..1]) and j+1 (v[2..3])
template <int ORD, class Kin>
__device__ __forceinline__ void depositS_values(const PState<ORD>& P, const PGeo& g, const Kin& kin, const Smem& S,
                                                int N, double (&v)[4]) {
    const double qm = P.qm;
    const double PX = P.px, PY = P.py;
    const double r1 = w1_at(S, N, g);
    const double Wx = r1 * g.c - 0.0 * g.s, Wy = r1 * g.s + 0.0 * g.c;
    const double Ez = lin(S.ez, g), Bz = lin(S.bz, g);
    double gam, invd;
    kin_get(kin, PX, PY, P.dl, gam, invd);
    const double ux = PX * invd, uy = PY * invd;
    const double ur = g.c * ux + g.s * uy, uth = g.c * uy - g.s * ux;
    const double dD = qm * ((PX * Wx + PY * Wy) * invd - Ez);
    const double ax = (qm * (gam * Wx + PY * Bz) * invd) * invd - PX * dD * invd * invd;
    const double ay = (qm * (gam * Wy - PX * Bz) * invd) * invd - PY * dD * invd * invd;
    const double wq = P.w * P.q;
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
        const int jj = g.j + cc;
        const double iv = S.iv[jj] * wq;
        const double Wc = cc ? g.W1 : g.W0;
        const double dWc = cc ? g.ih : -g.ih;
        const double Worc = cc ? g.Wor1 : g.Wor0;
        double Ar = ax * Wc + ux * ur * dWc;
        double Ai = ay * Wc + uy * ur * dWc;
        const double f2 = uth * Worc;
        Ar += f2 * uy;
        Ai -= f2 * ux;
        v[2 * cc] = iv * (Ar * g.c + Ai * g.s);
        v[2 * cc + 1] = iv * (Ai * g.c - Ar * g.s);
    }
}

// the S deposit of a slice, exact like the plasma deposit: phase A (run sums, exponent maxima into
// E[0..1] for S_r, S_i), phase B after a barrier (adds into the slice's S arrays, which start at 0),
// then each thread turns its own rows into values (depositS_finish) before the B+ solve reads them
template <bool kExp>
__device__ __forceinline__ bool depositS_runs(bool active, int j, double (&v)[4], int* E) {
    const int lane = threadIdx.x & 31;
    if (!active)
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = 0.0;
    const int key = active ? j : -1 - lane;
    const bool tail = warp_runs_sum<4>(key, v) && active;
    if constexpr (kExp) {
        int e[2] = {0, 0};
        if (tail) {
            e[0] = max(fx_bexp(v[0]), fx_bexp(v[2]));
            e[1] = max(fx_bexp(v[1]), fx_bexp(v[3]));
        }
        fx_max<2>(e, E);
    }
    return tail;
}

__device__ __forceinline__ void depositS_add(bool tail, int j, const double (&v)[4], const Src& s, const int* E,
                                             int bits) {
    if (!tail) return;
    const double sr = fx_scale(E[0], bits), si = fx_scale(E[1], bits);
    double* const adr[4] = {s.S1r + j, s.S1i + j, s.S1r + j + 1, s.S1i + j + 1};
    const double sc[4] = {sr, si, sr, si};
    fx_add<4>(adr, v, sc);
}

__device__ __forceinline__ void depositS_finish(const Src& s, int i, const int* E, int bits) {
    s.S1r[i] = fx_value(s.S1r + i, E[0], fx_quantum(E[0], bits));
    s.S1i[i] = fx_value(s.S1i + i, E[1], fx_quantum(E[1], bits));
}

// src/PlasmaSpecies.cpp:561-668 with uniform steps (the classical AB coefficients); returns 1 when the
// particle moved (2 when the wall reflected it, its whole history with it), 0 when it was removed beyond the wall, -1 when removed as trapped (Delta <= delta_min
// or gamma > max_qsa Delta: no longer quasi-static, src/PlasmaSpecies.cpp:636-650). kin: the particle's
// kinematics before the push, on return those after it (or KinNone)
template <int ORD, class Kin>
__device__ __forceinline__ int push_particle(PState<ORD>& P, const PGeo& g, Kin& kin, const Smem& S,
                                             const SweepArgs& A, bool first, const double (&ab)[5], double h) {
    const double qm = P.qm;
    const double X = P.x, Y = P.y, PX = P.px, PY = P.py, D = P.dl;
    const double r1 = w1_at(S, A.N, g);
    const double Wx = r1 * g.c - 0.0 * g.s, Wy = r1 * g.s + 0.0 * g.c;
    const double Ez = lin(S.ez, g), Bz = lin(S.bz, g);
    const double br = lin(S.bpr, g), bi = lin(S.bpi, g);
    const double Bx = br * g.c - bi * g.s, By = br * g.s + bi * g.c;
    double gam, invd;
    kin_get(kin, PX, PY, D, gam, invd);
    double fv[5];
    fv[0] = PX * invd;
    fv[1] = PY * invd;
    fv[2] = qm * (gam * Wx * invd + By + PY * Bz * invd);
    fv[3] = qm * (gam * Wy * invd - Bx - PX * Bz * invd);
    fv[4] = qm * ((PX * Wx + PY * Wy) * invd - Ez);
    if (first) {
#pragma unroll
        for (int m = 0; m < ORD; ++m)
#pragma unroll
            for (int v = 0; v < 5; ++v) P.h[m][v] = fv[v];
    } else {
#pragma unroll
        for (int m = ORD - 1; m > 0; --m)
#pragma unroll
            for (int v = 0; v < 5; ++v) P.h[m][v] = P.h[m - 1][v];
#pragma unroll
        for (int v = 0; v < 5; ++v) P.h[0][v] = fv[v];
    }
    double sum[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int m = 0; m < ORD; ++m) {
        const double cm = ab[m];
#pragma unroll
        for (int v = 0; v < 5; ++v) sum[v] += cm * P.h[m][v];
    }
    const double dxi = h;
    double xn = X + dxi * sum[0], yn = Y + dxi * sum[1];
    double pxn = PX + dxi * sum[2], pyn = PY + dxi * sum[3];
    const double dn = D + dxi * sum[4];
    const double gn = kin_next(kin, pxn, pyn, dn);
    if (!(dn > A.delta_min) || gn > A.max_qsa * dn) {
        P.w = 0.0;
        return -1;
    }
    const double R = A.R;
    const double rn = sqrt(xn * xn + yn * yn);
    int moved = 1;
    if (rn > R) {                    // specular reflection at the wall, incl. the history
        moved = 2;
        const double nx = xn / rn, ny = yn / rn;
        const double rr = 2.0 * R - rn;
        if (rr < 0.0) { P.w = 0.0; return 0; }
        xn = nx * rr; yn = ny * rr;
        const double pn = pxn * nx + pyn * ny;
        pxn -= 2.0 * pn * nx; pyn -= 2.0 * pn * ny;
        (void)kin_next(kin, pxn, pyn, dn);
#pragma unroll
        for (int m = 0; m < ORD; ++m) {
            const double a = P.h[m][0] * nx + P.h[m][1] * ny;
            P.h[m][0] -= 2.0 * a * nx; P.h[m][1] -= 2.0 * a * ny;
            const double b = P.h[m][2] * nx + P.h[m][3] * ny;
            P.h[m][2] -= 2.0 * b * nx; P.h[m][3] -= 2.0 * b * ny;
        }
    }
    P.x = xn; P.y = yn; P.px = pxn; P.py = pyn; P.dl = dn;
    return moved;
}

// Adams-Bashforth coefficients for history points t[0..ord) (t[0] the newest push) and the step h: the
// integrals over [t0, t0 + h] of the Lagrange basis, by 3-point Gauss-Legendre (exact for the degree <= 4
// needed), src/PlasmaSpecies.cpp:30-48
template <int ORD>
__device__ __forceinline__ void ab_variable(const double (&t)[ORD], double h, double (&c)[5]) {
    const double gx[3] = {-0.7745966692414834, 0.0, 0.7745966692414834};
    const double gw[3] = {5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0};
#pragma unroll
    for (int m = 0; m < 5; ++m) c[m] = 0.0;
#pragma unroll
    for (int m = 0; m < ORD; ++m) {
        double sm = 0.0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double tt = t[0] + 0.5 * h * (1.0 + gx[q]);
            double l = 1.0;
#pragma unroll
            for (int n = 0; n < ORD; ++n)
                if (n != m) l *= (tt - t[n]) / (t[m] - t[n]);
            sm += 0.5 * gw[q] * l;
        }
        c[m] = sm;
    }
}

// the radial cells a particle would cross in a step of dxi: its straight path's length over the cell
// size at the path's closest approach to the axis (src/PlasmaSpecies.cpp:814-830)
__device__ __forceinline__ double cells_crossed(const Smem& S, int N, double R, double X, double Y, double PX,
                                                double PY, double D, double dxi) {
    const double X1 = X + dxi * PX / D, Y1 = Y + dxi * PY / D;
    const double dx = X1 - X, dy = Y1 - Y, l2 = dx * dx + dy * dy;
    double t = l2 > 0.0 ? -(X * dx + Y * dy) / l2 : 0.0;
    t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
    const double xm = X + t * dx, ym = Y + t * dy;
    return sqrt(l2) * S.ih[locate(S.r, N, R, sqrt(xm * xm + ym * ym))];
}

// the beam sources of a sub-slice at xi_k + ds: slice k's, extrapolated linearly with their xi-derivative
// (src/Simulation.cpp:431-432); the derivative of rho - J_z itself is slice k's
template <bool kL2, bool kStat>
__device__ __forceinline__ BeamRow beam_row_at(const SweepArgs& A, const double* bsrc, int k, int j, double ds) {
    BeamRow r = beam_row<kL2, kStat>(A, bsrc, k, j);
    if (ds == 0.0) return r;
    // the xi-derivatives of J_z and J_theta by the same difference as that of rho - J_z
    const int K = A.K;
    auto row = [&](int kk) { return beam_row<kL2, kStat>(A, bsrc, kk, j); };
    double djz = 0.0, djt = 0.0;
    if (A.ngp) {
        const BeamRow p = k > 0 ? row(k - 1) : BeamRow{0.0, 0.0, guard_at(A, j, B_JZ0), guard_at(A, j, B_JP1I)};
        djz = (r.jz - p.jz) * A.idxi;
        djt = (r.jt - p.jt) * A.idxi;
    } else if (K > 1) {
        const BeamRow a = k == 0 ? r : row(k - 1), b = k == K - 1 ? r : row(k + 1);
        const double f = (k == 0 || k == K - 1) ? 1.0 : 0.5;
        djz = f * (b.jz - a.jz) * A.idxi;
        djt = f * (b.jt - a.jt) * A.idxi;
    }
    r.rt += ds * r.drt;
    r.jz += ds * djz;
    r.jt += ds * djt;
    return r;
}

// the two neighbours of row i in the 3-point stencils gm f[lo] + g0 f[i] + gp f[hi]: the one-sided wall stencil
// takes row N - 2 in place of row N + 1; at the axis the stencil is zero (gm = g0 = gp = 0)
__device__ __forceinline__ int row_lo(int i) { return max(i - 1, 0); }
__device__ __forceinline__ int row_hi(int i, int N) { return i == N ? N - 2 : i + 1; }

// right-hand side of system e (psi, E_z, B_z) at row i (src/Simulation.cpp:798-799, :517-527)
__device__ __forceinline__ double rhs_l0(const Smem& S, const Src& s, int N, int e, int i) {
    if (e == 0) return -s.rhot[i];
    if (e == 1) return -s.drho[i];
    // the odd gradient (f_1 / r_1 on the axis) plus f / r (f_1 / r_1 on the axis)
    const double* const f = s.jpi1;
    const double g = S.gm[i] * f[row_lo(i)] + S.g0[i] * f[i] + S.gp[i] * f[row_hi(i, N)];
    const double f1 = f[max(i, 1)], ir = S.ir[i];
    return -((i == 0 ? f1 * ir : g) + f1 * ir);
}

// row i of (L1D - chi) (sys 0) or (L1F - chi) (sys 1) with its right-hand side; cm = c_{i-1} (any value at row 0,
// where a = 0); sv: S_i or S_r (src/FieldSolver.cpp:172-191, src/Simulation.cpp:535-591)
__device__ __forceinline__ void row_b(const Smem& S, const Src& s, int N, double fc, int sys, int i, double sv,
                                      double& a, double& b, double& cm, double& d) {
    a = S.l1a[i];
    b = S.l1b[i];
    cm = S.l1c[row_lo(i)];
    const bool wall = i == N, in = i > 0 && (sys || !wall);      // in: not a Dirichlet row
    const double chi = s.chi[i];
    if (sys == 0) {
        d = -sv;
    } else {
        const double* const f = s.jz;
        const double jn = f[i];
        d = (S.gm[i] * f[row_lo(i)] + S.g0[i] * jn + S.gp[i] * f[row_hi(i, N)]) + sv;
        if (wall) { a = S.lfa; b = S.lfb; d -= fc * jn; }
    }
    b = in ? b - chi : b;
    d = in ? d : 0.0;
}

// One L0 system by a group of kG2 warps (e: 0..2, the group's number), rows [row0, row0 + R) per thread. L0 is
// D^-1 times a Laplacian: with w_i = V_i / 2 pi and g_i = r_mid,i / h_i its rows say that the flux g_i (x_{i+1} - x_i)
// is the sum of w d up to node i. The Thomas pivots of that matrix are -g_i / w_i exactly, so the two
// substitutions are plain sums: z_i = z_{i-1} + w_i d_i and x_i = x_{i+1} - z_i / g_i. rhs(i): d_i for i < N. On return
// v holds x of the thread's rows, z0 the flux into them and xn the x just after them. vw and gw are 0 at row N.
template <int kR, class Rhs>
__device__ __forceinline__ void l0_group(double* tot, const double* vw, const double* gw, int N, int e, int wl, int R,
                                         int row0, Rhs rhs, double (&v)[kR], double& z0, double& xn) {
    // rows past the thread's or the grid's end stand at row N, where w = 1 / g = 0: no branch, so that the loads
    // of all rows are in flight together
    double g[kR], sum = 0.0;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const int i = u < R ? min(row0 + u, N) : N;
        v[u] = vw[i] * rhs(i);
        g[u] = gw[i];
    }
#pragma unroll
    for (int u = 0; u < kR; ++u) sum += v[u];
    double z = group_sum<true, kG2>(sum, wl, tot + 8 * e, 1 + e);
    z0 = z;
    sum = 0.0;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        z += v[u];
        v[u] = -(z * g[u]);
    }
#pragma unroll
    for (int u = kR - 1; u >= 0; --u) sum += v[u];
    double x = group_sum<false, kG2>(sum, wl, tot + 24 + 8 * e, 1 + e);
    xn = x;
#pragma unroll
    for (int u = kR - 1; u >= 0; --u) {
        x += v[u];
        v[u] = x;
    }
}

// psi, E_z, B_z and W+ (src/Simulation.cpp:797-807, :501-532, :477-498)
template <int kR>
__device__ __forceinline__ void l0_solve(const Smem& S, const Src& s, int M, int N) {
    const int warp = threadIdx.x >> 5, e = warp / kG2, wl = warp - e * kG2;
    if (e >= 3) return;
    const int R = group_rows(M, kG2), row0 = (wl * 32 + (threadIdx.x & 31)) * R;
    double v[kR], z0, xn;
    l0_group<kR>(S.tot, S.vw, S.gw, N, e, wl, R, row0, [&](int i) { return rhs_l0(S, s, N, e, i); }, v, z0, xn);
    double* const out = e == 0 ? S.psi : (e == 1 ? S.ez : S.bz);
#pragma unroll
    for (int u = 0; u < kR; ++u)
        if (u < R && row0 + u < M) out[row0 + u] = v[u];
    if (e != 0) return;
    // W+ = -psi' on the thread's rows; psi just before them from the flux that enters them
    const double xm = v[0] - z0 * S.gw[min(row_lo(row0), N)];
    double w[kR];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const int i = u < R ? min(row0 + u, N) : N;
        const double lo = u ? v[u - 1] : xm, hi = (u + 1 < kR && u + 1 < R) ? v[u + 1 < kR ? u + 1 : u] : xn;
        w[u] = -(S.gm[i] * lo + S.g0[i] * v[u] + S.gp[i] * hi);          // (row 0: -0)
        // the row before the wall also gives the wall's one-sided value from psi_N, psi_{N-1}, psi_{N-2}
        if (u < R && row0 + u == N - 1) S.wr1[N] = -(S.g0[N] * hi + S.gm[N] * v[u] + S.gp[N] * lo);
    }
#pragma unroll
    for (int u = 0; u < kR; ++u)
        if (u < R && row0 + u < N) S.wr1[row0 + u] = w[u];
}

// One chi-shifted system by a group of kG4 warps (sy: 0 or 1), rows [row0, row0 + R) per thread: 1/u_i = p_{i-1} /
// p_i, where (p_i, p_{i-1}) is the first column of the product of T_i = [[b_i, -a_i c_{i-1}], [1, 0]] up to row i.
// row(i, a, b, cm, d): row i with cm = c_{i-1} and its right-hand side; c(i): c_i. On return x holds the solution
// on the thread's rows.
template <int kR, class Row, class C>
__device__ __forceinline__ void shifted_group(double* tot, int M, int sy, int wl, int R, int row0, Row row, C c,
                                              double (&x)[kR]) {
    double* const tp = tot + 64 + 32 * sy;
    double* const tf = tot + 128 + 16 * sy;
    double* const tb = tot + 160 + 16 * sy;
    double ra[kR], rb[kR], rc[kR];
    double m[4] = {1.0, 0.0, 0.0, 1.0};
    // rows past the thread's or the grid's end read row M - 1 and then become x = 0 rows (a = d = 0, b = 1), so that
    // the loads of all rows are in flight together
    double cc[kR];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const int i = u < R ? min(row0 + u, M - 1) : M - 1;
        row(i, ra[u], rb[u], rc[u], x[u]);
        cc[u] = c(i);
    }
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const bool on = u < R && row0 + u < M;
        ra[u] = on ? ra[u] : 0.0;
        rb[u] = on ? rb[u] : 1.0;
        x[u] = on ? x[u] : 0.0;
        const double t01 = -ra[u] * rc[u];
        const double n00 = rb[u] * m[0] + t01 * m[2], n01 = rb[u] * m[1] + t01 * m[3];
        m[2] = on ? m[0] : m[2]; m[3] = on ? m[1] : m[3];
        m[0] = on ? n00 : m[0]; m[1] = on ? n01 : m[1];
        if ((u & 3) == 3) renorm(m[0], m[1], m[2], m[3]);
    }
    renorm(m[0], m[1], m[2], m[3]);
    double p, q;
    group_pivots<kG4>(m, p, q, wl, tp, 4 + sy);
    // 1/u of the rows (into rc), the composite of the forward substitution
    double fA = 1.0, fB = 0.0;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const double pn = rb[u] * p - ra[u] * rc[u] * q;
        q = p;
        p = pn;
        pivot_scale(p, q);
        rc[u] = pivot_quot(q, p);
    }
    // (rows past the end carry y and x along: slope 1, nothing added)
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const bool on = u < R && row0 + u < M;
        ra[u] = on ? -rc[u] * ra[u] : 1.0;                   // forward: y_i = ra y_{i-1} + x
        x[u] = rc[u] * x[u];
        rc[u] = on ? -(cc[u] * rc[u]) : 1.0;                 // backward: x_i = rc x_{i+1} + y_i
        fB = fma(ra[u], fB, x[u]);
        fA *= ra[u];
    }
    double y = group_affine<true, kG4>(fA, fB, wl, tf, 4 + sy);
    double bA = 1.0, bB = 0.0;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
        const bool on = u < R && row0 + u < M;
        y = fma(ra[u], y, x[u]);
        x[u] = on ? y : 0.0;
    }
#pragma unroll
    for (int u = kR - 1; u >= 0; --u) {
        bB = fma(rc[u], bB, x[u]);
        bA *= rc[u];
    }
    double xx = group_affine<false, kG4>(bA, bB, wl, tb, 4 + sy);
#pragma unroll
    for (int u = kR - 1; u >= 0; --u) {
        xx = fma(rc[u], xx, x[u]);
        x[u] = xx;
    }
}

// B_r and B_theta (src/Simulation.cpp:535-591, m = 0: one pass): (L1D - chi) B_r0 = -S_i (rows 0, N Dirichlet)
// and (L1F - chi) B_theta0 = J_z' + S_r with flux wall J_z(R). kFinish: S_i and S_r are turned from the exact
// accumulators here, each by its only reader
template <int kR, bool kFinish>
__device__ __forceinline__ void bplus_solve(const Smem& S, const Src& s, int M, int N, double fc, int bits) {
    const int warp = threadIdx.x >> 5, sy = warp / kG4, wl = warp - sy * kG4;
    const int R = group_rows(M, kG4), row0 = (wl * 32 + (threadIdx.x & 31)) * R;
    double* const sa = sy ? s.S1r : s.S1i;
    const int es = kFinish ? S.fx[sy ? 7 : 8] : 0;
    const double qs = kFinish ? fx_quantum(es, bits) : 0.0;
    double x[kR];
    shifted_group<kR>(
        S.tot, M, sy, wl, R, row0,
        [&](int i, double& a, double& b, double& cm, double& d) {
            row_b(S, s, N, fc, sy, i, kFinish ? fx_value(sa + i, es, qs) : sa[i], a, b, cm, d);
        },
        [&](int i) { return S.l1c[i]; }, x);
    double* const out = sy ? S.bpi : S.bpr;
#pragma unroll
    for (int u = 0; u < kR; ++u)
        if (u < R && row0 + u < M) out[row0 + u] = x[u];
}

// The block-wide solves' own right-hand sides and rows (branches at the ends instead of clamped rows).
// right-hand sides of the psi, E_z, B_z systems at row i (src/Simulation.cpp:798-799, :517-527)
__device__ __forceinline__ void block_rhs(const Smem& S, const Src& s, int N, int i, double& d0, double& d1,
                                       double& d2) {
    d0 = d1 = d2 = 0.0;
    if (i < N) {
        d0 = -1.0 * s.rhot[i];
        d1 = -1.0 * s.drho[i];
        const double t1 = grad_at(S, N, s.jpi1, i, true);
        const double t2 = (i == 0 ? s.jpi1[1] : s.jpi1[i]) * S.ir[i];
        d2 = 1.0 * (-(t1 + t2));
    }
}

// row i of (L1D - chi) (sys 0) and (L1F - chi) (sys 1) with its right-hand side
// (src/FieldSolver.cpp:172-191, src/Simulation.cpp:535-591)
__device__ __forceinline__ void block_row(const Smem& S, const Src& s, int N, double fc, int sys, int i, double& a,
                                      double& b, double& cm, double& d) {
    if (sys == 0) {
        a = S.l1a[i]; b = S.l1b[i]; cm = i > 0 ? S.l1c[i - 1] : 0.0;
        if (i >= 1 && i < N) { b = b - s.chi[i]; d = 1.0 * (-s.S1i[i]); } else { d = 0.0; }
    } else {
        a = i == N ? S.lfa : S.l1a[i]; b = i == N ? S.lfb : S.l1b[i]; cm = i > 0 ? S.l1c[i - 1] : 0.0;
        if (i >= 1) {
            b = b - s.chi[i];
            d = 1.0 * (grad_at(S, N, s.jz, i, false) + s.S1r[i]);
            if (i == N) d -= fc * s.jz[N];
        } else {
            d = 0.0;
        }
    }
}

// The solves of grids with more than kThreads nodes: block-wide scans, thread t with the rows [t Rw, t Rw + Rw).
// (10,700 and 13,600 cycles per slice at 1001 nodes; groups of warps, with 7 rows per L0 thread and 5 per B+ thread
// in registers, took 17,800 and 18,700.)
template <int kMaxR>
__device__ __forceinline__ void l0_block(const Smem& S, const Src& s, int M, int N, int Rw) {
    const int row0 = threadIdx.x * Rw;
    // forward: y_i = (-a_i/u_i) y_{i-1} + d_i/u_i
    double cA = 1.0, cB[3] = {0.0, 0.0, 0.0};
    double dv[kMaxR][3];
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
        dv[u][0] = dv[u][1] = dv[u][2] = 0.0;
        if (u >= Rw || i >= M) continue;
        block_rhs(S, s, N, i, dv[u][0], dv[u][1], dv[u][2]);
        const double rr = S.l0r[i], af = S.l0f[i];
#pragma unroll
        for (int e = 0; e < 3; ++e) cB[e] = fma(af, cB[e], rr * dv[u][e]);
        cA *= af;
    }
    double yb[3];
    scan_fwd<3>(cA, cB, yb, S.tot);
    const double ypsi_prev = yb[0];                        // y of psi just before this thread's rows
    double y[kMaxR][3];
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
        y[u][0] = y[u][1] = y[u][2] = 0.0;
        if (u >= Rw || i >= M) continue;
        const double rr = S.l0r[i], af = S.l0f[i];
#pragma unroll
        for (int e = 0; e < 3; ++e) { yb[e] = fma(af, yb[e], rr * dv[u][e]); y[u][e] = yb[e]; }
    }
    // backward: x_i = (-c_i/u_i) x_{i+1} + y_i
    double bA = 1.0, bB[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int u = kMaxR - 1; u >= 0; --u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
        const double ab = S.l0b[i];
#pragma unroll
        for (int e = 0; e < 3; ++e) bB[e] = fma(ab, bB[e], y[u][e]);
        bA *= ab;
    }
    double xa[3];
    scan_bwd<3>(bA, bB, xa, S.tot + 8 * kW);
    // psi on the window [row0 - 1, row0 + Rw]: the rows of this thread, x after them (the
    // backward carry) and x before them, x_{row0-1} = y_{row0-1} - (c/u)_{row0-1} x_{row0}
    // with y_{row0-1} the forward carry -- so W+ = -psi' needs no further exchange
    double pw[kMaxR + 2];
    pw[kMaxR + 1] = 0.0;
    {
        double xr = xa[0];
#pragma unroll
        for (int u = kMaxR; u >= 1; --u) pw[u] = 0.0;
        const int last = (row0 + Rw <= M ? Rw : M - row0);
        if (last >= 0) pw[last + 1 > kMaxR + 1 ? kMaxR + 1 : last + 1] = xr;
    }
#pragma unroll
    for (int u = kMaxR - 1; u >= 0; --u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
        const double ab = S.l0b[i];
#pragma unroll
        for (int e = 0; e < 3; ++e) xa[e] = fma(ab, xa[e], y[u][e]);
        S.psi[i] = xa[0];
        S.ez[i] = xa[1];
        S.bz[i] = xa[2];
        pw[u + 1] = xa[0];
    }
    pw[0] = (row0 >= 1 && row0 < M) ? fma(S.l0b[row0 - 1], pw[1], ypsi_prev) : 0.0;
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
        if (i == 0) {
            S.wr1[0] = -0.0;
        } else if (i < N) {
            S.wr1[i] = -(S.gm[i] * pw[u] + S.g0[i] * pw[u + 1] + S.gp[i] * pw[u + 2]);
        }
        if (i == N - 1) {                                  // the one-sided wall stencil needs psi_{N-2..N}
            S.wr1[N] = -(S.g0[N] * pw[u + 2] + S.gm[N] * pw[u + 1] + S.gp[N] * pw[u]);
        }
    }
}

template <int kMaxR>
__device__ __forceinline__ void bplus_block(const Smem& S, const Src& s, int M, int N, double fc, int Rw) {
    const int row0 = threadIdx.x * Rw;
    // pivots: product of T_i = [[b_i, -a_i c_{i-1}], [1, 0]] over the thread's rows
    double m[2][4];
#pragma unroll
    for (int sy = 0; sy < 2; ++sy) { m[sy][0] = 1.0; m[sy][1] = 0.0; m[sy][2] = 0.0; m[sy][3] = 1.0; }
    double ra[kMaxR][2], rb[kMaxR][2], rc[kMaxR][2], rd[kMaxR][2];
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
#pragma unroll
        for (int sy = 0; sy < 2; ++sy) {
            ra[u][sy] = 0.0; rb[u][sy] = 1.0; rc[u][sy] = 0.0; rd[u][sy] = 0.0;
            if (u >= Rw || i >= M) continue;
            block_row(S, s, N, fc, sy, i, ra[u][sy], rb[u][sy], rc[u][sy], rd[u][sy]);
            const double t01 = -ra[u][sy] * rc[u][sy];
            const double n00 = rb[u][sy] * m[sy][0] + t01 * m[sy][2];
            const double n01 = rb[u][sy] * m[sy][1] + t01 * m[sy][3];
            m[sy][2] = m[sy][0]; m[sy][3] = m[sy][1];
            m[sy][0] = n00; m[sy][1] = n01;
            renorm(m[sy][0], m[sy][1], m[sy][2], m[sy][3]);
        }
    }
    double pp[2], qq[2];
    scan_pivots<2>(m, pp, qq, S.tot);
    // this thread's pivots (rc holds c_{i-1}; rinv = 1/u_i = p_{i-1}/p_i), forward composites
    double rinv[kMaxR][2];
    double fA[2] = {1.0, 1.0}, fB[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
#pragma unroll
        for (int sy = 0; sy < 2; ++sy) {
            rinv[u][sy] = 0.0;
            if (u >= Rw || i >= M) continue;
            const double pn = rb[u][sy] * pp[sy] - ra[u][sy] * rc[u][sy] * qq[sy];
            qq[sy] = pp[sy];
            pp[sy] = pn;
            const double rr = qq[sy] / pp[sy];
            const double sc = fabs(pp[sy]);
            if (sc > 1e100 || sc < 1e-100) { pp[sy] /= sc; qq[sy] /= sc; }
            rinv[u][sy] = rr;
            const double af = -rr * ra[u][sy];
            fB[sy] = fma(af, fB[sy], rr * rd[u][sy]);
            fA[sy] *= af;
        }
    }
    // forward substitution of both systems
    double yy[2];
    scan_fwd_n<2>(fA, fB, yy, S.tot + 8 * kW);
    double y[kMaxR][2];
#pragma unroll
    for (int u = 0; u < kMaxR; ++u) {
        const int i = row0 + u;
#pragma unroll
        for (int sy = 0; sy < 2; ++sy) {
            y[u][sy] = 0.0;
            if (u >= Rw || i >= M) continue;
            yy[sy] = fma(-rinv[u][sy] * ra[u][sy], yy[sy], rinv[u][sy] * rd[u][sy]);
            y[u][sy] = yy[sy];
        }
    }
    // backward substitution: x_i = -(c_i / u_i) x_{i+1} + y_i
    double bA[2] = {1.0, 1.0}, bB[2] = {0.0, 0.0};
#pragma unroll
    for (int u = kMaxR - 1; u >= 0; --u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
#pragma unroll
        for (int sy = 0; sy < 2; ++sy) {
            const double c = S.l1c[i];
            const double ab = -(c * rinv[u][sy]);
            bB[sy] = fma(ab, bB[sy], y[u][sy]);
            bA[sy] *= ab;
        }
    }
    double xx[2];
    scan_bwd_n<2>(bA, bB, xx, S.tot);
#pragma unroll
    for (int u = kMaxR - 1; u >= 0; --u) {
        const int i = row0 + u;
        if (u >= Rw || i >= M) continue;
#pragma unroll
        for (int sy = 0; sy < 2; ++sy) {
            const double c = S.l1c[i];
            xx[sy] = fma(-(c * rinv[u][sy]), xx[sy], y[u][sy]);
        }
        S.bpr[i] = xx[0];
        S.bpi[i] = xx[1];
    }
}

}  // namespace sweep_detail

using namespace sweep_detail;

// One sweep by the calling CTA (all kThreads threads). The gate G orders it against other CTAs when
// several time steps run concurrently (NoGate: a stand-alone sweep). Returns false if a gate wait
// gave up (the CTA then stops at the next slice boundary). EXT: the kernel also handles the smoothing
// filter (A.filter), static beam sources (A.bstat) and adaptive sub-slicing (A.max_cells); without it they are
// ignored, and the kernel of plain decks carries none of their code (sweep_ext).
template <int ORD, bool REG, int kMaxR, class Gate, bool EXT = false>
__device__ __forceinline__ bool sweep_body(const SweepArgs& A, double* smem_raw, Gate& gate) {
    const int M = A.M, N = A.N, K = A.K, Rw = kMaxR == 1 ? 1 : A.rows_per_thread;   // rows per thread
    const int tid = threadIdx.x;
    // with one row and one particle per thread (M <= kSweepThreads) the constants always fit shared memory
    constexpr bool kCS = REG && kMaxR == 1;
    // The particles' force history (5 ORD doubles each) is read and written once per slice, by the push: in
    // registers it takes 30 of a thread's 128 (ORD 3) through all the solves and what they displace goes to local
    // memory, of which 512 threads have more than the L1 left beside 150 KB of shared memory holds. So it lives in
    // shared memory (a ring of ORD slots), with single-buffered sources to make room for it and for L1: 14.7 -> 12.5 us
    // per slice at 257 nodes, 17.9 -> 14.9 at 512.
    constexpr int kHist = hist_doubles(ORD, REG, kMaxR, EXT);
    constexpr bool kHS = kHist > 0;
    // beam rows loaded ahead of their use: one per thread (10 doubles; with more they would displace the rest, and the
    // prefetched rows come from L2 at their use)
    constexpr int kPre = 1;
    const bool dbuf = !kHS && A.dbuf;
    const int ST = kHS ? kThreads : M;                          // distance between the shared arrays
    int hs = 0;                                                 // slot of the particle's newest force (a removed
                                                                // particle's history stands still, and its slot)
    const Smem S = carve<kCS, kHist>(smem_raw, A);
    const int np = A.np, npad = A.npad;
    const double R = A.R;
    const int row0 = tid * Rw;                                  // this thread's rows [row0, row0 + Rw)
    unsigned long long* tim = A.timing;
    if (tim && tid == 0) S.tmark[0] = clock64();
#define PHASE_MARK(ph)                                                        \
    do {                                                                      \
        if (tim && tid == 0) {                                                \
            const long long tn = clock64();                                   \
            atomicAdd(tim + (ph), (unsigned long long)(tn - S.tmark[0]));     \
            S.tmark[0] = tn;                                                  \
        }                                                                     \
    } while (0)
// parts of the solve phase, by thread 0 (a warp of the psi system): [5] the solves, [6] the next slice's start values
#define SUB_MARK(slot)                                                        \
    do {                                                                      \
        if (tim && tid == 0) {                                                \
            const long long tn = clock64();                                   \
            atomicAdd(tim + (slot), (unsigned long long)(tn - S.tmark[1]));   \
            S.tmark[1] = tn;                                                  \
        }                                                                     \
    } while (0)

    // ---------------- prologue: grid, operators, fresh plasma, background (src/Simulation.cpp:653-708)
    for (int j = tid; j < M; j += kThreads) {
        S.r[j] = A.r[j];
        S.iv[j] = A.inv_V[j];
        S.ih[j] = (j < N) ? A.inv_h[j] : 0.0;
        S.bgt[j] = 0.0;
        S.bgr[j] = 0.0;
        S.bpr[j] = 0.0;
        S.bpi[j] = 0.0;
        src_of(S, ST, 0).ne[j] = 0.0;
    }
    if (kCS || A.const_smem)
        for (int t = tid; t < consts0_arrays(M) * M; t += kThreads) {
            const int c = t / M;
            const_cast<double*>(S.gm)[c * ST + t - c * M] = A.consts0[t];
        }
    if (tid == 0) *S.lost = 0;
    if (tid < 14) S.fx[tid] = 0;
    if (tid < 9) S.fxp[tid] = 0;
    const int bits_p = fx_bits(np), bits_bg = fx_bits(A.nbg);
    PState<ORD> P;
    int J = 0;                                             // cell of the thread's particle
    PKeep kp{0.0, 0.0, 1.0, 0.0, {1.0, 1.0}};              // and its polar position and kinematics
    if (REG) {
        if (tid < np) {
            if (A.pin) {                                  // a later slab: the plasma handed on, with its history
                pload(P, A.pin, npad, tid);
            } else {
                P.x = A.p_init[tid]; P.y = A.p_init[npad + tid]; P.px = A.p_init[2 * npad + tid];
                P.py = A.p_init[3 * npad + tid]; P.dl = A.p_init[4 * npad + tid]; P.w = A.p_init[5 * npad + tid];
#pragma unroll
                for (int m = 0; m < ORD; ++m)
#pragma unroll
                    for (int v = 0; v < 5; ++v) P.h[m][v] = 0.0;
            }
            species_params(A, tid, P.q, P.qm);
            if (kHS) hist_put<ORD>(P, S, hs, true);
        } else {
            P.x = P.y = P.px = P.py = 0.0;
            P.dl = 1.0;
            P.w = 0.0;
            P.q = P.qm = -1.0;
#pragma unroll
            for (int m = 0; m < ORD; ++m)
#pragma unroll
                for (int v = 0; v < 5; ++v) P.h[m][v] = 0.0;
        }
    } else {
        for (int p = tid; p < np; p += kThreads) {
            if (A.pin) {
                for (int v = 0; v < 6 + 5 * ORD; ++v) gate.ps(A)[(size_t)v * npad + p] = A.pin[(size_t)v * npad + p];
            } else {
#pragma unroll
                for (int v = 0; v < 6; ++v) gate.ps(A)[(size_t)v * npad + p] = A.p_init[(size_t)v * npad + p];
                for (int v = 0; v < 5 * ORD; ++v) gate.ps(A)[(size_t)(6 + v) * npad + p] = 0.0;
            }
            if (A.pcache) {
                const double* src = A.pin ? A.pin : A.p_init;
#pragma unroll
                for (int v = 0; v < 6; ++v) S.pc[(size_t)v * A.pcache + p] = src[(size_t)v * npad + p];
            }
        }
    }
    __syncthreads();
    // immobile species deposit into the background; mobile ones are subtracted (neutralisation,
    // src/Simulation.cpp:672-684); src[0].ne is the scratch of the mobile deposit. Both exact: a pass
    // for the exponent maxima, a barrier, a pass of quantised adds, a barrier, then the values.
    double* const ne0 = src_of(S, ST, 0).ne;
    for (int pass = 0; pass < 2; ++pass) {
        int ebg = 0, ene = 0;
        for (int p = tid; p < A.nbg; p += kThreads) {
            const double x = A.bg_p[p], y = A.bg_p[A.nbg + p], wq = A.bg_p[2 * A.nbg + p];
            if (wq == 0.0) continue;
            const PGeo g = geometry(S.r, S.ih, N, R, x, y);
            const double a0 = wq * g.W0 * S.iv[g.j], a1 = wq * g.W1 * S.iv[g.j + 1];
            if (pass == 0) {
                ebg = max(ebg, max(fx_bexp(a0), fx_bexp(a1)));
            } else {
                const double sc = fx_scale(S.fx[9], bits_bg), v[4] = {a0, a0, a1, a1}, s4[4] = {sc, sc, sc, sc};
                double* const adr[4] = {S.bgt + g.j, S.bgr + g.j, S.bgt + g.j + 1, S.bgr + g.j + 1};
                fx_add<4>(adr, v, s4);
            }
        }
        if (A.neutralize)
            for (int p = tid; p < np; p += kThreads) {
                const double w = A.p_init[5 * (size_t)npad + p];
                if (w == 0.0) continue;
                double q, qm;
                species_params(A, p, q, qm);
                const PGeo g = geometry(S.r, S.ih, N, R, A.p_init[p], A.p_init[npad + p]);
                const double a0 = w * q * g.W0 * S.iv[g.j], a1 = w * q * g.W1 * S.iv[g.j + 1];
                if (pass == 0) {
                    ene = max(ene, max(fx_bexp(a0), fx_bexp(a1)));
                } else {
                    const double sc = fx_scale(S.fx[10], bits_p), v[2] = {a0, a1}, s2[2] = {sc, sc};
                    double* const adr[2] = {ne0 + g.j, ne0 + g.j + 1};
                    fx_add<2>(adr, v, s2);
                }
            }
        if (pass == 0) {
            const int e2[2] = {ebg, ene};
            fx_max<2>(e2, S.fx + 9);
        }
        __syncthreads();
    }
    for (int j = tid; j < M; j += kThreads) {
        const double qb = fx_quantum(S.fx[9], bits_bg), qn = fx_quantum(S.fx[10], bits_p);
        S.bgt[j] = fx_value(S.bgt + j, S.fx[9], qb);
        S.bgr[j] = fx_value(S.bgr + j, S.fx[9], qb);
        ne0[j] = fx_value(ne0 + j, S.fx[10], qn);
    }
    if (Gate::kActive && tid < 32) {                     // warp 0 checks the beam-source rows
        const bool ok = gate.before_rows(K - 1 < 2 ? K - 1 : 2);
        if (tid == 0) *S.flag = ok ? 1 : 0;
    }
    __syncthreads();
    if (Gate::kActive && !*S.flag) return false;
    if (EXT && A.filter) {              // the background is smoothed like the plasma (src/Simulation.cpp:685-690)
        if (A.neutralize)
            for (int j = tid; j < M; j += kThreads) {
                S.bgt[j] -= ne0[j];
                S.bgr[j] -= ne0[j];
            }
        __syncthreads();
        FilterSet<2> fb;
        fb.f[0] = S.bgt; fb.f[1] = S.bgr; fb.op[0] = fb.op[1] = 0;
        filter_rows<2, kMaxR>(fb, A.fconsts, M, Rw, S.ftot);
        __syncthreads();
    } else if (A.neutralize) {
        for (int j = tid; j < M; j += kThreads) {
            S.bgt[j] -= ne0[j];
            S.bgr[j] -= ne0[j];
        }
    }
    // slice 0's arrays accumulate its plasma deposit from zero; its start values (background + beam,
    // init_base) are added when the deposit is finished
    {
        const Src s0 = src_of(S, ST, 0);
        for (int j = tid; j < M; j += kThreads) {
#pragma unroll
            for (int c = 0; c < 7; ++c) dep_arr(s0, c)[j] = 0.0;
            s0.S1r[j] = 0.0;
            s0.S1i[j] = 0.0;
        }
    }
    __syncthreads();
    // deposit of slice 0
    const int lane = tid & 31;
    {
        const Src s0 = src_of(S, ST, 0);
        if (REG) {
            const bool act = tid < np && P.w != 0.0;
            double v[12];
            if (act) {
                polar(P.x, P.y, kp.rp, kp.ir, kp.c, kp.s);
                kp.k = kin_of(P.px, P.py, P.dl);
                J = locate(S.r, N, R, kp.rp);
                deposit_values(P, keep_geo(S, kp, J), kp.k, S, v);
            }
            const bool tail = deposit_runs<true>(act, J, P.q < 0.0, v, S.fx);
            __syncthreads();
            deposit_add(tail, J, P.q < 0.0, v, s0, S.fx, bits_p);
        } else {
            for (int pass = 0; pass < 2; ++pass) {
                if (pass == 1) __syncthreads();
                for (int base = tid - lane; base < np; base += kThreads) {
                    const int p = base + lane;
                    PState<ORD> Q;
                    bool act = false;
                    int j = 0;
                    double v[12];
                    if (p < np) {
                        pbase(Q, S, A, gate.ps(A), npad, p);
                        species_params(A, p, Q.q, Q.qm);
                        act = Q.w != 0.0;
                        if (act) {
                            // the first pass searches the cell and keeps it for the later passes
                            const PGeo g = pass == 0 ? geometry(S.r, S.ih, N, R, Q.x, Q.y)
                                                     : pgeo(S, A, N, R, p, Q.x, Q.y);
                            if (pass == 0 && A.pcache) S.pj[p] = g.j;
                            j = g.j;
                            deposit_values(Q, g, KinNone{}, S, v);
                        }
                    }
                    const bool neg = act && Q.q < 0.0;
                    if (pass == 0) {
                        deposit_runs<true>(act, j, neg, v, S.fx);
                    } else {
                        const bool tail = deposit_runs<false>(act, j, neg, v, S.fx);
                        deposit_add(tail, j, neg, v, s0, S.fx, bits_p);
                    }
                }
            }
        }
        __syncthreads();
        if (tid == 0)
            for (int c = 0; c < 7; ++c) S.fx[13] += (S.fx[c] == 2047) + (c < 2 && S.fx[9 + c] == 2047);
        for (int j = tid; j < M; j += kThreads) {
            double b0[7];
            init_base<EXT>(S, j, beam_row<Gate::kActive, EXT>(A, gate.bsrc(A), 0, j), M, b0);
            deposit_finish(s0, s0, j, b0, S.fx, bits_p);
        }
    }
    __syncthreads();
    PHASE_MARK(0);

    const double fc = A.flux_coef;
    // Adaptive sub-slicing only: the xi positions of the last ORD pushes (tn[0] the newest) give the
    // Adams-Bashforth coefficients of the next push: the classical ones for uniform steps, the variable-step ones
    // after a change (src/PlasmaSpecies.cpp:561-580). A slab whose plasma was pushed before continues uniform steps
    // of dxi. The state (tn, then the current xi and the last step) is in shared memory, so that plain sweeps hold no
    // registers for it: every thread reads one copy, thread 0 writes the other (barriers lie between two pushes).
    int abp = 0;
    const bool vsteps = EXT && A.max_cells > 0.0;
    if (vsteps && tid == 0) {
        for (int m = 0; m < ORD; ++m) S.absl[m] = -(m + 1) * A.dxi;
        S.absl[5] = 0.0;
        S.absl[6] = A.pin_pushed ? A.dxi : 0.0;
    }
    auto coeffs = [&](double h, bool first, double (&abc)[5]) {
        bool uniform = true;
        double tn[ORD];
        if (vsteps) {
            const double* const o = S.absl + 8 * abp;
            const double xcur = o[5];
#pragma unroll
            for (int m = 0; m < ORD; ++m) tn[m] = first ? xcur - m * h : (m == 0 ? xcur : o[m > 0 ? m - 1 : 0]);
#pragma unroll
            for (int m = 1; m < ORD; ++m) uniform = uniform && fabs((tn[m - 1] - tn[m]) - h) <= 1e-9 * h;
            abp ^= 1;
            if (tid == 0) {
                double* const w = S.absl + 8 * abp;
#pragma unroll
                for (int m = 0; m < ORD; ++m) w[m] = tn[m];
                w[5] = xcur + h;
                w[6] = h;
            }
        }
        if (uniform) {
#pragma unroll
            for (int m = 0; m < 5; ++m) abc[m] = A.ab[m];
        } else {
            ab_variable<ORD>(tn, h, abc);
        }
    };
    if (vsteps) __syncthreads();
    for (int k = 0; k < K; ++k) {
    // the passes of slice k: its own, then its sub-slices (adaptive sub-slicing, src/Simulation.cpp:755-781):
    // each pushes by dxi / nsub; a sub-slice re-deposits the plasma and re-solves the fields with the beam
    // sources extrapolated from slice k; only the slice itself is stored
    int nsub = 1;
    for (int ss = 0; ss < nsub; ++ss) {
        // the plasma state at the start of slice k (every slice, or the checkpoint slices)
        const int tevery = A.traj_every > 1 ? A.traj_every : 1;
        if (double* const trj = ss == 0 && k % tevery == 0 ? gate.traj(A) : nullptr) {
            double* T = trj + (size_t)(k / tevery) * (6 + 5 * (size_t)ORD) * npad;
            if (REG) {
                if (tid < np) {
                    if (kHS) hist_get<ORD>(P, S, hs);
                    T[tid] = P.x; T[npad + tid] = P.y; T[2 * (size_t)npad + tid] = P.px;
                    T[3 * (size_t)npad + tid] = P.py; T[4 * (size_t)npad + tid] = P.dl;
                    T[5 * (size_t)npad + tid] = P.w;
#pragma unroll
                    for (int m = 0; m < ORD; ++m)
#pragma unroll
                        for (int v = 0; v < 5; ++v) T[(6 + (size_t)m * 5 + v) * npad + tid] = P.h[m][v];
                }
            } else {
                for (int p = tid; p < np; p += kThreads)
                    for (int v = 0; v < 6 + 5 * ORD; ++v) T[(size_t)v * npad + p] = gate.ps(A)[(size_t)v * npad + p];
            }
        }
        const Src s = src_of(S, ST, dbuf ? (k & 1) : 0);
        const Src sn = src_of(S, ST, dbuf ? ((k + 1) & 1) : 0);
        if constexpr (EXT)
            if (A.filter) filter_sources<kMaxR>(s, S, A, Rw);
        if (tim && tid == 0) S.tmark[1] = clock64();
        // beam rows of slice k+1 for this thread's nodes: loaded here without a use, so that the latency
        // (L2 or DRAM) overlaps the solves
        BeamRaw pre[kPre];
        if (kPre == kMaxR && dbuf && k + 1 < K && ss == 0)
#pragma unroll
            for (int u = 0; u < kPre; ++u)
                raw_load<Gate::kActive>(A, gate.bsrc(A), k + 1, min(tid + u * kThreads, N), pre[u]);

        // the warp without a system brings the beam row after next towards L2 (a stand-alone sweep streams them
        // from DRAM; in a pipelined run they are not final yet, and in L2 anyway)
        if (!Gate::kActive && tid >= 3 * kG2 * 32 && ss == 0 && k + 3 < K) {
            const double* const nx = gate.bsrc(A) + (size_t)(k + 3) * M * A.bcs;
            for (int o = lane * 16; o < M * A.bcs; o += 32 * 16)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + o));
        }
        // ---------------- P2: psi, E_z, B_z with L0, W+
        if constexpr (kMaxR == 1) l0_solve<5>(S, s, M, N);
        else l0_block<kMaxR>(S, s, M, N, Rw);
        SUB_MARK(5);
        if (dbuf && k + 1 < K && ss == 0)
#pragma unroll
            for (int u = 0; u < kMaxR; ++u) {
                const int j = tid + u * kThreads;
                if (j >= M) continue;
                init_sources<EXT>(sn, S, j,
                                  kPre == kMaxR ? raw_row<Gate::kActive, EXT>(A, gate.bsrc(A), k + 1, j, pre[u < kPre ? u : 0])
                                                : beam_row<Gate::kActive, EXT>(A, gate.bsrc(A), k + 1, j), M);
            }
        SUB_MARK(6);
        __syncthreads();
        PHASE_MARK(1);

        // ---------------- P3: S+ (src/PlasmaSpecies.cpp:508-559), exact
        if (tid < 7) {                        // the plasma deposit's maxima (read last before P2's barrier)
            S.fxp[tid] = S.fx[tid];
            S.fx[tid] = 0;
        }
        if (tid == 7) *S.cmax = 0ull;         // the cells-crossed maximum (read last at the last P5)
        if (REG) {
            const bool act = tid < np && P.w != 0.0;
            double v[4];
            if (act) species_params(A, tid, P.q, P.qm);      // (from the arguments: no register between the phases)
            if (act) depositS_values(P, keep_geo(S, kp, J), kp.k, S, N, v);
            const bool tail = depositS_runs<true>(act, J, v, S.fx + 7);
            __syncthreads();
            depositS_add(tail, J, v, s, S.fx + 7, bits_p);
            __syncthreads();
        } else {
            for (int pass = 0; pass < 2; ++pass) {
                for (int base = tid - lane; base < np; base += kThreads) {
                    const int p = base + lane;
                    bool act = false;
                    int j = 0;
                    double v[4];
                    if (p < np) {
                        PState<ORD> Q;
                        pbase(Q, S, A, gate.ps(A), npad, p);
                        species_params(A, p, Q.q, Q.qm);
                        act = Q.w != 0.0;
                        if (act) {
                            const PGeo g = pgeo(S, A, N, R, p, Q.x, Q.y);
                            j = g.j;
                            depositS_values(Q, g, KinNone{}, S, N, v);
                        }
                    }
                    const bool tail = pass == 0 ? depositS_runs<true>(act, j, v, S.fx + 7)
                                                : depositS_runs<false>(act, j, v, S.fx + 7);
                    depositS_add(tail, j, v, s, pass == 0 ? S.fxp + 7 : S.fx + 7, bits_p);
                }
                __syncthreads();
                if (pass == 1 || !fx_moved<2>(S.fx + 7, S.fxp + 7)) break;
                for (int j = tid; j < M; j += kThreads) s.S1r[j] = s.S1i[j] = 0.0;
                __syncthreads();
            }
        }
        PHASE_MARK(2);
        if (tid == 0) S.fx[13] += (S.fx[7] == 2047) + (S.fx[8] == 2047);

        // ---------------- P4: B+
        if (kMaxR > 1 || (EXT && A.filter)) {
#pragma unroll
            for (int u = 0; u < kMaxR; ++u)
                if (u < Rw && row0 + u < M) depositS_finish(s, row0 + u, S.fx + 7, bits_p);
            if (EXT && A.filter) {          // S+ smoothed with F1 (src/Simulation.cpp:810-812): a thread's own rows
                FilterSet<2> fsS;
                fsS.f[0] = s.S1r; fsS.f[1] = s.S1i; fsS.op[0] = fsS.op[1] = 1;
                filter_rows<2, kMaxR>(fsS, A.fconsts, M, Rw, S.ftot);
                if (kMaxR == 1) __syncthreads();
            }
        }
        if constexpr (kMaxR == 1) {
            if (EXT && A.filter) bplus_solve<3, false>(S, s, M, N, fc, bits_p);
            else bplus_solve<3, true>(S, s, M, N, fc, bits_p);
        } else {
            bplus_block<kMaxR>(S, s, M, N, fc, Rw);
        }
        __syncthreads();
        PHASE_MARK(3);

        // ---------------- P5: store slice k; push k -> k+1 (or to the next sub-slice) and deposit
        if (tid >= 7 && tid < 9) {                // the S deposit's maxima (read last before P4's barrier)
            S.fxp[tid] = S.fx[tid];
            S.fx[tid] = 0;
        }
        // adaptive sub-slicing, decided in the slice's own pass from the particles as they stand
        // (src/Simulation.cpp:837-847): nsub = ceil(max cells crossed / max_cells_per_step), at least
        // ceil(dxi / (2 h_last)) (the step at most doubles), at most substep_max
        if (EXT && ss == 0 && A.max_cells > 0.0 && k + 1 < K) {
            double c = 0.0;
            if (REG) {
                if (tid < np && P.w != 0.0) c = cells_crossed(S, N, R, P.x, P.y, P.px, P.py, P.dl, A.dxi);
            } else {
                for (int p = tid; p < np; p += kThreads) {
                    const double* ps = gate.ps(A);
                    if (ps[5 * (size_t)npad + p] == 0.0) continue;
                    c = fmax(c, cells_crossed(S, N, R, ps[p], ps[npad + p], ps[2 * (size_t)npad + p],
                                              ps[3 * (size_t)npad + p], ps[4 * (size_t)npad + p], A.dxi));
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) c = fmax(c, __shfl_xor_sync(FULL, c, o));
            if (lane == 0 && c > 0.0) atomicMax(S.cmax, (unsigned long long)__double_as_longlong(c));
            __syncthreads();
            const double cm = __longlong_as_double((long long)*S.cmax);
            int n = cm <= A.max_cells ? 1 : (int)ceil(cm / A.max_cells);
            const double hlast = S.absl[8 * abp + 6];
            if (hlast > 0.0) n = max(n, (int)ceil(A.dxi / (2.0 * hlast) - 1e-9));
            nsub = min(n, A.substep_max > 0 ? A.substep_max : 64);
            if (tid == 0 && nsub > 1) S.fx[11] += nsub - 1;
        }
        const double hstep = A.dxi / nsub;
        const bool to_next = ss == nsub - 1;       // this push's deposit builds slice k+1, else the next sub-slice
        // The accumulators of the deposit: buffer s (with double-buffered sources its slice is stored and the
        // next slice's start values already sit in sn; with one buffer s is sn). Its values go to sn for
        // the next slice, or stay in s for the next sub-slice. Zeroed (all 9 arrays) after the store.
        const Src acc = s;
        const Src dst = to_next ? sn : s;
        {
            const size_t fb = (size_t)k * M;
            // a node's 6 field components start on 16 bytes when the field store does
            const bool f16 = (reinterpret_cast<uintptr_t>(gate.fld(A)) & 15) == 0;
            for (int j = tid; j < M; j += kThreads) {
                if (ss == 0) {
                    double* F = gate.fld(A) + (fb + j) * F_NC0;
                    const double br = S.bpr[j], bi = S.bpi[j], w1 = S.wr1[j];
                    put2(F + F_EP1R, w1 + bi, 0.0 - br, f16);
                    put2(F + F_BP1R, br, bi, f16);
                    put2(F + F_EZ0, S.ez[j], S.bz[j], f16);
                    double* D = gate.diag(A) + (fb + j) * D_NC0;
                    D[D_PSI0] = S.psi[j];
                    D[D_NE0] = s.ne[j];
                    D[D_NI0] = s.ni[j];
                    if (double* const W = gate.wrec(A)) W[fb + j] = w1;
                }
                if (k + 1 < K) {
#pragma unroll
                    for (int c = 0; c < 7; ++c) dep_arr(acc, c)[j] = 0.0;
                    acc.S1r[j] = 0.0;
                    acc.S1i[j] = 0.0;
                }
            }
        }
        if (k + 1 < K) {
            // the beam part the deposit's values start from, for this thread's rows: slice k+1's (one buffer), loaded
            // here without a use so that the push hides the latency, or slice k's extrapolated to the next sub-slice
            BeamRaw raw[kPre];
            if (kPre == kMaxR && to_next && !dbuf)
#pragma unroll
                for (int u = 0; u < kPre; ++u)
                    raw_load<Gate::kActive>(A, gate.bsrc(A), k + 1, min(tid + u * kThreads, N), raw[u]);
            const bool first = (k == 0) && (ss == 0) && !A.pin_pushed;
            double abc[5];
            coeffs(hstep, first, abc);
            if (REG) {
                bool act = tid < np && P.w != 0.0;
                double v[12];
                if (act) {
                    species_params(A, tid, P.q, P.qm);
                    if (kHS && !first) hist_get<ORD>(P, S, hs);
                    const int pr = push_particle(P, keep_geo(S, kp, J), kp.k, S, A, first, abc, hstep);
                    if (kHS) {
                        hs = hs + 1 == ORD ? 0 : hs + 1;
                        hist_put<ORD>(P, S, hs, first || pr == 2);
                    }
                    if (pr > 0) {
                        polar(P.x, P.y, kp.rp, kp.ir, kp.c, kp.s);
                        J = locate_from(S.r, N, R, kp.rp, J);
                        deposit_values(P, keep_geo(S, kp, J), kp.k, S, v);
                    } else {
                        act = false;
                        atomicAdd(S.lost, 1);
                        if (pr < 0) atomicAdd(S.fx + 12, 1);
                    }
                }
                const bool tail = deposit_runs<true>(act, J, P.q < 0.0, v, S.fx);
                __syncthreads();                  // (the maxima, and the accumulators cleared after the store above)
                deposit_add(tail, J, P.q < 0.0, v, acc, S.fx, bits_p);
                __syncthreads();
            } else {
                // pass 0 pushes, takes the exponent maxima and adds in the quanta of the last deposit; pass 1, when
                // the maxima moved, recomputes the deposit values of the pushed particles and adds them again
                __syncthreads();                  // the accumulators have been cleared, after the store above
                for (int pass = 0; pass < 2; ++pass) {
                    for (int base = tid - lane; base < np; base += kThreads) {
                        const int p = base + lane;
                        bool act = false;
                        int j = 0;
                        double v[12];
                        PState<ORD> Q;
                        if (p < np) {
                            pbase(Q, S, A, gate.ps(A), npad, p);
                            species_params(A, p, Q.q, Q.qm);
                            if (Q.w != 0.0) {
                                if (pass == 0) {
                                    phist(Q, gate.ps(A), npad, p);
                                    const PGeo g = pgeo(S, A, N, R, p, Q.x, Q.y);
                                    KinNone kin;
                                    const int pr = push_particle(Q, g, kin, S, A, first, abc, hstep);
                                    if (pr > 0) {
                                        PGeo g2;
                                        if (A.pcache) {        // the new cell by a short walk from the old one
                                            const int jn = locate_from(S.r, N, R, sqrt(Q.x * Q.x + Q.y * Q.y), g.j);
                                            g2 = geometry_in(S.r, S.ih, Q.x, Q.y, jn);
                                            S.pj[p] = jn;
                                        } else {
                                            g2 = geometry(S.r, S.ih, N, R, Q.x, Q.y);
                                        }
                                        j = g2.j;
                                        deposit_values(Q, g2, kin, S, v);
                                        act = true;
                                    } else {
                                        atomicAdd(S.lost, 1);
                                        if (pr < 0) atomicAdd(S.fx + 12, 1);
                                    }
                                    pstore(Q, gate.ps(A), npad, p);
                                    pbase_put(Q, S, A, p);
                                } else {
                                    const PGeo g2 = pgeo(S, A, N, R, p, Q.x, Q.y);
                                    j = g2.j;
                                    deposit_values(Q, g2, KinNone{}, S, v);
                                    act = true;
                                }
                            }
                        }
                        const bool neg = act && Q.q < 0.0;
                        const bool tail = pass == 0 ? deposit_runs<true>(act, j, neg, v, S.fx)
                                                    : deposit_runs<false>(act, j, neg, v, S.fx);
                        deposit_add(tail, j, neg, v, acc, pass == 0 ? S.fxp : S.fx, bits_p);
                    }
                    __syncthreads();
                    if (pass == 1 || !fx_moved<7>(S.fx, S.fxp)) break;
                    deposit_clear(acc, M);
                    __syncthreads();
                }
            }
            if (tid == 0)
                for (int c = 0; c < 7; ++c) S.fx[13] += S.fx[c] == 2047;
#pragma unroll
            for (int u = 0; u < kMaxR; ++u) {
                const int i = tid + u * kThreads;
                if (i >= M) continue;
                double b0[7];
                if (to_next && dbuf) {
#pragma unroll
                    for (int c = 0; c < 7; ++c) b0[c] = dep_arr(sn, c)[i];
                } else {
                    init_base<EXT>(S, i,
                                   to_next ? (kPre == kMaxR ? raw_row<Gate::kActive, EXT>(A, gate.bsrc(A), k + 1, i,
                                                                                          raw[u < kPre ? u : 0])
                                                            : beam_row<Gate::kActive, EXT>(A, gate.bsrc(A), k + 1, i))
                                           : beam_row_at<Gate::kActive, EXT>(A, gate.bsrc(A), k, i, (ss + 1) * hstep),
                                   M, b0);
                }
                deposit_finish(dst, acc, i, b0, S.fx, bits_p);
            }
        }
        if (Gate::kActive && to_next) gate.slice_done_all(k);          // every thread, before the barrier
        __syncthreads();
        PHASE_MARK(4);
        if (Gate::kActive && to_next) {
            if (tid < 32) {                                   // warp 0: publish slice k, check the next rows
                bool ok = true;
                if (tid == 0) ok = gate.slice_done(k);
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (ok && k + 1 < K) ok = gate.before_rows(k + 3 < K ? k + 3 : K - 1);
                if (tid == 0) *S.flag = ok ? 1 : 0;
            }
            __syncthreads();
            if (!*S.flag) return false;
        }
    }   // the passes of slice k
    }
    if (A.pout) {
        // a slab that hands its plasma on: push the last slice too (src/Simulation.cpp:755, the push of the
        // last local slice produces the state entering the next slab), no deposit
        const bool first = (K == 1) && !A.pin_pushed;
        double abc[5];
        coeffs(A.dxi, first, abc);
        if (REG) {
            if (tid < np && P.w != 0.0) {
                if (kHS && !first) hist_get<ORD>(P, S, hs);
                const int pr = push_particle(P, keep_geo(S, kp, J), kp.k, S, A, first, abc, A.dxi);
                if (pr <= 0) { atomicAdd(S.lost, 1); if (pr < 0) atomicAdd(S.fx + 12, 1); }
            } else if (kHS && tid < np) {
                hist_get<ORD>(P, S, hs);               // a particle removed earlier
            }
            if (tid < np) pstore(P, A.pout, npad, tid);
        } else {
            for (int p = tid; p < np; p += kThreads) {
                PState<ORD> Q;
                pload(Q, gate.ps(A), npad, p);
                species_params(A, p, Q.q, Q.qm);
                if (Q.w != 0.0) {
                    KinNone kin;
                    const int pr = push_particle(Q, geometry(S.r, S.ih, N, R, Q.x, Q.y), kin, S, A, first, abc, A.dxi);
                    if (pr <= 0) { atomicAdd(S.lost, 1); if (pr < 0) atomicAdd(S.fx + 12, 1); }
                }
                pstore(Q, gate.ps(A), npad, p);
                pstore(Q, A.pout, npad, p);
            }
        }
        __syncthreads();
    }
    if (REG && tid < np) {
        if (kHS && !A.pout) hist_get<ORD>(P, S, hs);
        pstore(P, gate.ps(A), npad, tid);
    }
    if (tid == 0 && A.counters) {
        atomicAdd(&A.counters[0], (unsigned long long)*S.lost);
        if (S.fx[13]) atomicAdd(&A.counters[1], (unsigned long long)S.fx[13]);
        if (S.fx[12]) atomicAdd(&A.counters[2], (unsigned long long)S.fx[12]);
        if (S.fx[11]) atomicAdd(&A.counters[3], (unsigned long long)S.fx[11]);
    }
    return true;
#undef PHASE_MARK
#undef SUB_MARK
}



}  // namespace qzb
