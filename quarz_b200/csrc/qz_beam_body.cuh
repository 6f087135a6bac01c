// qz_beam_body.cuh -- device functions of the beam path (deposit, gather + Vay push, moment sums),
// shared by the stand-alone beam kernels (qz_beam.cu) and the time-step pipeline (qz_pipeline.cu).
//
// Beam::deposit (src/Beam.cpp:725-785), Beam::advance with the Vay pusher (src/Beam.cpp:948-1131,
// src/Pushers.hpp:63-68), Beam::sums (src/Beam.cpp:1133-1155).
#pragma once
#include "qz_device.cuh"
#include "qz_internal.h"

namespace qzb {
namespace beam_detail {

// kL2: the data was written by other SMs during the same launch, so it is read from L2 (ld.global.cg)
template <bool kL2>
__device__ __forceinline__ double fload(const double* p) { return kL2 ? __ldcg(p) : *p; }
// two neighbouring doubles: one 16-byte load when the address allows it (kVec)
template <bool kL2, bool kVec>
__device__ __forceinline__ double2 fload2(const double* p) {
    if constexpr (kVec) {
        const double2* q = reinterpret_cast<const double2*>(p);
        return kL2 ? __ldcg(q) : *q;
    } else {
        return make_double2(fload<kL2>(p), fload<kL2>(p + 1));
    }
}

// The deposit of one particle (src/Beam.cpp:725-785): its cell, weights, and the values f[c] that every corner
// multiplies by its weight: B_NC0 or B_NC1 components, or (kDep0) the three the m = 0 sweep reads, rho - J_z, J_z
// and J_theta (not the beam's J_r and rho; a field file deposits its beam density again). jguess: a nearby
// radial cell (the gather's, before the push moved the particle), or < 0
constexpr int kDep0 = 3;
template <int NC>
struct DepOne {
    int k, j;
    double d0, tk, t, f[NC];
};

template <int NC>
__device__ __forceinline__ bool dep_one(const BeamArgs& B, double X, double Y, double PX, double PY, double PZ,
                                        double XI, double wi, int jguess, DepOne<NC>& D) {
    const double r = sqrt(X * X + Y * Y);
    if (r > B.R) return false;
    double c = 1.0, s = 0.0;
    if (r > 0.0) {
        const Recip ir(r);
        c = ir(X);
        s = ir(Y);
    }
    const double sx = (XI - B.xi_min) * B.idxi;
    D.k = B.ngp ? (int)floor(sx + 0.5) : (int)floor(sx);
    if (D.k < -1 || D.k >= B.K) return false;
    D.tk = B.ngp ? 0.0 : sx - D.k;
    const double p2 = PX * PX + PY * PY;
    const double gam = sqrt(1.0 + p2 + PZ * PZ);
    const double omvz = (1.0 + p2) / (gam * (gam + PZ));
    const Recip ig(gam);
    const double vz = ig(PZ), vx = ig(PX), vy = ig(PY);
    const double vr = c * vx + s * vy, vt = c * vy - s * vx;
    D.j = locate_near(B.r, B.N, B.R, r, jguess);
    const double t = (r - B.r[D.j]) * B.inv_h[D.j];
    D.t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
    D.d0 = wi * B.q;
    if constexpr (NC == kDep0) {
        D.f[0] = omvz; D.f[1] = vz; D.f[2] = vt;
    } else {
        D.f[B_RT0] = omvz; D.f[B_JZ0] = vz; D.f[B_JP1R] = vr; D.f[B_JP1I] = vt; D.f[B_RHO0] = 1.0;
    }
    if constexpr (NC == B_NC1) {
        const double c2 = c * c - s * s, s2 = 2.0 * c * s;
        D.f[B_RT1R] = omvz * c; D.f[B_RT1I] = -omvz * s;
        D.f[B_JZ1R] = vz * c; D.f[B_JZ1I] = -vz * s;
        D.f[B_RHO1R] = c; D.f[B_RHO1I] = -s;
        D.f[B_JP0R] = vx; D.f[B_JP0I] = vy;
        D.f[B_JP2R] = vx * c2 + vy * s2; D.f[B_JP2I] = vy * c2 - vx * s2;
    }
    return true;
}

// adds a particle's deposit to its nodes, each value by the calling lane
template <int NC>
__device__ __forceinline__ void lane_deposit(const BeamArgs& B, double* __restrict__ bsrc, const DepOne<NC>& D) {
#pragma unroll 1
    for (int a = 0; a < (B.ngp ? 1 : 2); ++a) {
        const int kk = D.k + a;
        if (kk < 0 || kk >= B.K) continue;
        const double Wk = a ? D.tk : 1.0 - D.tk;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            double* const o = bsrc + ((size_t)kk * B.M + D.j + b) * NC;
            const double d = D.d0 * Wk * (b ? D.t : 1.0 - D.t) * B.inv_V[D.j + b] * B.idxi;
            if (B.fx_scale) {                                    // exact (m = 0 runs of qz_sim)
                const double sc = B.fx_scale[D.j + b];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    double hi = 0.0, lo = 0.0;
                    beam_fx_split(d * D.f[c], sc, B.fx_inv2s, B.fx_2s, hi, lo);
                    atomicAdd(o + c, hi);
                    atomicAdd(o + c + B.fx_lo, lo);
                }
            } else {
#pragma unroll
                for (int c = 0; c < NC; ++c) atomicAdd(o + c, d * D.f[c]);
            }
        }
    }
}

template <int NC>
__device__ __forceinline__ void deposit_one(const BeamArgs& B, double* __restrict__ bsrc, double X, double Y,
                                            double PX, double PY, double PZ, double XI, double wi, int jguess = -1) {
    DepOne<NC> D;
    if (dep_one<NC>(B, X, Y, PX, PY, PZ, XI, wi, jguess, D)) lane_deposit<NC>(B, bsrc, D);
}

// The deposit of a warp's particles into compact m = 0 beam sources: kDep0 values per node, or (kExact) their
// high limbs and then their low limbs, so that a particle's 2 nodes of a row are 6 or 12 contiguous doubles. A
// reduction instruction of a particle per lane costs its SM one cycle per lane and value; here the values go
// through shared memory and consecutive lanes add consecutive addresses (0.4 cycles per value). Lanes in the
// same cell are summed first. The exact limbs are integers, so no order of the adds shows in the sums.
template <bool kExact>
struct WarpDep3 {
    static constexpr int kW = 2 * kDep0 * (kExact ? 2 : 1);      // values of a row
    double val[32][kW + 1];                                      // odd row length: no bank conflicts
    long off[32];
    unsigned mask[32];
    unsigned char lead[32];
};

// every lane of the warp calls it; act: the lane has a particle to deposit
template <bool kExact>
__device__ __forceinline__ void warp_deposit3(const BeamArgs& B, double* __restrict__ bsrc, bool act,
                                              const DepOne<kDep0>& D, WarpDep3<kExact>& W) {
    constexpr int kW = WarpDep3<kExact>::kW;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned key = act ? (unsigned)((D.k + 1) * B.M + D.j) : 0xffffffffu - lane;
    const unsigned same = __match_any_sync(FULL, key);
    const bool lead = act && lane == __ffs(same) - 1;
    if (lead) {
        W.off[lane] = ((long)D.k * B.M + D.j) * (kW / 2);
        W.mask[lane] = same;
    }
    double w2[2];
    if (act) {
        w2[0] = D.d0 * (1.0 - D.t) * B.inv_V[D.j] * B.idxi;
        w2[1] = D.d0 * D.t * B.inv_V[D.j + 1] * B.idxi;
    }
#pragma unroll 1
    for (int a = 0; a < (B.ngp ? 1 : 2); ++a) {
        // rows ahead of or behind the box are nobody's to add to (kept out by their index: a value that is not finite
        // times a zero weight is not zero)
        const int kk = D.k + a;
        const bool in = kk >= 0 && kk < B.K;
        const unsigned leads = __ballot_sync(FULL, lead && in);
        if (lead && in) W.lead[__popc(leads & ((1u << lane) - 1u))] = (unsigned char)lane;
        const int total = __popc(leads) * kW;
        if (act && in) {
            const double Wk = a ? D.tk : 1.0 - D.tk;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const double d = w2[b] * Wk;
#pragma unroll
                for (int c = 0; c < kDep0; ++c) {
                    const double v = d * D.f[c];
                    if constexpr (kExact) {
                        double hi = 0.0, lo = 0.0;
                        beam_fx_split(v, B.fx_scale[D.j + b], B.fx_inv2s, B.fx_2s, hi, lo);
                        W.val[lane][b * 2 * kDep0 + c] = hi;
                        W.val[lane][b * 2 * kDep0 + kDep0 + c] = lo;
                    } else {
                        W.val[lane][b * kDep0 + c] = v;
                    }
                }
            }
        }
        __syncwarp();
        double* const row = bsrc + (size_t)a * B.M * (kW / 2);
        for (int q = lane; q < total; q += 32) {
            const int sl = q / kW, w = q - sl * kW, src = W.lead[sl];
            double v = W.val[src][w];
            for (unsigned m = W.mask[src] & ~(1u << src); m; m &= m - 1) v += W.val[__ffs(m) - 1][w];
            if (v != 0.0) atomicAdd(row + W.off[src] + w, v);
        }
        __syncwarp();
    }
}

// The part of the m = 1 deposit that the m = 1 sweep reads (rho - J_z, J_z and J_perp in modes 0 and 1,
// J_perp also in mode 2; not the beam densities), per corner: deposit_setup1 takes the particle's cell,
// weights and velocities once (as dep_one with mode 1, src/Beam.cpp:725-785), deposit_corner1 the 12
// values of corner (row k + a, node j + b), deposit_add1 adds them with FP64 reductions.
constexpr int kDep1 = 12;
struct Dep1 {
    int k, j;
    double d0, tk, t, c, s, omvz, vz, vx, vy, vr, vt;
};
__device__ __forceinline__ bool deposit_setup1(const BeamArgs& B, double X, double Y, double PX, double PY, double PZ,
                                               double XI, double wi, int jguess, Dep1& D) {
    const double R = B.R;
    const double r = sqrt(X * X + Y * Y);
    if (r > R) return false;
    D.c = r > 0.0 ? X / r : 1.0;
    D.s = r > 0.0 ? Y / r : 0.0;
    const double sx = (XI - B.xi_min) * B.idxi;
    D.k = B.ngp ? (int)floor(sx + 0.5) : (int)floor(sx);
    if (D.k < -1 || D.k >= B.K) return false;
    D.tk = B.ngp ? 0.0 : sx - D.k;
    const double p2 = PX * PX + PY * PY;
    const double gam = sqrt(1.0 + p2 + PZ * PZ);
    D.omvz = (1.0 + p2) / (gam * (gam + PZ));
    D.vz = PZ / gam; D.vx = PX / gam; D.vy = PY / gam;
    D.vr = D.c * D.vx + D.s * D.vy;
    D.vt = D.c * D.vy - D.s * D.vx;
    D.j = locate_near(B.r, B.N, R, r, jguess);
    const double t = (r - B.r[D.j]) * B.inv_h[D.j];
    D.t = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
    D.d0 = wi * B.q;
    return true;
}
// corner (a, b): v in the order B_RT0, B_RT1R, B_RT1I, B_JZ0, B_JZ1R, B_JZ1I, B_JP0R, B_JP0I, B_JP1R,
// B_JP1I, B_JP2R, B_JP2I; zero for a row outside the box or the second row of the ngp shape
__device__ __forceinline__ void deposit_corner1(const BeamArgs& B, const Dep1& D, int a, int b,
                                                double (&v)[kDep1]) {
    const int kk = D.k + a;
    const bool row = (a == 0 || !B.ngp) && kk >= 0 && kk < B.K;
    const double Wk = a ? D.tk : 1.0 - D.tk, Wr = b ? D.t : 1.0 - D.t;
    const double d = row ? D.d0 * Wk * Wr * B.inv_V[D.j + b] * B.idxi : 0.0;
    const double c2 = D.c * D.c - D.s * D.s, s2 = 2.0 * D.c * D.s;
    v[0] = d * D.omvz; v[1] = d * D.omvz * D.c; v[2] = -d * D.omvz * D.s;
    v[3] = d * D.vz; v[4] = d * D.vz * D.c; v[5] = -d * D.vz * D.s;
    v[6] = d * D.vx; v[7] = d * D.vy;
    v[8] = d * D.vr; v[9] = d * D.vt;
    v[10] = d * (D.vx * c2 + D.vy * s2); v[11] = d * (D.vy * c2 - D.vx * s2);
}
__device__ __forceinline__ void deposit_add1(const BeamArgs& B, double* __restrict__ bsrc, int kk, int jj,
                                             const double (&v)[kDep1]) {
    if (kk < 0 || kk >= B.K) return;
    constexpr int comp[kDep1] = {B_RT0, B_RT1R, B_RT1I, B_JZ0, B_JZ1R, B_JZ1I, B_JP0R, B_JP0I, B_JP1R, B_JP1I,
                                 B_JP2R, B_JP2I};
    double* o = bsrc + ((size_t)kk * B.M + jj) * B_NC1;
#pragma unroll
    for (int c = 0; c < kDep1; ++c) atomicAdd(o + comp[c], v[c]);
}

// bilinear (xi, r) gather and mode sums at the particle (src/Beam.cpp:972-1008). kVec: fld starts on a
// 16-byte boundary (its rows of 6 or 18 doubles then do too), so the components are read two at a time
template <bool kL2, bool kVec = false>
__device__ __forceinline__ void gather(const BeamArgs& B, const double* __restrict__ fld, double X, double Y,
                                       double XI, double& c, double& sn, V3& E, V3& Bf, int* jcell = nullptr) {
    const double r = sqrt(X * X + Y * Y);
    c = 1.0;
    sn = 0.0;
    if (r > 0.0) {
        const Recip ir(r);
        c = ir(X);
        sn = ir(Y);
    }
    double s = (XI - B.xi_min) * B.idxi;
    const int nloc = B.K;
    int k;
    double tk;
    if (B.ngp) {
        k = (int)floor(s + 0.5);
        k = k < 0 ? 0 : (k > nloc - 1 ? nloc - 1 : k);
        tk = 0.0;
    } else {
        k = (int)floor(s);
        if (k < 0) { k = 0; s = 0.0; }
        if (k > nloc - 2) { k = nloc - 2; s = nloc - 1; }
        tk = s - k;
    }
    const int k1 = B.ngp ? k : k + 1;
    int j;
    double t;
    weights(B.r, B.inv_h, B.N, B.R, r, j, t);
    if (jcell) *jcell = j;
    const int nc = B.modes ? F_NC1 : F_NC0;
    const double* f00 = fld + ((size_t)k * B.M + j) * nc;
    const double* f01 = f00 + nc;
    const double* f10 = fld + ((size_t)k1 * B.M + j) * nc;
    const double* f11 = f10 + nc;
    // components comp and comp + 1 (comp even): a complex field component, or E_z and B_z
    auto bil = [&](int comp, double& u, double& v) {
        const double2 a = fload2<kL2, kVec>(f00 + comp), b = fload2<kL2, kVec>(f01 + comp);
        const double2 d = fload2<kL2, kVec>(f10 + comp), e = fload2<kL2, kVec>(f11 + comp);
        u = (1.0 - tk) * ((1.0 - t) * a.x + t * b.x) + tk * ((1.0 - t) * d.x + t * e.x);
        v = (1.0 - tk) * ((1.0 - t) * a.y + t * b.y) + tk * ((1.0 - t) * d.y + t * e.y);
    };
    double er, ei, br, bi, ez, bz;
    bil(F_EP1R, er, ei);
    bil(F_BP1R, br, bi);
    bil(F_EZ0, ez, bz);
    E.x = er * c - ei * sn;
    E.y = er * sn + ei * c;
    Bf.x = br * c - bi * sn;
    Bf.y = br * sn + bi * c;
    E.z = ez;
    Bf.z = bz;
    if (B.modes) {
        // eval_vector / eval_scalar with m = 1 (src/SliceData.hpp:70-83)
        const double c2 = c * c - sn * sn, s2 = 2.0 * c * sn;
        double r0, i0, r2, i2;
        bil(F_EP0R, r0, i0);
        bil(F_EP2R, r2, i2);
        E.x += r0 + r2 * c2 - i2 * s2;
        E.y += i0 + r2 * s2 + i2 * c2;
        bil(F_BP0R, r0, i0);
        bil(F_BP2R, r2, i2);
        Bf.x += r0 + r2 * c2 - i2 * s2;
        Bf.y += i0 + r2 * s2 + i2 * c2;
        bil(F_EZ1R, r0, i0);
        E.z += 2.0 * (r0 * c - i0 * sn);
        bil(F_BZ1R, r0, i0);
        Bf.z += 2.0 * (r0 * c - i0 * sn);
    }
}


// One particle of Beam::advance (src/Beam.cpp:948-1131): gather at the old position, optional explicit
// start-up kick with the same fields (h_start != 0, src/Beam.cpp:1038-1044), Vay with h = q/m dt_kick/2,
// drift, removal at the wall or outside the box. Returns false when the particle was removed.
struct PState7 {
    double x, y, px, py, pz, xi, w;
};

template <bool kL2, bool kVec = false>
__device__ __forceinline__ bool push_one(const BeamArgs& B, const double* __restrict__ fld, PState7& p, double h,
                                         double h_start, double dt, int* jcell = nullptr) {
    double c, sn;
    V3 E, Bf;
    gather<kL2, kVec>(B, fld, p.x, p.y, p.xi, c, sn, E, Bf, jcell);
    V3 u = {p.px, p.py, p.pz};
    if (h_start != 0.0) {
        const double g0 = sqrt(1.0 + dot3(u, u));
        const double ig = 1.0 / g0;
        const V3 v = {ig * u.x, ig * u.y, ig * u.z};
        const V3 vxb = cross3(v, Bf);
        const double h2 = 2.0 * h_start;
        u = {u.x + h2 * (E.x + vxb.x), u.y + h2 * (E.y + vxb.y), u.z + h2 * (E.z + vxb.z)};
    }
    u = vay(u, E, Bf, h);
    const double p2 = u.x * u.x + u.y * u.y;
    const double gam = sqrt(1.0 + p2 + u.z * u.z);
    const double omvz = (1.0 + p2) / (gam * (gam + u.z));
    const Recip ig(gam);
    const double xn = p.x + ig(u.x) * dt, yn = p.y + ig(u.y) * dt;
    const double xin = p.xi + omvz * dt;
    const double xmin = B.xi_min, xmax = B.xi_min + (B.K - 1) * B.dxi;
    p.x = xn; p.y = yn; p.px = u.x; p.py = u.y; p.pz = u.z; p.xi = xin;
    if (xn * xn + yn * yn >= B.R * B.R || xin < xmin || xin > xmax) {
        p.w = 0.0;
        return false;
    }
    return true;
}

// the weighted moments of Beam::sums (src/Beam.cpp:1133-1155) of one particle, added to acc[17]
__device__ __forceinline__ void sums_add(double* acc, const PState7& p, double gref, double xiref) {
    const double g = sqrt(1.0 + p.px * p.px + p.py * p.py + p.pz * p.pz);
    const double G = g - gref, XI = p.xi - xiref;
    const double v[15] = {G, G * G, XI, XI * XI, p.x * p.x + p.y * p.y, p.x, p.y, p.x * p.x, p.y * p.y,
                          p.px, p.py, p.px * p.px, p.py * p.py, p.x * p.px, p.y * p.py};
    acc[16] += 1.0;
    acc[0] += p.w;
#pragma unroll
    for (int c = 0; c < 15; ++c) acc[c + 1] += p.w * v[c];
}

// sums_add into one lane's accumulators in shared memory (a[c * 32], c = 0..16): the same operations
__device__ __forceinline__ void sums_add_lane(double* a, const PState7& p, double gref, double xiref) {
    const double g = sqrt(1.0 + p.px * p.px + p.py * p.py + p.pz * p.pz);
    const double G = g - gref, XI = p.xi - xiref;
    const double v[15] = {G, G * G, XI, XI * XI, p.x * p.x + p.y * p.y, p.x, p.y, p.x * p.x, p.y * p.y,
                          p.px, p.py, p.px * p.px, p.py * p.py, p.x * p.px, p.y * p.py};
    a[16 * 32] += 1.0;
    a[0] += p.w;
#pragma unroll
    for (int c = 0; c < 15; ++c) a[(c + 1) * 32] += p.w * v[c];
}

// the xi cell of a particle for bucketing: floor((xi - xi_min)/dxi) clamped to [-1, K-1]
__device__ __forceinline__ int xi_cell(const BeamArgs& B, double xi) {
    const double s = (xi - B.xi_min) * B.idxi;
    if (!(s >= -1.0)) return -1;
    if (s >= (double)(B.K - 1)) return B.K - 1;
    return (int)floor(s);
}

}  // namespace beam_detail
}  // namespace qzb
