// Spalart-Allmaras one-equation model (turbulenceModel 1) on the device.
//
// nu~ is component 6 of the level's state arrays ([6][N]).  Each edge loop
// of the reference becomes a node gather over the CSR incidence lists in
// edge order (then the boundary edges in their order), and every expression
// keeps the reference's operation order, so the results equal the CPU
// restatement bit for bit:
//   k_sa_grad      makeTurbulentTimeSteps  (def_par:12878-13100) and
//                  makeSADiffusion pass 1  (def_par:7436-7560): Galerkin
//                  gradient of nu~ and the cb2 term
//   k_sa_diff      makeSADiffusion pass 2  (def_par:7560-7809)
//   k_sa_conv      makeSARHS               (def_par:6809-6950)
//   k_sa_stage     the nu~ part of one RK stage / of restrictGrid's coarse
//                  and fine one-step updates: makeSASourceTerm (def_par:
//                  9285-9371), the diffusion term, solveTurbulenceSystem,
//                  the increment and solution conditions, nullifyOuterBoundary,
//                  updateSolutionVector, the FAS source, limitTurbulence and
//                  the far-field value (def_par:1002-1181, 12141-12430)
// k_sa_stage runs before the mean-flow node update of the same stage: it
// reads the stage-start density, which that update overwrites.
#include <cuda_runtime.h>

#include "gather.cuh"
#include "kernels.h"
#include "pinned_math.h"

namespace flite {

namespace {
__device__ __forceinline__ int tid() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ bool sa_wall(unsigned char cls) { return cls == BC_WALL || cls == BC_IWALL; }
__device__ __forceinline__ bool sa_far(unsigned char cls) { return cls == BC_FAR3 || cls == BC_FAR4; }
__device__ __forceinline__ double rp_exhaust(const Params &P, const LevelView &L, unsigned char cls) {
    return sa_exhaust(P, cls, eo_relax(P, *L.cyc));
}
}  // namespace

// The gathers take a thread or a group of lanes per node (lanes_of): on the
// coarse levels of a 738,100-node mesh (78,360 to 53 nodes) a thread per node
// takes 10 to 30 us a launch, one thread's chain of loads and divisions.
//
// makeTurbulentTimeSteps (def_par:12878-13100, ts) and the Galerkin gradient of
// nu~ with the cb2 term of makeSADiffusion (def_par:7436-7560), which read nu~ of
// the same neighbours
namespace {
struct SaConst {
    double oneOverSigma = 3.0 / 2.0, oneOverKappaSquared = 1.0 / (0.41 * 0.41);
    double cb1 = 0.1355, cb2 = 0.622, ct3 = 1.1;
};
// the terms of incidence t: v[0] the convective term, v[1] the other node's
// diffusion term (def_par:12930-12935)
__device__ __forceinline__ void sa_ts_terms(const Params &P, const LevelView &L, const int2 t, const double *m,
                                            double ro, double oRe, double *v) {
    const SaConst k;
    const int N = L.N, e = t.x >= 0 ? t.x : ~t.x, j = t.y;
    const double wx = L.wx[e], wy = L.wy[e], wz = L.wz[e];
    const double al = (wx * wx + wy * wy) + wz * wz;
    const double vn = ((wx * m[0] + wy * m[1]) + wz * m[2]) * ro;
    v[0] = P.turbK * sqrt(al) + fabs(vn);
    const double vis = k.oneOverSigma * (L.mu[j] + 3.0 * k.cb2 * L.u[5 * (size_t)N + j] * oRe);
    v[1] = 2.0 * vis * al;
}
// boundary entry q: the two terms of each of the two sums
__device__ __forceinline__ void sa_ts_bterms(const Params &P, const LevelView &L, int q, double oRe, double *v) {
    const SaConst k;
    const int N = L.N;
    const double *nt = L.u + 5 * (size_t)N;
    const int b = L.binc[q] >> 1, side = L.binc[q] & 1;
    const int2 nd = L.bedge[b];
    const double wx = L.bwx[b], wy = L.bwy[b], wz = L.bwz[b];
    const double al = (wx * wx + wy * wy) + wz * wz;
    const int j1 = nd.x, j2 = nd.y;
    const double ro1 = 1. / L.u[j1], ro2 = 1. / L.u[j2];
    double vn1 = ((wx * L.u[N + j1] + wy * L.u[2 * N + j1]) + wz * L.u[3 * N + j1]) * ro1;
    double vn2 = ((wx * L.u[N + j2] + wy * L.u[2 * N + j2]) + wz * L.u[3 * N + j2]) * ro2;
    vn1 = P.turbK * sqrt(al) + fabs(vn1);
    vn2 = P.turbK * sqrt(al) + fabs(vn2);
    v[0] = side == 0 ? vn1 : vn2;
    v[1] = vn1 + vn2;
    const double vis1 = k.oneOverSigma * (L.mu[j1] + 3.0 * k.cb2 * nt[j1] * oRe);
    const double vis2 = k.oneOverSigma * (L.mu[j2] + 3.0 * k.cb2 * nt[j2] * oRe);
    const double dv1 = 2.0 * vis1 * al, dv2 = 2.0 * vis2 * al;
    v[2] = side == 0 ? dv1 : dv2;
    v[3] = dv1 + dv2;
}
__device__ __forceinline__ void sa_ts_store(const LevelView &L, int i, double acc, double h, double oRe) {
    const SaConst k;
    const double cw1 = k.cb1 * k.oneOverKappaSquared + (1.0 + k.cb2) * k.oneOverSigma;
    const double nti = L.u[5 * (size_t)L.N + i];
    const double V = L.V[i];
    const double dt = 0.5 / (acc / V + h / (V * V));
    double dInvSquared = L.wdist[i] > 1.0e-10 ? 1.0 / L.wdist[i] : 1.0e10;
    dInvSquared = dInvSquared * dInvSquared;
    const double S = (fabs(L.divg[i]) +
                      k.cb1 * (L.vort[i] + (1.0 + k.ct3) * nti * k.oneOverKappaSquared * dInvSquared * oRe)) +
                     cw1 * nti * dInvSquared * oRe;
    L.dtT[i] = dt / (1.0 + 0.5 * S * dt);
}
// the gradient terms of incidence t (ti: this node's nu~), with its sign
__device__ __forceinline__ void sa_grad_terms(const LevelView &L, const int2 t, double ti, double *v) {
    const int e = t.x >= 0 ? t.x : ~t.x;
    const double tj = L.u[5 * (size_t)L.N + t.y];
    const double s = t.x >= 0 ? ti + tj : tj + ti;  // (nu1 + nu2) in the edge's order
    const double f[3] = {L.wx[e] * s, L.wy[e] * s, L.wz[e] * s};
    for (int c = 0; c < 3; ++c) v[c] = t.x >= 0 ? f[c] : -f[c];
}
__device__ __forceinline__ void sa_grad_bterms(const Params &P, const LevelView &L, int q, double *v) {
    const double *nt = L.u + 5 * (size_t)L.N;
    const int b = L.binc[q] >> 1, side = L.binc[q] & 1;
    const int2 nd = L.bedge[b];
    const double w[3] = {L.bwx[b], L.bwy[b], L.bwz[b]};
    const double t1 = nt[nd.x], t2 = nt[nd.y];
    if (P.boundaryTerm == 1) {
        const double a = side == 0 ? 3. * t1 + t2 : t1 + 3. * t2;
        for (int c = 0; c < 3; ++c) v[c] = a * w[c];
    } else {
        const double a = side == 0 ? t1 : t2;
        for (int c = 0; c < 3; ++c) v[c] = 4. * a * w[c];
    }
}
}  // namespace

// the node, lane and idle groups of a gather kernel
#define SA_NODE()                                                    \
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;               \
    const int i_raw = U > 1 ? tid() / U : tid();                     \
    if (U == 1 && i_raw >= L.N) return;                              \
    const bool active = i_raw < L.N;                                 \
    const int i = active ? i_raw : L.N - 1;                          \
    const int N = L.N

template <int U>
__global__ void k_sa_grad(Params P, LevelView L, int ts) {
    SA_NODE();
    const double oRe = 1. / P.Re;
    const double ti = L.u[5 * (size_t)N + i];
    const double ri = L.u[i], ro = 1. / ri;
    const double m[3] = {L.u[N + i], L.u[2 * N + i], L.u[3 * N + i]};
    double g[3] = {0.0, 0.0, 0.0}, x[2] = {0.0, 0.0};
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 4);
        if (ts) {
            group_sum<U, 2, 1, double>(
                gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
                [&](int q, double *v) { sa_ts_terms(P, L, L.inc[q], m, ro, oRe, v); }, x);
            group_sum<U, 2, 2, double>(
                gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl,
                [&](int q, double *v) { sa_ts_bterms(P, L, q, oRe, v); }, x);
        }
        group_sum<U, 3, 1, double>(
            gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
            [&](int q, double *v) { sa_grad_terms(L, L.inc[q], ti, v); }, g);
        group_sum<U, 3, 1, double>(
            gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl,
            [&](int q, double *v) { sa_grad_bterms(P, L, q, v); }, g);
        if (!active || gl) return;
    } else {
        walk<2, 5>(
            L, i,
            [&](const int2 t, double *v) {
                if (ts) sa_ts_terms(P, L, t, m, ro, oRe, v);
                sa_grad_terms(L, t, ti, v + 2);
            },
            [&](const double *v) {
                if (ts) {
                    x[0] = x[0] + v[0];
                    x[1] = x[1] + v[1];
                }
                for (int c = 0; c < 3; ++c) g[c] = g[c] + v[2 + c];
            });
        for (int q = L.binc_ptr[i]; q < L.binc_ptr[i + 1]; ++q) {
            double v[4];
            if (ts) {
                sa_ts_bterms(P, L, q, oRe, v);
                x[0] = (x[0] + v[0]) + v[1];
                x[1] = (x[1] + v[2]) + v[3];
            }
            sa_grad_bterms(P, L, q, v);
            for (int c = 0; c < 3; ++c) g[c] = g[c] + v[c];
        }
    }
    if (ts) sa_ts_store(L, i, x[0], x[1], oRe);
    const double sigma = 2. / 3., cb2 = 0.622;
    const double fact = oRe * cb2 / sigma;
    const double vt = 1. / L.V[i];
    const double dx = g[0] * vt, dy = g[1] * vt, dz = g[2] * vt;
    L.sag[i] = dx;
    L.sag[N + i] = dy;
    L.sag[2 * N + i] = dz;
    const double vp = (g[0] * dx + g[1] * dy) + g[2] * dz;
    L.sanh[i] = 0.0 - fact * vp;
    L.savis[i] = P.Re * L.mu[i] / ri + ti;
}

// makeSADiffusion's edge terms (def_par:7560-7809): the viscosity of a node
// (savis) and its gradient are this launch's input from k_sa_grad
template <int U>
__global__ void k_sa_diff(Params P, LevelView L) {
    SA_NODE();
    const double sigma = 2. / 3., oRe = 1. / P.Re;
    const double fact = oRe / sigma;
    auto fd = [&](int n, double wx, double wy, double wz) {
        return L.savis[n] * ((wx * L.sag[n] + wy * L.sag[N + n]) + wz * L.sag[2 * N + n]);
    };
    const double vi = L.savis[i], gi[3] = {L.sag[i], L.sag[N + i], L.sag[2 * N + i]};
    auto terms = [&](const int2 t, double *v) {
        const int e = t.x >= 0 ? t.x : ~t.x;
        const double wx = L.wx[e], wy = L.wy[e], wz = L.wz[e];
        const double fi = vi * ((wx * gi[0] + wy * gi[1]) + wz * gi[2]), fj = fd(t.y, wx, wy, wz);
        const double f = fact * (t.x >= 0 ? fi + fj : fj + fi);
        v[0] = t.x >= 0 ? -f : f;
    };
    auto bterms = [&](int q, double *v) {
        const int b = L.binc[q] >> 1, side = L.binc[q] & 1;
        const int2 nd = L.bedge[b];
        const double wx = L.bwx[b], wy = L.bwy[b], wz = L.bwz[b];
        const double fd1 = fd(nd.x, wx, wy, wz), fd2 = fd(nd.y, wx, wy, wz);
        if (P.boundaryTerm == 1) v[0] = -(fact * (side == 0 ? 3. * fd1 + fd2 : fd1 + 3. * fd2));
        else v[0] = -(fact * 4. * (side == 0 ? fd1 : fd2));
    };
    double acc[1] = {0.0};
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 1);
        group_sum<U, 1, 1, double>(
            gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl, [&](int q, double *v) { terms(L.inc[q], v); }, acc);
        group_sum<U, 1, 1, double>(gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl, bterms, acc);
        if (!active || gl) return;
    } else {
        walk<2, 1>(L, i, terms, [&](const double *v) { acc[0] = acc[0] + v[0]; });
        for (int q = L.binc_ptr[i]; q < L.binc_ptr[i + 1]; ++q) {
            double v[1];
            bterms(q, v);
            acc[0] = acc[0] + v[0];
        }
    }
    L.turbDiff[i] = acc[0] + L.sanh[i];
}

// makeSARHS (def_par:6809-6950): the nu~ convection, velocities from saprim
template <int U>
__global__ void k_sa_conv(Params P, LevelView L, int td) {
    SA_NODE();
    const double* __restrict__ nt = L.u + 5 * (size_t)N;
    auto prim = [&](int n, double *q) {
        q[0] = L.saprim[n]; q[1] = L.saprim[N + n]; q[2] = L.saprim[2 * (size_t)N + n];
        q[3] = nt[n];
    };
    double qi[4];
    prim(i, qi);
    auto terms = [&](const int2 t, double *v) {
        const int e = t.x >= 0 ? t.x : ~t.x;
        double qj[4];
        prim(t.y, qj);
        const bool first = t.x >= 0;
        const double u1 = first ? qi[0] : qj[0], v1 = first ? qi[1] : qj[1], w1 = first ? qi[2] : qj[2];
        const double u2 = first ? qj[0] : qi[0], v2 = first ? qj[1] : qi[1], w2 = first ? qj[2] : qi[2];
        const double t1 = first ? qi[3] : qj[3], t2 = first ? qj[3] : qi[3];
        const double wx = L.wx[e], wy = L.wy[e], wz = L.wz[e];
        double fconv = (wx * (u1 * t1 + u2 * t2) + wy * (v1 * t1 + v2 * t2)) + wz * (w1 * t1 + w2 * t2);
        if (fabs(t1 - t2) > 1.0e-20) {
            const double ax = (u2 * t2 - u1 * t1) / (t1 - t2);
            const double ay = (v2 * t2 - v1 * t1) / (t1 - t2);
            const double az = (w2 * t2 - w1 * t1) / (t1 - t2);
            fconv = fconv + fabs((wx * ax + wy * ay) + wz * az) * (t1 - t2);
        }
        v[0] = first ? fconv : -fconv;
    };
    // an unsteady stage's time difference comes first (def_par:1073)
    double acc[1] = {td ? time_difference(P, L, L.u, i, 5) : 0.0};
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 1);
        group_sum<U, 1, 1, double>(
            gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl, [&](int q, double *v) { terms(L.inc[q], v); }, acc);
        if (!active || gl) return;
    } else {
        walk<2, 1>(L, i, terms, [&](const double *v) { acc[0] = acc[0] + v[0]; });
    }
    L.rhs[5 * (size_t)N + i] = acc[0];
}
#undef SA_NODE
#define SA_INST(U)                                                  \
    template __global__ void k_sa_grad<U>(Params, LevelView, int);  \
    template __global__ void k_sa_diff<U>(Params, LevelView);       \
    template __global__ void k_sa_conv<U>(Params, LevelView, int);
SA_INST(1)
SA_INST(4)
SA_INST(8)
SA_INST(16)
SA_INST(32)
#undef SA_INST

// makeSASourceTerm at node i added to r; the laminar viscosity floor writes
// 0.1*Re into the array, as the reference does (def_par:9321-9323)
__device__ __forceinline__ double sa_source(const Params &P, const LevelView &L, int i, double r) {
    using namespace flite_pm;
    const int N = L.N;
    const double oRe = 1. / P.Re;
    const double cb1 = 0.1355, cb2 = 0.622, kappa = 0.41, kappaSquared = kappa * kappa, sigma = 2. / 3.;
    const double cw1 = cb1 / kappaSquared + (1.0 + cb2) / sigma;
    const double cw2 = 0.3, cw3 = 2.0, cv1 = 7.1, ct3 = 1.1, ct4 = 2.0;
    const double cv1Tripled = pm_cube(cv1), cw3InSixth = pm_pow6(cw3), oneOverSix = 1. / 6.;
    const double vt = L.V[i];
    const double mucurl = dmax(L.u[5 * (size_t)N + i], 0.0);
    double mu = L.mu[i];
    if (mu < 0.1 / P.Re) {
        mu = 0.1 * P.Re;
        L.mu[i] = mu;
    }
    double Ksi = L.u[i] * oRe * mucurl / mu;
    Ksi = dmax(Ksi, 0.001);
    const double ft2 = ct3 * pm_exp(-ct4 * Ksi * Ksi);
    const double K3 = pm_cube(Ksi);
    const double d = dmax(L.wdist[i], 1.0e-10);
    const double muOverd = mucurl / d, dSquared = d * d;
    const double fv1 = K3 / (K3 + cv1Tripled);
    const double fv2 = 1.0 - (Ksi / (1.0 + Ksi * fv1));
    const double fv3 = 1.0;
    const double Scurl = fv3 * L.vort[i] + oRe * mucurl * fv2 / (kappaSquared * dSquared);
    double rr;
    if (fabs(Scurl) > 1.0e-10) {
        rr = oRe * mucurl / (Scurl * kappaSquared * dSquared);
        if (rr < 0.0) rr = 0.0;
        if (rr > 100.0) rr = 100.0;
    } else {
        rr = 100.0;
    }
    const double gg = rr + cw2 * (pm_pow6(rr) - rr);
    const double radicand = (1.0 + cw3InSixth) / (pm_pow6(gg) + cw3InSixth);
    const double fw = radicand > 1.0e-10 ? gg * pm_exp(oneOverSix * pm_log(radicand))
                                         : pm_exp(oneOverSix * pm_log(1.0 + cw3InSixth));
    r = r - vt * cb1 * (1.0 - ft2) * Scurl * mucurl;
    r = r + oRe * vt * (cw1 * fw - cb1 * ft2 / kappaSquared) * muOverd * muOverd;
    r = r - vt * mucurl * L.divg[i];
    return r;
}

__global__ void k_sa_stage(Params P, LevelView L, int mode, int stage, int turb) {
    int i = tid();
    if (i >= L.N) return;
    const size_t o6 = 5 * (size_t)L.N + i;
    const unsigned char cls = L.bc[i];
    // convection from k_sa_conv (after the time difference of an unsteady
    // stage, which is all of it when the turbulence is not recomputed)
    double r = turb ? L.rhs[o6] : (P.addts && mode == MODE_STAGE ? time_difference(P, L, L.u, i, 5) : 0.0);
    if (turb) r = sa_source(P, L, i, r);
    // restrictGrid adds the (last computed) diffusion term whether or not
    // the turbulence is recomputed (def_par:12238-12240, 12315-12317)
    if (turb || mode != MODE_STAGE) r = r + L.turbDiff[i];
    // solveTurbulenceSystem: the local step, or the explicit global one
    r = ((P.unsteady && P.explicit_) ? *L.ptsg : L.dtT[i]) * r / L.V[i];
    if (sa_wall(cls) || is_exhaust(cls)) r = 0.0;
    if (is_inlet(cls)) r = P.engRelax * r;  // the engine inlets' relaxation (def_par:5084-5099)
    if (L.grid > 1 && (cls == BC_FAR3 || is_engine(cls))) r = 0.0;  // nullifyOuterBoundary
    const double dtJ = stage > 0 ? P.turbCFL * P.RK[stage - 1] : P.turbCFL;
    double un = L.uprev[o6] - dtJ * r;
    un = dmax(un, 0.0);
    if (sa_wall(cls)) un = 0.0;
    // the exhausts' nu~; an inlet's is zeroed on level 1 by k_engine_finish
    // when its momenta are scaled
    if (is_exhaust(cls)) un = rp_exhaust(P, L, cls);
    if (mode == MODE_STAGE) {
        if (L.grid > 1 && turb) un = un - P.RK[stage - 1] * L.src[o6];
        if (turb) {  // limitTurbulence
            un = dmax(un, 0.0);
            if (un > P.maxTurb) un = P.maxTurb;
        }
        if (sa_far(cls)) un = 0.1;
        L.u[o6] = un;
    } else if (mode == MODE_RCOARSE) {
        if (sa_far(cls)) un = 0.1;
        L.src[o6] = un - L.uprev[o6];
    } else {  // MODE_RFINE
        if (L.grid > 1) un = un - L.src[o6];
        // limitTurbulence(finegrp, rhs(:,6)): floors the increment array and
        // caps the state's nu~ (def_par:1259-1290, 12361-12363)
        un = dmax(un, 0.0);
        if (L.u[o6] > P.maxTurb) L.u[o6] = P.maxTurb;
        if (sa_far(cls)) un = 0.1;
        L.rhs[o6] = un - L.uprev[o6];
    }
}

}  // namespace flite
