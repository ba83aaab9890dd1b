// CUDA kernels of the flow-solver hot path (sm_100a, FP64).
//
// Layout and scheduling:
//  * node state is SoA [component][node] so node kernels read and write each
//    component coalesced;
//  * the interior edges' central fluxes are computed by both endpoints inside
//    the node kernel; the upwind fluxes once per edge into an edge buffer
//    [E][5], which the node kernel reads.  Either way a node sums its
//    incident edges in edge order, which reproduces the reference's scatter
//    loop (rhs(i1)+=f, rhs(i2)-=f in edge order) bit for bit, with no atomics;
//  * every gather has two shapes: a thread per node on large levels, several
//    lanes per node on small ones (gather.cuh);
//  * cheap edge terms (time step, JST Laplacian and sensor, JST flux,
//    gradients, min/max) are recomputed by both endpoints inside a node
//    gather, which replaces an edge buffer round trip by reads of the
//    neighbour's state;
//  * everything the reference does per node after the residual (add the
//    dissipation, multiply by dt/V, boundary conditions on the increment,
//    the clipped update, boundary conditions on the solution, the FAS
//    source, the density floor, the far-field conditions) is fused into the
//    node kernel that gathers the residual;
//  * the kernels of the multigrid cycle also have a group form (template
//    flag B): one launch serves every case of a batch's case group, the
//    case in blockIdx.y and its parameters and level views among the
//    arguments (FLITE_CASE_P / FLITE_CASE_L).
#include <cuda_runtime.h>

#include "flux.cuh"
#include "gather.cuh"
#include "kernels.h"
#include "pinned_math.h"

namespace flite {

static __device__ __forceinline__ int tid() { return blockIdx.x * blockDim.x + threadIdx.x; }

// ---- makePressureField (def_par:13612-13630) ------------------------------
// One pass over the state: the pressure, the node records, and on request the
// (u, v, w, T) of the viscous routine (def_par:5260-5270; each edge of the
// reference divides again, the quotients are the same numbers) and the start
// of a relaxation step (def_par:983-987), which would each read the state
// again in a launch of their own.  Bound by its bytes: 40 read, 56 written
// per node, 40 more with the step's copy and 32 with the primitives.
template <bool BND, bool B>
__global__ void k_state_pass(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_, int what, const int *src) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int i = tid();
    const int N = L.N;
    if (i >= N) {
        // a boundary edge; its nodes' pressures are formed here as the node
        // threads form them
        if (!BND || i - N >= L.B) return;
        const auto state = [&](int j) {
            NodeState s;
            s.r = L.u[j]; s.ru = L.u[N + j]; s.rv = L.u[2 * N + j]; s.rw = L.u[3 * N + j]; s.E = L.u[4 * N + j];
            s.p = pressure(P, s.r, s.ru, s.rv, s.rw, s.E);
            return s;
        };
        double g1[5], g2[5];
        boundary_flux(P, L, i - N, state, g1, g2);
        double *o = L.bflux + (size_t)(i - N) * 10;
        for (int k = 0; k < 5; ++k) { o[k] = g1[k]; o[5 + k] = g2[k]; }
        return;
    }
    const double r = L.u[i], ru = L.u[N + i], rv = L.u[2 * N + i], rw = L.u[3 * N + i], E = L.u[4 * N + i];
    if (what & STATE_STEP) {
        if (i == 0) *L.cyc = *src;
        L.uprev[i] = r; L.uprev[N + i] = ru; L.uprev[2 * N + i] = rv; L.uprev[3 * N + i] = rw; L.uprev[4 * N + i] = E;
        if (L.nvar == 6) L.uprev[5 * (size_t)N + i] = L.u[5 * (size_t)N + i];
    }
    const double p = pressure(P, r, ru, rv, rw, E);
    L.p[i] = p;
    if (what & STATE_REC) store_node(L.q, i, r, ru, rv, rw, E, p);
    if (L.saprim) store_saprim(L, i, r, ru, rv, rw);
    if (what & STATE_HPRIM) { L.hprim[i] = ru / r; L.hprim[N + i] = rv / r; L.hprim[2 * N + i] = rw / r; }
    if (what & STATE_PRIM) {
        const double gOg = P.gamma / (P.gamma - 1.0);
        L.prim[i] = ru / r;
        L.prim[N + i] = rv / r;
        L.prim[2 * N + i] = rw / r;
        L.prim[3 * N + i] = gOg * p / r;
    }
}

// ---- makeTimeSteps (def_par:13335-13610) as a node gather -----------------
// The pieces of the gather, shared by the separate kernel and the fused walks
// below, with a thread or a group of lanes per node.
//
// interior edge t of node i (momentum m, 1/rho ro, cc = max(gamma p/rho,
// 0.001)): the convective and acoustic terms, and with viscosity the other
// node's viscous term (def_par:13432-13433; with SA the viscosity is
// mu + nu~/Re)
__device__ __forceinline__ void ts_terms(const Params &P, const LevelView &L, int2 t, double m1, double m2, double m3,
                                         double ro, double cc, double *v) {
    const int N = L.N;
    const int e = t.x >= 0 ? t.x : ~t.x;
    const double wx = L.wx[e], wy = L.wy[e], wz = L.wz[e];
    const double al = (wx * wx + wy * wy) + wz * wz;
    const double vn = ((wx * m1 + wy * m2) + wz * m3) * ro;
    v[0] = fabs(vn);
    v[1] = sqrt(cc * al);
    if (P.viscous) {
        const int j = t.y;
        const double vis = dmax(P.am, P.sa ? L.mu[j] + L.u[5 * N + j] / P.Re : L.mu[j]);
        v[2] = 2.0 * vis * al / L.u[j];
    }
}
__device__ __forceinline__ void ts_add(const Params &P, const double *v, double &acc, double &h) {
    acc = (acc + v[0]) + v[1];
    if (P.viscous) h = h + v[2];
}
// boundary edge binc[k]: v[0..3] the convective and acoustic terms of the
// node's side and of both, v[4..5] the viscous ones
__device__ __forceinline__ void ts_bterms(const Params &P, const LevelView &L, int k, double *v) {
    const int N = L.N;
    const double c1 = P.gamma;
    const int b = L.binc[k] >> 1, side = L.binc[k] & 1;
    const int2 nd = L.bedge[b];
    const double wx = L.bwx[b], wy = L.bwy[b], wz = L.bwz[b];
    const double al = (wx * wx + wy * wy) + wz * wz;
    const int j1 = nd.x, j2 = nd.y;
    const double ro1 = 1. / L.u[j1], ro2 = 1. / L.u[j2];
    double cc1 = dmax(c1 * L.p[j1] * ro1, 0.001);
    double cc2 = dmax(c1 * L.p[j2] * ro2, 0.001);
    double vn1 = ((wx * L.u[N + j1] + wy * L.u[2 * N + j1]) + wz * L.u[3 * N + j1]) * ro1;
    double vn2 = ((wx * L.u[N + j2] + wy * L.u[2 * N + j2]) + wz * L.u[3 * N + j2]) * ro2;
    vn1 = fabs(vn1); vn2 = fabs(vn2);
    cc1 = sqrt(cc1 * al); cc2 = sqrt(cc2 * al);
    v[0] = side == 0 ? vn1 : vn2;
    v[1] = vn1 + vn2;
    v[2] = side == 0 ? cc1 : cc2;
    v[3] = cc1 + cc2;
    if (P.viscous) {
        const double vis1 = dmax(P.am, P.sa ? L.mu[j1] + L.u[5 * N + j1] / P.Re : L.mu[j1]);
        const double vis2 = dmax(P.am, P.sa ? L.mu[j2] + L.u[5 * N + j2] / P.Re : L.mu[j2]);
        const double dv1 = 2.0 * vis1 * al / L.u[j1];
        const double dv2 = 2.0 * vis2 * al / L.u[j2];
        v[4] = side == 0 ? dv1 : dv2;
        v[5] = dv1 + dv2;
    } else {
        v[4] = v[5] = 0.0;
    }
}
__device__ __forceinline__ void ts_badd(const Params &P, const double *x, double &acc, double &h) {
    acc = (((acc + x[0]) + x[1]) + x[2]) + x[3];
    if (P.viscous) h = (h + x[4]) + x[5];
}
__device__ __forceinline__ void ts_store(const LevelView &L, int i, double acc, double h) {
    const double V = L.V[i];
    const double dt = 0.5 / (acc / V + h / (V * V));
    L.dt[i] = dt;
    L.vdt[i] = V / dt;  // V/dt of the dissipation coefficient d0
}
// the boundary edges of node i in order, then dt and V/dt
__device__ __forceinline__ void ts_finish(const Params &P, const LevelView &L, int i, double acc, double h) {
    for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
        double v[6];
        ts_bterms(P, L, k, v);
        ts_badd(P, v, acc, h);
    }
    ts_store(L, i, acc, h);
}

// node i's time step with U lanes (lane gl, the warp's slab gs of 8 terms)
template <int U>
__device__ __forceinline__ void ts_group(const Params &P, const LevelView &L, int i, bool active, int gl, double *gs,
                                         double m1, double m2, double m3, double ro, double cc) {
    const int N = L.N;
    // sum 0: the convective and acoustic terms; sum 1: the viscous ones
    double x[2] = {0.0, 0.0};
    group_sum<U, 2, 2, double>(
        gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
        [&](int k, double *v) { ts_terms(P, L, L.inc[k], m1, m2, m3, ro, cc, v); }, x);
    group_sum<U, 2, 4, double>(
        gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl, [&](int k, double *v) { ts_bterms(P, L, k, v); }, x);
    if (active && gl == 0) ts_store(L, i, x[0], x[1]);
}

template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 4 : 1) k_timestep(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    const double ro = 1. / L.u[i];
    const double m1 = L.u[N + i], m2 = L.u[2 * N + i], m3 = L.u[3 * N + i];
    const double cc = dmax(P.gamma * L.p[i] * ro, 0.001);
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 8);
        ts_group<U>(P, L, i, active, gl, gs, m1, m2, m3, ro, cc);
    } else {
        double acc = 0.0, h = 0.0;
        walk<2, 3>(
            L, i, [&](const int2 t, double *v) { ts_terms(P, L, t, m1, m2, m3, ro, cc, v); },
            [&](const double *v) { ts_add(P, v, acc, h); });
        ts_finish(P, L, i, acc, h);
    }
}

// ---- makeArtificialDissipation2, passes 1-2 and the node finish -----------
// (def_par:11513-11780): undivided Laplacian with dE+dp, pressure sensor
struct LapAcc {
    double l[5], s7, s8;
};
// interior edge t of node i (state ui, pressure pi)
__device__ __forceinline__ void lap_terms(const Params &P, const LevelView &L, int2 t, const double *ui, double pi,
                                          double *v) {
    const int N = L.N;
    const int j = t.y;
    double df = 1.0;
    if (P.useDissW) df = 1. / L.slen[t.x >= 0 ? t.x : ~t.x];
    const double uj[5] = {L.u[j], L.u[N + j], L.u[2 * N + j], L.u[3 * N + j], L.u[4 * N + j]};
    const double pj = L.p[j];
    // The edge's first node subtracts its differences d(i, j), the second adds
    // d(j, i): the same terms, as -(x - y) is y - x, up to the order of the
    // pressures in the last one (a zero's sign is lost in the sums)
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = (uj[c] - ui[c]) * df;
    const bool first = t.x >= 0;
    v[4] = (((uj[4] - ui[4]) + (first ? -pi : pj)) + (first ? pj : -pi)) * df;
    v[5] = pj - pi; v[6] = pj + pi;
}
__device__ __forceinline__ void lap_add(const double *v, LapAcc &a) {
#pragma unroll
    for (int c = 0; c < 5; ++c) a.l[c] = a.l[c] + v[c];
    a.s7 = a.s7 + v[5]; a.s8 = a.s8 + v[6];
}
__device__ __forceinline__ void lap_store(const LevelView &L, int i, const LapAcc &a) {
    const int N = L.N;
    const double fact = 1. / L.conn[i];
    L.sens[i] = 12. * fabs(a.s7 / a.s8);
#pragma unroll
    for (int c = 0; c < 5; ++c) L.lap[c * N + i] = fact * a.l[c];
}

// node i's Laplacian and sensor with U lanes (a slab of 7 terms)
template <int U>
__device__ __forceinline__ void lap_group(const Params &P, const LevelView &L, int i, bool active, int gl, double *gs,
                                          const double *ui, double pi) {
    double x[7] = {0, 0, 0, 0, 0, 0, 0};
    group_sum<U, 7, 1, double>(
        gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
        [&](int k, double *v) { lap_terms(P, L, L.inc[k], ui, pi, v); }, x);
    if (active && gl == 0) {
        const LapAcc a = {{x[0], x[1], x[2], x[3], x[4]}, x[5], x[6]};
        lap_store(L, i, a);
    }
}

template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 3 : 1) k_jst_lap(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    const double ui[5] = {L.u[i], L.u[N + i], L.u[2 * N + i], L.u[3 * N + i], L.u[4 * N + i]};
    const double pi = L.p[i];
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 7);
        lap_group<U>(P, L, i, active, gl, gs, ui, pi);
    } else {
        LapAcc a = {{0, 0, 0, 0, 0}, 0, 0};
        walk<2, 7>(
            L, i, [&](const int2 t, double *v) { lap_terms(P, L, t, ui, pi, v); },
            [&](const double *v) { lap_add(v, a); });
        lap_store(L, i, a);
    }
}

// ---- makeArtificialDissipation2, pass 3 (def_par:11770-11906), scalar -----
// interior edge t of node i (Laplacian Li, state Ui, V/dt vdi, connectivity
// coni, sensor si): the fourth- and second-order terms with the sign of
// this node
__device__ __forceinline__ void jflux_terms(const Params &P, const LevelView &L, const double *u, int2 t, double k4,
                                            double vdi, double coni, double si, const double *Li, const double *Ui,
                                            double *v) {
    const int N = L.N;
    const int j = t.y;
    const double vdj = L.vdt[j];
    const bool first = t.x >= 0;
    double d0 = first ? dmin(vdi, vdj) : dmin(vdj, vdi);
    d0 = d0 / (coni + L.conn[j]);
    const double sj = L.sens[j];
    const double d2 = d0 * P.k2 * (first ? dmax(si, sj) : dmax(sj, si));
    double d4 = d0 * k4;
    d4 = d4 > d2 ? d4 - d2 : 0.0;
    // acc - (Li - Lj) d4 + (Ui - Uj) d2 for the edge's first node, acc +
    // (Lj - Li) d4 - (Uj - Ui) d2 for its second: the same terms
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        v[2 * c] = (L.lap[c * N + j] - Li[c]) * d4;
        v[2 * c + 1] = (Ui[c] - u[c * N + j]) * d2;
    }
}
__device__ __forceinline__ void jflux_add(const double *v, double *acc) {
#pragma unroll
    for (int c = 0; c < 5; ++c) acc[c] = (acc[c] + v[2 * c]) + v[2 * c + 1];
}

// node i's scalar JST flux with U lanes (a slab of 10 terms) at the state u;
// every lane gets the sums
template <int U>
__device__ __forceinline__ void jflux_group(const Params &P, const LevelView &L, const double *u, int i, bool active,
                                            int gl, double *gs, double *acc) {
    const int N = L.N;
    const double k4 = L.grid == 1 ? P.k4 : P.cgdf;
    double Li[5], Ui[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) { acc[c] = 0.0; Li[c] = L.lap[c * N + i]; Ui[c] = u[c * N + i]; }
    const double vdi = L.vdt[i], coni = L.conn[i], si = L.sens[i];
    group_sum<U, 5, 2, double>(
        gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
        [&](int k, double *v) { jflux_terms(P, L, u, L.inc[k], k4, vdi, coni, si, Li, Ui, v); }, acc);
}

template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 2 : 1) k_jst_flux(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    double acc[5] = {0, 0, 0, 0, 0};
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 10);
        jflux_group<U>(P, L, L.u, i, active, gl, gs, acc);
        if (!active || gl) return;
    } else {
        const double k4 = L.grid == 1 ? P.k4 : P.cgdf;
        double Li[5], Ui[5];
        for (int c = 0; c < 5; ++c) { Li[c] = L.lap[c * N + i]; Ui[c] = L.u[c * N + i]; }
        const double vdi = L.vdt[i], coni = L.conn[i], si = L.sens[i];
        walk<2, 10>(
            L, i, [&](const int2 t, double *v) { jflux_terms(P, L, L.u, t, k4, vdi, coni, si, Li, Ui, v); },
            [&](const double *v) { jflux_add(v, acc); });
    }
    for (int c = 0; c < 5; ++c) L.diss[c * N + i] = acc[c];
}

// ---- makeArtificialDissipation2, pass 3, matrix variant (def_par:11814-
// 11898): the one-dimensional Roe matrix |A| along edge e (i1 -> i2), with
// Harten's correction, applied to the Laplacian and state differences
__device__ __forceinline__ void matrix_diss(const Params &P, const LevelView &L, int e, int i1, int i2,
                                            double *d4v, double *d2v) {
    const int N = L.N;
    const double H = P.harten;
    const double eps1 = 1. / dmax(H, 1.e-5), gam1 = P.gm1;
    double rnx = L.wx[e], rny = L.wy[e], rnz = L.wz[e];
    const double al = sqrt((rnx * rnx + rny * rny) + rnz * rnz);
    const double vmo1 = 1. / al;
    rnx = rnx * vmo1; rny = rny * vmo1; rnz = rnz * vmo1;
    const double rhol = L.u[i1];
    double rho1 = 1. / rhol;
    const double uxl = L.u[N + i1] * rho1, vyl = L.u[2 * N + i1] * rho1, wzl = L.u[3 * N + i1] * rho1;
    const double hl = (L.u[4 * N + i1] + L.p[i1]) * rho1;
    const double rhor = L.u[i2];
    rho1 = 1. / rhor;
    const double uxr = L.u[N + i2] * rho1, vyr = L.u[2 * N + i2] * rho1, wzr = L.u[3 * N + i2] * rho1;
    const double hr = (L.u[4 * N + i2] + L.p[i2]) * rho1;
    const double di = sqrt(rhor / rhol), d1 = 1.0 / (di + 1.0);
    const double ui = (di * uxr + uxl) * d1, vi = (di * vyr + vyl) * d1, wi = (di * wzr + wzl) * d1;
    const double hi = (di * hr + hl) * d1;
    const double ci2 = gam1 * (hi - 0.5 * ((ui * ui + vi * vi) + wi * wi));
    const double ci = sqrt(ci2);
    const double af = 0.5 * ((ui * ui + vi * vi) + wi * wi);
    const double ucp = (ui * rnx + vi * rny) + wi * rnz;
    double l1 = fabs(ucp + ci), l2 = fabs(ucp - ci), l3 = fabs(ucp);
    if (l1 < H) l1 = 0.5 * (l1 * l1 * eps1 + H);
    if (l2 < H) l2 = 0.5 * (l2 * l2 * eps1 + H);
    if (l3 < H) l3 = 0.5 * (l3 * l3 * eps1 + H);
    const double s1 = 0.5 * (l1 + l2), s2 = 0.5 * (l1 - l2);
    auto apply = [&](double *d) {
        const double al1x = gam1 * ((((af * d[0] - ui * d[1]) - vi * d[2]) - wi * d[3]) + d[4]);
        const double al2x = ((-ucp * d[0] + d[1] * rnx) + d[2] * rny) + d[3] * rnz;
        const double cc1 = ((s1 - l3) * al1x / ci2) + (s2 * al2x / ci);
        const double cc2 = (s2 * al1x / ci) + (s1 - l3) * al2x;
        d[0] = al * (l3 * d[0] + cc1);
        d[1] = al * ((l3 * d[1] + cc1 * ui) + cc2 * rnx);
        d[2] = al * ((l3 * d[2] + cc1 * vi) + cc2 * rny);
        d[3] = al * ((l3 * d[3] + cc1 * wi) + cc2 * rnz);
        d[4] = al * ((l3 * d[4] + cc1 * hi) + cc2 * ucp);
    };
    apply(d4v);
    apply(d2v);
}

// the matrix variant's pass 3 as a node gather in edge order; each edge's
// matrix terms are evaluated in the edge's own node order at both ends
__global__ void k_jst_flux_matrix(Params P, LevelView L) {
    const int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    const double k4 = L.grid == 1 ? P.k4 : P.cgdf;
    double acc[5] = {0, 0, 0, 0, 0};
    FLITE_FOR_INC(L, i, t) {
        const bool first = t.x >= 0;
        const int e = first ? t.x : ~t.x;
        const int i1 = first ? i : t.y, i2 = first ? t.y : i;
        double d4v[5], d2v[5];
        for (int c = 0; c < 5; ++c) {
            d4v[c] = L.lap[c * N + i1] - L.lap[c * N + i2];
            d2v[c] = L.u[c * N + i1] - L.u[c * N + i2];
        }
        matrix_diss(P, L, e, i1, i2, d4v, d2v);
        const double d2 = P.k2 * dmax(L.sens[i1], L.sens[i2]);
        const double d4 = k4 > d2 ? k4 - d2 : 0.0;
        for (int c = 0; c < 5; ++c)
            acc[c] = first ? (acc[c] - d4v[c] * d4) + d2v[c] * d2 : (acc[c] + d4v[c] * d4) - d2v[c] * d2;
    }
    for (int c = 0; c < 5; ++c) L.diss[c * N + i] = acc[c];
}

// ---- makeArtificialDissipation1 (def_par:10706-11482), level 1 -----------
// the linearity-preserving dissipation of Crumpton et al.  Pass 1, per node
// in edge order: the gradient sums of (rho, rho u, rho v, rho w, rho E), the
// undivided Laplacian L(U), the sum of the edge factors and L(x); then the
// boundary faces, the volume scaling, L^(U) = L(U) - (grad U).L(x) (L(x) = 0
// on boundary nodes) and the pressure sensor.  Writes L^ to lap, the sensor
// to sens and the factor sum to lpw.
__global__ void k_lp_sums(Params P, LevelView L) {
    const int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    double g[15], l[5], lx[3] = {0.0, 0.0, 0.0}, s21 = 0.0, pd = 0.0, ps = 0.0;
    for (int c = 0; c < 15; ++c) g[c] = 0.0;
    for (int c = 0; c < 5; ++c) l[c] = 0.0;
    FLITE_FOR_INC(L, i, t) {
        const bool first = t.x >= 0;
        const int e = first ? t.x : ~t.x;
        const int i1 = first ? i : t.y, i2 = first ? t.y : i;
        const EdgeW ew = load_edgew(L.ew, e);
        const double w[3] = {ew.wx, ew.wy, ew.wz};
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 5; ++c) {
                const double sv = (L.u[c * N + i1] + L.u[c * N + i2]) * w[a];
                g[5 * a + c] = first ? g[5 * a + c] + sv : g[5 * a + c] - sv;
            }
        double df = 1.0;
        if (P.useDissW) df = 1. / L.slen[e];
        for (int c = 0; c < 5; ++c) {
            const double d = L.u[c * N + i1] - L.u[c * N + i2];
            l[c] = first ? l[c] - d * df : l[c] + d * df;
        }
        s21 = s21 + df;
        const double dx[3] = {L.cx[i1] - L.cx[i2], L.cy[i1] - L.cy[i2], L.cz[i1] - L.cz[i2]};
        for (int a = 0; a < 3; ++a) lx[a] = first ? lx[a] - dx[a] * df : lx[a] + dx[a] * df;
        const double dp = L.p[i1] - L.p[i2], sp = L.p[i1] + L.p[i2];
        pd = first ? pd - dp : pd + dp;
        ps = ps + sp;
    }
    for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
        const int b = L.binc[k] >> 1, side = L.binc[k] & 1;
        const int2 nd = L.bedge[b];
        const double w[3] = {L.bwx[b], L.bwy[b], L.bwz[b]};
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 5; ++c) {
                const double q1 = L.u[c * N + nd.x], q2 = L.u[c * N + nd.y];
                double v;
                if (P.boundaryTerm == 1) v = side == 0 ? (3. * q1 + q2) * w[a] : (q1 + 3. * q2) * w[a];
                else v = side == 0 ? 4. * q1 * w[a] : 4. * w[a];  // the reference's second term has no state
                g[5 * a + c] = g[5 * a + c] + v;
            }
    }
    if (P.useDissW) s21 = 3.0 * s21;
    const double vt = 1. / L.V[i];
    for (int c = 0; c < 15; ++c) g[c] = g[c] * vt;
    if (i < L.Nb) lx[0] = lx[1] = lx[2] = 0.0;
    for (int c = 0; c < 5; ++c)
        L.lap[c * N + i] = ((l[c] + g[c] * lx[0]) + g[5 + c] * lx[1]) + g[10 + c] * lx[2];
    L.sens[i] = 12. * fabs(pd / ps);
    L.lpw[i] = s21;
}

// pass 2: the edge terms, as a node gather in edge order; under
// useMatrixDissipation the scalar coefficient divided by each end's factor
// sum, otherwise the Roe matrix (the reference's branch order)
__global__ void k_lp_flux(Params P, LevelView L) {
    const int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    double acc[5] = {0, 0, 0, 0, 0};
    FLITE_FOR_INC(L, i, t) {
        const bool first = t.x >= 0;
        const int e = first ? t.x : ~t.x;
        const int i1 = first ? i : t.y, i2 = first ? t.y : i;
        double d4v[5], d2v[5];
        for (int c = 0; c < 5; ++c) {
            d4v[c] = L.lap[c * N + i1] - L.lap[c * N + i2];
            d2v[c] = L.u[c * N + i1] - L.u[c * N + i2];
        }
        double d2, d4, d41, d42;
        if (P.matrixDiss) {
            const double d0 = dmin(L.vdt[i1], L.vdt[i2]) / (L.conn[i1] + L.conn[i2]);
            d2 = d0 * P.k2 * dmax(L.sens[i1], L.sens[i2]);
            d4 = d0 * P.k4;
            d4 = d4 > d2 ? d4 - d2 : 0.0;
            d41 = d4 / L.lpw[i1];
            d42 = d4 / L.lpw[i2];
        } else {
            matrix_diss(P, L, e, i1, i2, d4v, d2v);
            d2 = P.k2 * dmax(L.sens[i1], L.sens[i2]);
            d4 = P.k4;
            d4 = d4 > d2 ? d4 - d2 : 0.0;
            d41 = d42 = d4;
        }
        for (int c = 0; c < 5; ++c)
            acc[c] = first ? (acc[c] - d4v[c] * d41) + d2v[c] * d2 : (acc[c] + d4v[c] * d42) - d2v[c] * d2;
    }
    for (int c = 0; c < 5; ++c) L.diss[c * N + i] = acc[c];
}

// ---- makeArtificialDissipation3 (def_par:11995-12139) ---------------------
template <int U>
__global__ void k_first_order_diss(Params P, LevelView L) {
    int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    double acc[5] = {0, 0, 0, 0, 0};
    const double vdi = L.vdt[i], coni = L.conn[i];
    FLITE_FOR_INC(L, i, t) {
        int j = t.y;
        double vdj = L.vdt[j];
        const bool first = t.x >= 0;
        double d0 = first ? dmin(vdi, vdj) : dmin(vdj, vdi);
        d0 = d0 / (first ? (coni + L.conn[j]) : (L.conn[j] + coni));
        double d2 = d0 * P.cgdf;
        for (int c = 0; c < 5; ++c) {
            double dk = first ? L.u[c * N + i] - L.u[c * N + j] : L.u[c * N + j] - L.u[c * N + i];
            acc[c] = first ? acc[c] + dk * d2 : acc[c] - dk * d2;
        }
    }
    for (int c = 0; c < 5; ++c) L.diss[c * N + i] = acc[c];
}

// ---- makeViscosityTerm, wide stencil (def_par:5198-5893) ------------------
// pass 1: Galerkin gradients of (u, v, w, T), then per node the Sutherland
// viscosity (T^1.5 evaluated as T*sqrt(T)), the stress tensor and heat
// flux, the adiabatic-wall projection and the wall stress (level 1)
// the boundary-face terms of node i's Galerkin gradients of (u, v, w, T)
// (def_par:5322-5409), added to g in boundary-edge order
__device__ __forceinline__ void visc_grad_bterms(const LevelView &L, int k, double *d) {
    const int N = L.N;
    int b = L.binc[k] >> 1, side = L.binc[k] & 1;
    int2 nd = L.bedge[b];
    const double q1[4] = {L.prim[nd.x], L.prim[N + nd.x], L.prim[2 * N + nd.x], L.prim[3 * N + nd.x]};
    const double q2[4] = {L.prim[nd.y], L.prim[N + nd.y], L.prim[2 * N + nd.y], L.prim[3 * N + nd.y]};
    const double w[3] = {L.bwx[b], L.bwy[b], L.bwz[b]};
    for (int a = 0; a < 3; ++a)
        for (int c = 0; c < 4; ++c) {
            double sm = q1[c] + q2[c];
            double own = side == 0 ? q1[c] : q2[c];
            d[a * 4 + c] = (2. * own + sm) * w[a];
        }
}

// from node i's summed gradients g: Sutherland's viscosity, the SA eddy
// viscosity, vorticity and divergence, the stress tensor and heat flux, the
// adiabatic-wall projection and the wall stress (def_par:5460-5640)
__device__ __forceinline__ void visc_grad_finish(const Params &P, const LevelView &L, int i, const double *g) {
    const int N = L.N;
    const double gOg = P.gamma / (P.gamma - 1.0);
    const double vt = 1. / L.V[i];
    double dudx = g[0] * vt, dvdx = g[1] * vt, dwdx = g[2] * vt, dTdx = g[3] * vt;
    double dudy = g[4] * vt, dvdy = g[5] * vt, dwdy = g[6] * vt, dTdy = g[7] * vt;
    double dudz = g[8] * vt, dvdz = g[9] * vt, dwdz = g[10] * vt, dTdz = g[11] * vt;
    const double tempConv = (P.gamma - 1.0) * P.mach * P.mach;
    double T = gOg * L.p[i] / L.u[i];
    if (T <= 0.001) T = 0.001;
    double a = tempConv * T;
    double mu = (1. / P.Re) * ((a * sqrt(a)) * ((P.Tinf + 198.6) / (tempConv * P.Tinf * T + 198.6)));
    double kc = (1. / P.Pr) * mu;
    L.mu[i] = mu;
    if (P.sa) {
        const double a1 = dudy - dvdx, a2 = dvdz - dwdy, a3 = dwdx - dudz;
        L.vort[i] = sqrt((a1 * a1 + a2 * a2) + a3 * a3);
        L.divg[i] = (dudx + dvdy) + dwdz;
        // turbulent viscosity of the SA model (def_par:5556-5566)
        double tvc = (1. / P.Re) * L.u[i] * L.u[5 * N + i];
        const double ksi3 = flite_pm::pm_cube(tvc / mu);
        tvc = tvc * ksi3 / (ksi3 + 357.9);
        mu = mu + tvc;
        kc = kc + tvc * P.oPrt;
    }
    const double twoThirds = 2. / 3., fourThirds = 4. / 3.;
    double tau[9];
    tau[0] = mu * (fourThirds * dudx - twoThirds * (dvdy + dwdz));
    tau[1] = mu * (dudy + dvdx);
    tau[2] = mu * (dudz + dwdx);
    tau[3] = mu * (fourThirds * dvdy - twoThirds * (dudx + dwdz));
    tau[4] = mu * (dvdz + dwdy);
    tau[5] = mu * (fourThirds * dwdz - twoThirds * (dudx + dvdy));
    tau[6] = kc * dTdx;
    tau[7] = kc * dTdy;
    tau[8] = kc * dTdz;
    const unsigned char cls = L.bc[i];
    if (L.grid == 1 && cls != BC_NONE) {
        double n0 = L.nx[i], n1 = L.ny[i], n2 = L.nz[i];
        if (cls == BC_WALL) {  // setTemperatureForAdiabaticWall (def_par:5170-5196)
            double nt = (tau[6] * n0 + tau[7] * n1) + tau[8] * n2;
            tau[6] = tau[6] - nt * n0;
            tau[7] = tau[7] - nt * n1;
            tau[8] = tau[8] - nt * n2;
        }
        L.wstress[i] = (tau[0] * n0 + tau[1] * n1) + tau[2] * n2;
        L.wstress[N + i] = (tau[1] * n0 + tau[3] * n1) + tau[4] * n2;
        L.wstress[2 * N + i] = (tau[2] * n0 + tau[4] * n1) + tau[5] * n2;
    }
    for (int c = 0; c < 9; ++c) L.tau[c * N + i] = tau[c];
}

// interior edge t of node i (u, v, w, T of the node qi): the edge's terms
// of the 12 gradient sums, added with the sign of this node
__device__ __forceinline__ void vgrad_terms(const LevelView &L, int2 t, const double *qi, double *v) {
    const int N = L.N, e = t.x >= 0 ? t.x : ~t.x, j = t.y;
    const double qj[4] = {L.prim[j], L.prim[N + j], L.prim[2 * N + j], L.prim[3 * N + j]};
    const double w[3] = {L.wx[e], L.wy[e], L.wz[e]};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double ws = t.x >= 0 ? w[a] : -w[a];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[a * 4 + c] = (qi[c] + qj[c]) * ws;
    }
}
__device__ __forceinline__ void vgrad_add(const double *v, double *g) {
#pragma unroll
    for (int c = 0; c < 12; ++c) g[c] = g[c] + v[c];
}
// the boundary edges of node i in order
__device__ __forceinline__ void visc_grad_boundary(const LevelView &L, int i, double *g) {
    for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
        double v[12];
        visc_grad_bterms(L, k, v);
#pragma unroll
        for (int c = 0; c < 12; ++c) g[c] = g[c] + v[c];
    }
}

// node i's 12 gradient sums with U lanes (a slab of 12 terms), boundary
// edges included; every lane gets them
template <int U>
__device__ __forceinline__ void vgrad_group(const LevelView &L, int i, bool active, int gl, double *gs, double *g) {
    const int N = L.N;
    const double qi[4] = {L.prim[i], L.prim[N + i], L.prim[2 * N + i], L.prim[3 * N + i]};
#pragma unroll
    for (int c = 0; c < 12; ++c) g[c] = 0.0;
    group_sum<U, 12, 1, double>(
        gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
        [&](int k, double *v) { vgrad_terms(L, L.inc[k], qi, v); }, g);
    group_sum<U, 12, 1, double>(
        gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl, [&](int k, double *d) { visc_grad_bterms(L, k, d); }, g);
}

template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 2 : 1) k_visc_grad(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    double g[12];
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 12);
        vgrad_group<U>(L, i, active, gl, gs, g);
        if (!active || gl) return;
    } else {
        for (int c = 0; c < 12; ++c) g[c] = 0.0;
        const double qi[4] = {L.prim[i], L.prim[N + i], L.prim[2 * N + i], L.prim[3 * N + i]};
        walk<2, 12>(
            L, i, [&](const int2 t, double *v) { vgrad_terms(L, t, qi, v); },
            [&](const double *v) { vgrad_add(v, g); });
        visc_grad_boundary(L, i, g);
    }
    visc_grad_finish(P, L, i, g);
}

// the viscous flux of an edge from the stress/heat-flux and velocity of its
// first (a, ua) and second (b, ub) node (def_par:5688-5720)
__device__ __forceinline__ void visc_edge_flux(const double *a, const double *b, const double *ua, const double *ub,
                                               double wx, double wy, double wz, double *f) {
    double dt[9];
    for (int c = 0; c < 9; ++c) dt[c] = a[c] + b[c];
    double dut1 = ((((ua[0] * a[0] + ub[0] * b[0]) + ua[1] * a[1]) + ub[1] * b[1]) + ua[2] * a[2]) + ub[2] * b[2];
    double dut2 = ((((ua[0] * a[1] + ub[0] * b[1]) + ua[1] * a[3]) + ub[1] * b[3]) + ua[2] * a[4]) + ub[2] * b[4];
    double dut3 = ((((ua[0] * a[2] + ub[0] * b[2]) + ua[1] * a[4]) + ub[1] * b[4]) + ua[2] * a[5]) + ub[2] * b[5];
    f[0] = (wx * dt[0] + wy * dt[1]) + wz * dt[2];
    f[1] = (wx * dt[1] + wy * dt[3]) + wz * dt[4];
    f[2] = (wx * dt[2] + wy * dt[4]) + wz * dt[5];
    f[3] = (wx * (dt[6] + dut1) + wy * (dt[7] + dut2)) + wz * (dt[8] + dut3);
}

// the two terms of each component of boundary edge binc[k] for its node
// (def_par:5730-5800); g[8] = 0 for symmetry and inviscid-wall faces,
// which contribute nothing
__device__ __forceinline__ void visc_flux_bterms(const LevelView &L, int k, double *g) {
    const int N = L.N;
    int bb = L.binc[k] >> 1, side = L.binc[k] & 1;
    int ind = L.bind[bb];
    g[8] = (ind == 2 || ind == 9) ? 0.0 : 1.0;
    if (g[8] == 0.0) return;
    int2 nd = L.bedge[bb];
    double a[9], b[9], ua[3], ub[3];
    for (int c = 0; c < 9; ++c) { a[c] = L.tau[c * N + nd.x]; b[c] = L.tau[c * N + nd.y]; }
    ua[0] = L.prim[nd.x]; ua[1] = L.prim[N + nd.x]; ua[2] = L.prim[2 * N + nd.x];
    ub[0] = L.prim[nd.y]; ub[1] = L.prim[N + nd.y]; ub[2] = L.prim[2 * N + nd.y];
    const double wx = L.bwx[bb], wy = L.bwy[bb], wz = L.bwz[bb];
    double dt[9];
    for (int c = 0; c < 9; ++c) dt[c] = a[c] + b[c];
    double d11 = (ua[0] * a[0] + ua[1] * a[1]) + ua[2] * a[2];
    double d12 = (ub[0] * b[0] + ub[1] * b[1]) + ub[2] * b[2];
    double d21 = (ua[0] * a[1] + ua[1] * a[3]) + ua[2] * a[4];
    double d22 = (ub[0] * b[1] + ub[1] * b[3]) + ub[2] * b[4];
    double d31 = (ua[0] * a[2] + ua[1] * a[4]) + ua[2] * a[5];
    double d32 = (ub[0] * b[2] + ub[1] * b[4]) + ub[2] * b[5];
    double dut1 = d11 + d12, dut2 = d21 + d22, dut3 = d31 + d32;
    g[0] = (wx * dt[0] + wy * dt[1]) + wz * dt[2];
    g[1] = (wx * dt[1] + wy * dt[3]) + wz * dt[4];
    g[2] = (wx * dt[2] + wy * dt[4]) + wz * dt[5];
    g[3] = (wx * (dt[6] + dut1) + wy * (dt[7] + dut2)) + wz * (dt[8] + dut3);
    const double *o = side == 0 ? a : b;
    double do1 = side == 0 ? d11 : d12, do2 = side == 0 ? d21 : d22, do3 = side == 0 ? d31 : d32;
    g[4] = 2.0 * ((wx * o[0] + wy * o[1]) + wz * o[2]);
    g[5] = 2.0 * ((wx * o[1] + wy * o[3]) + wz * o[4]);
    g[6] = 2.0 * ((wx * o[2] + wy * o[4]) + wz * o[5]);
    g[7] = 2.0 * ((wx * (o[6] + do1) + wy * (o[7] + do2)) + wz * (o[8] + do3));
}

// node i's boundary-edge terms added to acc in boundary-edge order
__device__ __forceinline__ void visc_flux_boundary(const LevelView &L, int i, double *acc) {
    for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
        double v[9];
        visc_flux_bterms(L, k, v);
        if (v[8] == 0.0) continue;
        for (int c = 0; c < 4; ++c) acc[c] = (acc[c] + v[c]) + v[4 + c];
    }
}

// pass 2: viscous edge fluxes gathered per node and subtracted from the
// dissipation vector (def_par:5662-5892)
// interior edge t of node i (tensor ti, velocity ui): the edge flux with the
// sign of this node (x - y is x + (-y))
__device__ __forceinline__ void vflux_terms(const LevelView &L, const int2 t, const double *ti, const double *ui,
                                            double *g) {
    const int N = L.N, e = t.x >= 0 ? t.x : ~t.x, j = t.y;
    double tj[9], uj[3];
    for (int c = 0; c < 9; ++c) tj[c] = L.tau[c * N + j];
    uj[0] = L.prim[j]; uj[1] = L.prim[N + j]; uj[2] = L.prim[2 * N + j];
    const bool first = t.x >= 0;
    double f[4];
    visc_edge_flux(first ? ti : tj, first ? tj : ti, first ? ui : uj, first ? uj : ui, L.wx[e], L.wy[e], L.wz[e], f);
    for (int c = 0; c < 4; ++c) g[c] = first ? f[c] : -f[c];
}
// node i's viscous fluxes with U lanes (a slab of 8 terms); every lane gets
// the sums
template <int U>
__device__ __forceinline__ void vflux_group(const LevelView &L, int i, bool active, int gl, double *gs, double *acc) {
    const int N = L.N;
    double ti[9];
    for (int c = 0; c < 9; ++c) ti[c] = L.tau[c * N + i];
    const double ui[3] = {L.prim[i], L.prim[N + i], L.prim[2 * N + i]};
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c] = 0.0;
    group_sum<U, 4, 1, double>(
        gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
        [&](int k, double *v) { vflux_terms(L, L.inc[k], ti, ui, v); }, acc);
    // a face that does not count leaves zeros
    group_sum<U, 4, 2, double>(
        gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl,
        [&](int k, double *v) {
            double t[9];
            visc_flux_bterms(L, k, t);
            if (t[8] == 0.0) return;
#pragma unroll
            for (int c = 0; c < 4; ++c) { v[2 * c] = t[c]; v[2 * c + 1] = t[4 + c]; }
        },
        acc);
}

template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 2 : 1) k_visc_flux(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    double acc[4] = {0, 0, 0, 0};
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 8);
        vflux_group<U>(L, i, active, gl, gs, acc);
        if (!active || gl) return;
    } else {
        double ti[9];
        for (int c = 0; c < 9; ++c) ti[c] = L.tau[c * N + i];
        const double ui[3] = {L.prim[i], L.prim[N + i], L.prim[2 * N + i]};
        walk<2, 4>(
            L, i, [&](const int2 t, double *v) { vflux_terms(L, t, ti, ui, v); },
            [&](const double *v) {
                for (int c = 0; c < 4; ++c) acc[c] = acc[c] + v[c];
            });
        visc_flux_boundary(L, i, acc);
    }
    for (int c = 0; c < 4; ++c) L.diss[(1 + c) * N + i] = L.diss[(1 + c) * N + i] - acc[c];
}

// ---- fused walks of one incidence list --------------------------------------
// Gathers that read the same neighbours and write disjoint arrays share one
// walk of the node's incidence list: the incidences, their edges and the
// neighbours' state are read once for both.  Each sum keeps its own
// accumulators and its own order, so the results are those of the separate
// kernels bit for bit.
//
// makeTimeSteps with passes 1-2 of makeArtificialDissipation2: the time
// step reads mu of the neighbours (the previous viscous pass) and writes dt
// and V/dt; the Laplacian reads u and p and writes the Laplacian and sensor
template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 3 : 1) k_ts_lap(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;
    const int N = L.N;
    const double ui[5] = {L.u[i], L.u[N + i], L.u[2 * N + i], L.u[3 * N + i], L.u[4 * N + i]};
    const double pi = L.p[i];
    const double ro = 1. / ui[0];
    const double cc = dmax(P.gamma * pi * ro, 0.001);
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 8);
        lap_group<U>(P, L, i, active, gl, gs, ui, pi);
        ts_group<U>(P, L, i, active, gl, gs, ui[1], ui[2], ui[3], ro, cc);
    } else {
        double acc = 0.0, h = 0.0;
        LapAcc a = {{0, 0, 0, 0, 0}, 0, 0};
        walk<1, 10>(
            L, i,
            [&](const int2 t, double *v) {
                ts_terms(P, L, t, ui[1], ui[2], ui[3], ro, cc, v);
                lap_terms(P, L, t, ui, pi, v + 3);
            },
            [&](const double *v) {
                ts_add(P, v, acc, h);
                lap_add(v + 3, a);
            });
        lap_store(L, i, a);
        ts_finish(P, L, i, acc, h);
    }
}

// pass 3 of makeArtificialDissipation2 (scalar) with pass 1 of
// makeViscosityTerm: the JST terms read the Laplacian, sensor, V/dt and u of
// the neighbours and write the dissipation; the gradients read u, v, w, T
// and write mu, the stress tensor and the wall stress
template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 2 : 1) k_jflux_vgrad(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;
    const int N = L.N;
    double g[12];
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 12);
        double acc[5];
        jflux_group<U>(P, L, L.u, i, active, gl, gs, acc);
        if (active && gl == 0)
            for (int c = 0; c < 5; ++c) L.diss[c * N + i] = acc[c];
        vgrad_group<U>(L, i, active, gl, gs, g);
        if (!active || gl) return;
    } else {
        const double k4 = L.grid == 1 ? P.k4 : P.cgdf;
        double acc[5] = {0, 0, 0, 0, 0};
        double Li[5], Ui[5];
        for (int c = 0; c < 5; ++c) { Li[c] = L.lap[c * N + i]; Ui[c] = L.u[c * N + i]; }
        const double vdi = L.vdt[i], coni = L.conn[i], si = L.sens[i];
        const double qi[4] = {L.prim[i], L.prim[N + i], L.prim[2 * N + i], L.prim[3 * N + i]};
        for (int c = 0; c < 12; ++c) g[c] = 0.0;
        walk<1, 22>(
            L, i,
            [&](const int2 t, double *v) {
                jflux_terms(P, L, L.u, t, k4, vdi, coni, si, Li, Ui, v);
                vgrad_terms(L, t, qi, v + 10);
            },
            [&](const double *v) {
                jflux_add(v, acc);
                vgrad_add(v + 10, g);
            });
        for (int c = 0; c < 5; ++c) L.diss[c * N + i] = acc[c];
        visc_grad_boundary(L, i, g);
    }
    visc_grad_finish(P, L, i, g);
}

// ---- makeViscosityTerm2, the compact stencil (def_par:5896-6807) ---------
// pass 1: the Galerkin gradients of (u, v, w, T) as in k_visc_grad (with the
// FV boundary form under boundaryTerm 2), then per node the viscosity and
// the gradients scaled by mu (velocity) and k (temperature), stored with mu
// and k as tau[14][N]; the adiabatic-wall projection and the wall stress of
// the wall nodes on level 1; zero temperature gradients on every boundary
// node of isentropic (adiabatic) walls
__device__ __forceinline__ void visc2_grad_finish(const Params &P, const LevelView &L, int i, const double *g) {
    const int N = L.N;
    const double gOg = P.gamma / (P.gamma - 1.0);
    const double vt = 1. / L.V[i];
    double gs[12];
    for (int c = 0; c < 12; ++c) gs[c] = g[c] * vt;
    const double dudx = gs[0], dvdx = gs[1], dwdx = gs[2];
    const double dudy = gs[4], dvdy = gs[5], dwdy = gs[6];
    const double dudz = gs[8], dvdz = gs[9], dwdz = gs[10];
    const double tempConv = (P.gamma - 1.0) * P.mach * P.mach;
    double T = gOg * L.p[i] / L.u[i];
    if (T <= 0.001) T = 0.001;
    double a = tempConv * T;
    double mu = (1. / P.Re) * ((a * sqrt(a)) * ((P.Tinf + 198.6) / (tempConv * P.Tinf * T + 198.6)));
    double kc = (1. / P.Pr) * mu;
    L.mu[i] = mu;
    if (P.sa) {
        const double a1 = dudy - dvdx, a2 = dvdz - dwdy, a3 = dwdx - dudz;
        L.vort[i] = sqrt((a1 * a1 + a2 * a2) + a3 * a3);
        L.divg[i] = (dudx + dvdy) + dwdz;
        double tvc = (1. / P.Re) * L.u[i] * L.u[5 * N + i];
        const double ksi3 = flite_pm::pm_cube(tvc / mu);
        tvc = tvc * ksi3 / (ksi3 + 357.9);
        mu = mu + tvc;
        kc = kc + tvc * P.oPrt;
    }
#pragma unroll
    for (int q = 0; q < 12; ++q) gs[q] = ((q & 3) == 3 ? kc : mu) * gs[q];
    const unsigned char cls = L.bc[i];
    if (L.grid == 1 && cls == BC_WALL) {
        const double n0 = L.nx[i], n1 = L.ny[i], n2 = L.nz[i];
        const double nt = (gs[3] * n0 + gs[7] * n1) + gs[11] * n2;
        gs[3] = gs[3] - nt * n0;
        gs[7] = gs[7] - nt * n1;
        gs[11] = gs[11] - nt * n2;
        const double twoThirds = 2. / 3., fourThirds = 4. / 3.;
        const double c1 = fourThirds * gs[0] - twoThirds * (gs[5] + gs[10]), c2 = gs[4] + gs[1];
        const double c3 = gs[8] + gs[2], c4 = fourThirds * gs[5] - twoThirds * (gs[0] + gs[10]);
        const double c5 = gs[9] + gs[6], c6 = fourThirds * gs[10] - twoThirds * (gs[0] + gs[5]);
        L.wstress[i] = (c1 * n0 + c2 * n1) + c3 * n2;
        L.wstress[N + i] = (c2 * n0 + c4 * n1) + c5 * n2;
        L.wstress[2 * N + i] = (c3 * n0 + c5 * n1) + c6 * n2;
    }
    if (P.isentropic && i < L.Nb) gs[3] = gs[7] = gs[11] = 0.0;
    for (int q = 0; q < 12; ++q) L.tau[q * N + i] = gs[q];
    L.tau[12 * N + i] = mu;
    L.tau[13 * N + i] = kc;
}

template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 3 : 1) k_visc2_grad(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    double g[12];
    for (int c = 0; c < 12; ++c) g[c] = 0.0;
    auto prim = [&](int j, double *q) {
        q[0] = L.prim[j]; q[1] = L.prim[N + j]; q[2] = L.prim[2 * N + j]; q[3] = L.prim[3 * N + j];
    };
    double qi[4];
    prim(i, qi);
    auto iterms = [&](const int2 t, double *d) {
        int e = t.x >= 0 ? t.x : ~t.x;
        double qj[4];
        prim(t.y, qj);
        const double w[3] = {L.wx[e], L.wy[e], L.wz[e]};
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 4; ++c) {
                double x = (t.x >= 0 ? qi[c] + qj[c] : qj[c] + qi[c]) * w[a];
                d[a * 4 + c] = t.x >= 0 ? x : -x;
            }
    };
    auto bterms = [&](int k, double *d) {
        if (P.boundaryTerm == 1) {
            visc_grad_bterms(L, k, d);
            return;
        }
        // boundaryTerm 2: 4 q w_b of the node itself (def_par:6113-6138)
        const int b = L.binc[k] >> 1, side = L.binc[k] & 1;
        const int2 nd = L.bedge[b];
        const int j = side == 0 ? nd.x : nd.y;
        double q[4];
        prim(j, q);
        const double w[3] = {L.bwx[b], L.bwy[b], L.bwz[b]};
        for (int a = 0; a < 3; ++a)
            for (int c = 0; c < 4; ++c) d[a * 4 + c] = 4. * q[c] * w[a];
    };
    auto add = [&](const double *d) {
        for (int c = 0; c < 12; ++c) g[c] = g[c] + d[c];
    };
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 12);
        group_sum<U, 12, 1, double>(gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
                                         [&](int k, double *v) { iterms(L.inc[k], v); }, g);
        group_sum<U, 12, 1, double>(gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl, bterms, g);
        if (!active || gl) return;
    } else {
        FLITE_FOR_INC(L, i, t) {
            double v[12];
            iterms(t, v);
            add(v);
        }
        for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
            double v[12];
            bterms(k, v);
            add(v);
        }
    }
    visc2_grad_finish(P, L, i, g);
}

// node j's data of the compact flux: scaled gradients (12), mu, k,
// velocity and temperature (from 1/rho as the routine forms them) and
// coordinates (zero on coarse levels)
struct Visc2Node {
    double G[12], mu, k, v[4], x[3];
};
__device__ __forceinline__ void load_visc2(const Params &P, const LevelView &L, int j, Visc2Node &o) {
    const int N = L.N;
    for (int q = 0; q < 12; ++q) o.G[q] = L.tau[q * N + j];
    o.mu = L.tau[12 * N + j];
    o.k = L.tau[13 * N + j];
    const double ri = 1.0 / L.u[j];
    o.v[0] = L.u[N + j] * ri; o.v[1] = L.u[2 * N + j] * ri; o.v[2] = L.u[3 * N + j] * ri;
    o.v[3] = (P.gamma / (P.gamma - 1.0)) * L.p[j] * ri;
    o.x[0] = L.cx[j]; o.x[1] = L.cy[j]; o.x[2] = L.cz[j];
}

// the compact flux of an edge from its first (a) and second (b) node
// (def_par:6432-6556)
__device__ __forceinline__ void visc2_edge_flux(const Visc2Node &a, const Visc2Node &b, double slen, double wx,
                                                double wy, double wz, double *f) {
    const double twoThirds = 2. / 3., fourThirds = 4. / 3.;
    const double inv = 1.0 / slen;
    const double r[3] = {(b.x[0] - a.x[0]) * inv, (b.x[1] - a.x[1]) * inv, (b.x[2] - a.x[2]) * inv};
    double G[4][3];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int d = 0; d < 3; ++d) G[q][d] = a.G[d * 4 + q] + b.G[d * 4 + q];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double dr = (G[q][0] * r[0] + G[q][1] * r[1]) + G[q][2] * r[2];
#pragma unroll
        for (int d = 0; d < 3; ++d) G[q][d] = G[q][d] - dr * r[d];
        const double cf = q < 3 ? a.mu + b.mu : a.k + b.k;
        const double dq = cf * (b.v[q] - a.v[q]) * inv;
#pragma unroll
        for (int d = 0; d < 3; ++d) G[q][d] = G[q][d] + dq * r[d];
    }
    const double dt1 = fourThirds * G[0][0] - twoThirds * (G[1][1] + G[2][2]), dt2 = G[0][1] + G[1][0];
    const double dt3 = G[0][2] + G[2][0], dt4 = fourThirds * G[1][1] - twoThirds * (G[0][0] + G[2][2]);
    const double dt5 = G[1][2] + G[2][1], dt6 = fourThirds * G[2][2] - twoThirds * (G[0][0] + G[1][1]);
    const double dt7 = G[3][0], dt8 = G[3][1], dt9 = G[3][2];
    const double au = 0.5 * (a.v[0] + b.v[0]), av = 0.5 * (a.v[1] + b.v[1]), aw = 0.5 * (a.v[2] + b.v[2]);
    const double dut1 = (au * dt1 + av * dt2) + aw * dt3;
    const double dut2 = (au * dt2 + av * dt4) + aw * dt5;
    const double dut3 = (au * dt3 + av * dt5) + aw * dt6;
    f[0] = (wx * dt1 + wy * dt2) + wz * dt3;
    f[1] = (wx * dt2 + wy * dt4) + wz * dt5;
    f[2] = (wx * dt3 + wy * dt5) + wz * dt6;
    f[3] = (wx * (dt7 + dut1) + wy * (dt8 + dut2)) + wz * (dt9 + dut3);
}

// pass 2: the compact edge fluxes and the boundary faces' 4 w_b times each
// node's own stress, gathered per node and subtracted from the dissipation
template <int U, bool B>
__global__ void __launch_bounds__(256, U == 1 ? 2 : 1) k_visc2_flux(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    const int N = L.N;
    Visc2Node me;
    load_visc2(P, L, i, me);
    double acc[4] = {0, 0, 0, 0};
    auto iterms = [&](const int2 t, double *g) {
        const int e = t.x >= 0 ? t.x : ~t.x;
        Visc2Node nb;
        load_visc2(P, L, t.y, nb);
        double f[4];
        if (t.x >= 0) visc2_edge_flux(me, nb, L.slen[e], L.wx[e], L.wy[e], L.wz[e], f);
        else visc2_edge_flux(nb, me, L.slen[e], L.wx[e], L.wy[e], L.wz[e], f);
        for (int c = 0; c < 4; ++c) g[c] = t.x >= 0 ? f[c] : -f[c];
    };
    // a boundary face of this node: g[4] = 1 when it counts (not symmetry or
    // inviscid wall)
    auto bterms = [&](int k, double *g) {
        const int bb = L.binc[k] >> 1;
        const int ind = L.bind[bb];
        g[4] = (ind == 2 || ind == 9) ? 0.0 : 1.0;
        if (g[4] == 0.0) return;
        const double twoThirds = 2. / 3., fourThirds = 4. / 3.;
        const double wx = L.bwx[bb], wy = L.bwy[bb], wz = L.bwz[bb];
        const double *G = me.G;
        const double t1 = fourThirds * G[0] - twoThirds * (G[5] + G[10]), t2 = G[4] + G[1], t3 = G[8] + G[2];
        const double t4 = fourThirds * G[5] - twoThirds * (G[0] + G[10]), t5 = G[9] + G[6];
        const double t6 = fourThirds * G[10] - twoThirds * (G[0] + G[5]);
        double t7 = G[3], t8 = G[7], t9 = G[11];
        if (P.isentropic) t7 = t8 = t9 = 0.0;
        const double *v = me.v;
        const double d1 = (v[0] * t1 + v[1] * t2) + v[2] * t3;
        const double d2 = (v[0] * t2 + v[1] * t4) + v[2] * t5;
        const double d3 = (v[0] * t3 + v[1] * t5) + v[2] * t6;
        g[0] = 4.0 * ((wx * t1 + wy * t2) + wz * t3);
        g[1] = 4.0 * ((wx * t2 + wy * t4) + wz * t5);
        g[2] = 4.0 * ((wx * t3 + wy * t5) + wz * t6);
        g[3] = 4.0 * ((wx * (t7 + d1) + wy * (t8 + d2)) + wz * (t9 + d3));
    };
    auto iadd = [&](const double *g) {
        for (int c = 0; c < 4; ++c) acc[c] = acc[c] + g[c];
    };
    auto badd = [&](const double *g) {
        if (g[4] == 0.0) return;
        for (int c = 0; c < 4; ++c) acc[c] = acc[c] + g[c];
    };
    if constexpr (U > 1) {
        FLITE_GROUP_SLAB(double, 4);
        group_sum<U, 4, 1, double>(gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
                                        [&](int k, double *v) { iterms(L.inc[k], v); }, acc);
        group_sum<U, 4, 1, double>(
            gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl,
            [&](int k, double *v) {
                double t[5];
                bterms(k, t);
                if (t[4] == 0.0) return;
#pragma unroll
                for (int c = 0; c < 4; ++c) v[c] = t[c];
            },
            acc);
        if (!active || gl) return;
    } else {
        FLITE_FOR_INC(L, i, t) {
            double v[4];
            iterms(t, v);
            iadd(v);
        }
        for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
            double v[5];
            bterms(k, v);
            badd(v);
        }
    }
    for (int c = 0; c < 4; ++c) L.diss[(1 + c) * N + i] = L.diss[(1 + c) * N + i] - acc[c];
}

__global__ void k_fill(double *a, size_t n, double v) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}

// ---- computeGradient, Galerkin (def_par:2923-3245), and LocalMinMax --------
// (def_par:3248-3459) in one walk of the incidences (MINMAX; alone without
// automatic clipping).  Both read (rho, u, v, w, rho E) of the other node,
// with the quotients formed once per node (hprim) and not per incidence.
__device__ __forceinline__ void hllc_prim(const LevelView &L, int j, double *q) {
    const int N = L.N;
    q[0] = L.u[j]; q[1] = L.hprim[j]; q[2] = L.hprim[N + j]; q[3] = L.hprim[2 * N + j]; q[4] = L.u[4 * N + j];
}
template <bool MINMAX>
__global__ void __launch_bounds__(256) k_gradient(Params P, LevelView L) {
    const int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    double g[15], mn[5], mx[5];
#pragma unroll
    for (int c = 0; c < 15; ++c) g[c] = 0.0;
#pragma unroll
    for (int c = 0; c < 5; ++c) { mn[c] = 1.0e15; mx[c] = 1.0e15; }
    double qi[5];
    hllc_prim(L, i, qi);
    walk<2, 9>(L, i, [&](const int2 t, double *v) {
        const int e = t.x >= 0 ? t.x : ~t.x;
        hllc_prim(L, t.y, v);
        const double w[3] = {L.wx[e], L.wy[e], L.wz[e]};
        for (int a = 0; a < 3; ++a) v[5 + a] = t.x >= 0 ? w[a] : -w[a];
        v[8] = t.x >= 0 ? 1.0 : 0.0;
    }, [&](const double *v) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 5; ++c) g[a * 5 + c] = g[a * 5 + c] + (qi[c] + v[c]) * v[5 + a];
        if (MINMAX) {
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const double a = v[8] != 0.0 ? qi[c] : v[c], b = v[8] != 0.0 ? v[c] : qi[c];
                mn[c] = dmin(mn[c], dmin(a, b));
                mx[c] = dmin(mx[c], dmin(-a, -b));
            }
        }
    });
    for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
        const int b = L.binc[k] >> 1, side = L.binc[k] & 1;
        const int2 nd = L.bedge[b];
        double q1[5], q2[5];
        hllc_prim(L, nd.x, q1);
        hllc_prim(L, nd.y, q2);
        const double w[3] = {L.bwx[b], L.bwy[b], L.bwz[b]};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const double s = q1[c] + q2[c];
                const double own = side == 0 ? q1[c] : q2[c];
                g[a * 5 + c] = g[a * 5 + c] + (2. * own + s) * w[a];
            }
    }
    const double vt = 1. / L.V[i];
#pragma unroll
    for (int c = 0; c < 15; ++c) L.grad[c * N + i] = g[c] * vt;
    if (MINMAX) {
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            L.bnd[c * N + i] = mn[c] - qi[c];
            L.bnd[(c + 5) * N + i] = -mx[c] - qi[c];
        }
    }
}
template __global__ void k_gradient<false>(Params, LevelView);
template __global__ void k_gradient<true>(Params, LevelView);

// ---- the upwind extension's level-1 records (no reference counterpart) ----
// primitives (rho, (rho u)/rho, ..., rho E) and coordinates of every node
__global__ void k_prim_rec(LevelView L) {
    int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    const double r = L.u[i];
    PrimRec o;
    o.r = r; o.u = L.u[N + i] / r; o.v = L.u[2 * N + i] / r; o.w = L.u[3 * N + i] / r; o.E = L.u[4 * N + i];
    o.x = L.cx[i]; o.y = L.cy[i]; o.z = L.cz[i];
    store_pairs<PrimRec, 4>(L.qp, N, i, o);
}
// the Galerkin gradient of k_gradient (computeGradient, def_par:2923-3245),
// in the same summation order, from the primitive records, stored as
// component-major records
__global__ void __launch_bounds__(256) k_gradient_rec(LevelView L) {
    int i = tid();
    if (i >= L.N) return;
    double g[15];
#pragma unroll
    for (int c = 0; c < 15; ++c) g[c] = 0.0;
    const PrimRec Qi = load_prim(L.qp, L.N, i);
    const double qi[5] = {Qi.r, Qi.u, Qi.v, Qi.w, Qi.E};
    walk<3, 8>(L, i, [&](const int2 t, double *v) {
        const int e = t.x >= 0 ? t.x : ~t.x;
        const double2 a0 = __ldg(L.qp + t.y), a1 = __ldg(L.qp + L.N + t.y);
        v[0] = a0.x; v[1] = a0.y; v[2] = a1.x; v[3] = a1.y; v[4] = __ldg(&(L.qp + 2 * (size_t)L.N + t.y)->x);
        const double w[3] = {L.wx[e], L.wy[e], L.wz[e]};
        for (int a = 0; a < 3; ++a) v[5 + a] = t.x >= 0 ? w[a] : -w[a];
    }, [&](const double *v) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 5; ++c) g[a * 5 + c] = g[a * 5 + c] + (qi[c] + v[c]) * v[5 + a];
    });
    for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
        const int b = L.binc[k] >> 1, side = L.binc[k] & 1;
        const int2 nd = L.bedge[b];
        const PrimRec Q1 = load_prim(L.qp, L.N, nd.x), Q2 = load_prim(L.qp, L.N, nd.y);
        const double q1[5] = {Q1.r, Q1.u, Q1.v, Q1.w, Q1.E}, q2[5] = {Q2.r, Q2.u, Q2.v, Q2.w, Q2.E};
        const double w[3] = {L.bwx[b], L.bwy[b], L.bwz[b]};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const double sum = q1[c] + q2[c];
                const double own = side == 0 ? q1[c] : q2[c];
                g[a * 5 + c] = g[a * 5 + c] + (2. * own + sum) * w[a];
            }
    }
    const double vt = 1. / L.V[i];
    GradRec o;
#pragma unroll
    for (int c = 0; c < 5; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a) o.g[3 * c + a] = g[a * 5 + c] * vt;
    o.g[15] = 0.0;
    store_pairs<GradRec, 8>(L.gq, L.N, i, o);
}

// ---- LSComputeGradient + computegradhat (def_par:2593-2920) ---------------
// the moment matrix is the same for the five scalars and is built once; the
// right-hand sides of the five scalars are gathered in the same edge order
__global__ void k_ls_gradient(Params P, LevelView L) {
    int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    double m[6] = {0, 0, 0, 0, 0, 0}, b[5][3];
    for (int sc = 0; sc < 5; ++sc) b[sc][0] = b[sc][1] = b[sc][2] = 0.0;
    const double ri = L.u[i];
    const double qi[5] = {ri, L.u[N + i] / ri, L.u[2 * N + i] / ri, L.u[3 * N + i] / ri, L.u[4 * N + i]};
    FLITE_FOR_INC(L, i, t) {
        int j = t.y;
        const bool first = t.x >= 0;
        const int i1 = first ? i : j, i2 = first ? j : i;
        double dx = L.cx[i2] - L.cx[i1], dy = L.cy[i2] - L.cy[i1], dz = L.cz[i2] - L.cz[i1];
        double dist1 = 1. / ((dx * dx + dy * dy) + dz * dz);
        m[0] = m[0] + dx * dx * dist1; m[1] = m[1] + dx * dy * dist1; m[2] = m[2] + dx * dz * dist1;
        m[3] = m[3] + dy * dy * dist1; m[4] = m[4] + dy * dz * dist1; m[5] = m[5] + dz * dz * dist1;
        const double rj = L.u[j];
        const double qj[5] = {rj, L.u[N + j] / rj, L.u[2 * N + j] / rj, L.u[3 * N + j] / rj, L.u[4 * N + j]};
        for (int sc = 0; sc < 5; ++sc) {
            double dr2 = first ? qj[sc] - qi[sc] : qi[sc] - qj[sc];  // q(i2) - q(i1)
            b[sc][0] = b[sc][0] + dr2 * dx * dist1;
            b[sc][1] = b[sc][1] + dr2 * dy * dist1;
            b[sc][2] = b[sc][2] + dr2 * dz * dist1;
        }
    }
    double a11 = m[0], a12 = m[1], a13 = m[2], a21 = m[1], a22 = m[3], a23 = m[4], a31 = m[2], a32 = m[4], a33 = m[5];
    double c11 = a22 * a33 - a23 * a32, c21 = a23 * a31 - a21 * a33, c31 = a21 * a32 - a22 * a31;
    double det = (a11 * c11 + a12 * c21) + a13 * c31;
    if (fabs(det) > 0.0) det = 1.0 / det;
    c11 = det * c11; c21 = det * c21; c31 = det * c31;
    double c12 = det * (a13 * a32 - a12 * a33), c22 = det * (a11 * a33 - a13 * a31);
    double c32 = det * (a12 * a31 - a11 * a32), c13 = det * (a12 * a23 - a13 * a22);
    double c23 = det * (a13 * a21 - a23 * a11), c33 = det * (a11 * a22 - a12 * a21);
    for (int sc = 0; sc < 5; ++sc) {
        double b1 = b[sc][0], b2 = b[sc][1], b3 = b[sc][2];
        L.grad[sc * N + i] = (c11 * b1 + c12 * b2) + c13 * b3;
        L.grad[(5 + sc) * N + i] = (c21 * b1 + c22 * b2) + c23 * b3;
        L.grad[(10 + sc) * N + i] = (c31 * b1 + c32 * b2) + c33 * b3;
    }
}

// ---- LocalMinMax (def_par:3248-3459) beside least-squares gradients ---------------------------------------
__global__ void k_minmax(Params P, LevelView L) {
    int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    double mn[5], mx[5];
    for (int c = 0; c < 5; ++c) { mn[c] = 1.0e15; mx[c] = 1.0e15; }
    double qi[5];
    hllc_prim(L, i, qi);
    FLITE_FOR_INC(L, i, t) {
        double qj[5];
        hllc_prim(L, t.y, qj);
        // amin1(q(i1), q(i2)) with the edge's own node order
        for (int c = 0; c < 5; ++c) {
            double a = t.x >= 0 ? qi[c] : qj[c], b = t.x >= 0 ? qj[c] : qi[c];
            mn[c] = dmin(mn[c], dmin(a, b));
            mx[c] = dmin(mx[c], dmin(-a, -b));
        }
    }
    for (int c = 0; c < 5; ++c) {
        L.bnd[c * N + i] = mn[c] - qi[c];
        L.bnd[(c + 5) * N + i] = -mx[c] - qi[c];
    }
}

// ---- interior edge flux into the edge buffer ------------------------------
// What bounds the HLLC order-2 kernel: the chains of dependent FP64
// instructions (two limited, clipped reconstructions, some twenty divisions
// and fifteen square roots an edge: 2,850 thread instructions) and the loads
// between them, not a rate (on 5,094,100 edges 0.87 ms with 46 % of the issue
// slots, 28 % of the FP64 pipe, 35 % of L1 and 10 % of DRAM in use at 43 % of
// the warps; 1.25 ms and 3,800 instructions with two-sided branches).  The
// limiter's and the wave regions' branches run once instead of per side, in 7
// blocks of 128 threads (72 registers; the spills cost less than 2 blocks of
// 256 at 128 registers): the RANS cycle on 738,100 nodes 12.2 -> 9.8 ms (10.5
// with the 128 registers), the HLLC cycle on 80,640 nodes 1.63 -> 1.17 ms.
// The other fluxes take three blocks of 256 (80 registers, 48 to 76 bytes of
// spills in Roe and HLLC order 1) for the loads in flight: 815,425 nodes with
// three blocks and without a bound (106 to 150 registers), us: central (moving
// meshes) 126 and 164, LLF 140 and 140, Roe 173 and 222, HLLC order 1 215 and
// 276; 14,161 nodes 8.7 and 9.0, 9.1 and 9.2, 9.6 and 11.0, 10.9 and 11.5.
// The block's fluxes (at most 256 x 5) are staged in shared memory and
// written as one contiguous run of 16-byte stores; the block size is even,
// so the run starts on a 16-byte boundary.
__device__ __forceinline__ void store_block_fluxes(double *flux, const double *sf, int e0, int count) {
    const int n = 5 * count;
    double2 *o = reinterpret_cast<double2 *>(flux + (size_t)e0 * 5);
    const double2 *src = reinterpret_cast<const double2 *>(sf);
    for (int k = threadIdx.x; k < n / 2; k += blockDim.x) o[k] = src[k];
    if ((n & 1) && threadIdx.x == 0) flux[(size_t)e0 * 5 + n - 1] = sf[n - 1];
}
template <int FT, bool O2>
__global__ void __launch_bounds__(edge_threads(FT, O2), FT == 4 && O2 ? 7 : 3) k_edge_flux(Params P, LevelView L) {
    __shared__ __align__(16) double sf[256 * 5];
    const int e0 = blockIdx.x * blockDim.x, e = e0 + threadIdx.x;
    if (e < L.E) {
        const int2 nd = L.edge[e];
        double f[5];
        edge_flux<FT, O2>(P, L, e, nd.x, nd.y, f);
#pragma unroll
        for (int k = 0; k < 5; ++k) sf[threadIdx.x * 5 + k] = f[k];
    }
    __syncthreads();
    store_block_fluxes(L.flux, sf, e0, min((int)blockDim.x, L.E - e0));
}
template __global__ void k_edge_flux<1, false>(Params, LevelView);
template __global__ void k_edge_flux<2, false>(Params, LevelView);
template __global__ void k_edge_flux<3, false>(Params, LevelView);
template __global__ void k_edge_flux<3, true>(Params, LevelView);
template __global__ void k_edge_flux<4, false>(Params, LevelView);
template __global__ void k_edge_flux<4, true>(Params, LevelView);

// the upwind extension's level-1 edge flux into the edge buffer, stored as
// k_edge_flux stores.  Bound by FP64 latency, so by the warps in flight (283 us
// for 5,591,360 edges: FP64 pipe 56 %, L1 49 %, DRAM 24 %, 42 % of the warps);
// cycles of a mid-size case (ms) with 256 threads and 2, 3 blocks
// 2.66, 2.44, with 128 threads and 4 to 8 blocks 2.62, 2.47, 2.42, 2.39
// (7 blocks, 40 bytes of spills), 2.42.
__global__ void __launch_bounds__(kMusclThreads, 7) k_edge_flux_muscl(Params P, LevelView L) {
    __shared__ __align__(16) double sf[kMusclThreads * 5];
    const int e0 = blockIdx.x * blockDim.x, e = e0 + threadIdx.x;
    if (e < L.E) {
        const int2 nd = L.edge[e];
        double f[5];
        edge_flux_muscl(P, L, e, nd.x, nd.y, f);
#pragma unroll
        for (int k = 0; k < 5; ++k) sf[threadIdx.x * 5 + k] = f[k];
    }
    __syncthreads();
    store_block_fluxes(L.flux, sf, e0, min((int)blockDim.x, L.E - e0));
}

// ---- boundary-edge contributions ------------------------------------------
template <bool B>
__global__ void k_bnd_flux(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_) {
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    int b = tid();
    if (b >= L.B) return;
    double g1[5], g2[5];
    boundary_flux(P, L, b, [&](int j) { return load_state(L, j); }, g1, g2);
    double *o = L.bflux + (size_t)b * 10;
    for (int k = 0; k < 5; ++k) { o[k] = g1[k]; o[5 + k] = g2[k]; }
    if (L.bgterm) {
        boundary_gcl(P, L, b, g1, g2);
        double *t = L.bgterm + (size_t)b * 10;
        for (int k = 0; k < 5; ++k) { t[k] = g1[k]; t[5 + k] = g2[k]; }
    }
}

// ---- mixed precision ------------------------------------------------------
// The interior central flux of an edge is G(u1; w) + G(u2; w) with the
// one-sided flux G(u; w) = F(u).w.  FLITE_MIXED evaluates it as
//   G(u; w) = G(ua; w) + dG,
// where ua is an FP64 anchor state whose interior-edge residual was summed in
// FP64, and dG is computed in FP32 from the increments du = u - ua and
// dp = p - pa in a form whose every term carries an increment:
//   dv   = (dm - va drho) / rho
//   dG_0 = dm.w
//   dG_k = dm_k (v.w) + ma_k (dv.w) + dp w_k          k = 1..3
//   dG_4 = (dE + dp)(v.w) + (Ea + pa)(dv.w)
// so its rounding error is relative to the increment, not to the flux: the
// iteration converges to the FP64 fixed point.  The anchor is refreshed by an
// FP64 evaluation at the first stage of every relaxation step (and at the
// coarse-level evaluation of restrictGrid).

// the node's record for the increments: anchor primitives and u - ua (FP64
// difference, rounded once), p - pa
__device__ __forceinline__ void store_delta(const LevelView &L, DeltaRec *dq, int i, const double *u, double p) {
    const int N = L.N;
    DeltaRec o;
    o.ra = L.a32[i]; o.vax = L.a32[N + i]; o.vay = L.a32[2 * N + i]; o.vaz = L.a32[3 * N + i];
    o.ha = L.a32[4 * N + i];
    o.dr = (float)(u[0] - L.ua[i]);
    o.dmx = (float)(u[1] - L.ua[N + i]);
    o.dmy = (float)(u[2] - L.ua[2 * N + i]);
    o.dmz = (float)(u[3] - L.ua[3 * N + i]);
    o.dE = (float)(u[4] - L.ua[4 * N + i]);
    o.dp = (float)(p - L.pa[i]);
    o.pad = 0.f;
    float4 *d = reinterpret_cast<float4 *>(dq + i);
    const float4 *v = reinterpret_cast<const float4 *>(&o);
    d[0] = v[0]; d[1] = v[1]; d[2] = v[2];
}
template <bool B>
__global__ void k_delta_state(CaseArg<B, LevelView> L_) {
    FLITE_CASE_L(B, L);
    int i = tid();
    if (i >= L.N) return;
    const int N = L.N;
    const double u[5] = {L.u[i], L.u[N + i], L.u[2 * N + i], L.u[3 * N + i], L.u[4 * N + i]};
    store_delta(L, L.dq, i, u, L.p[i]);
}

// the rows of a level from its incidence lists; entries past a node's
// degree (never used) are the node itself as second node of edge 0
__global__ void k_make_rows(LevelView L, int nrows, int2 *rows) {
    const int i = tid();
    if (i >= L.N) return;
    const int beg = L.inc_ptr[i], deg = L.inc_ptr[i + 1] - beg, s = i / kRow;
    const int first = L.row_ptr[s], last = (s + 1) * kRow < L.N ? L.row_ptr[s + 1] : nrows;
    for (int k = 0; k < last - first; ++k)
        rows[(size_t)(first + k) * kRow + i % kRow] = k < deg ? L.inc[beg + k] : make_int2(~0, i);
}
// the device's edge numbers by rows: the number of edges whose first node
// holds them in each row (a warp per row: kRow is the warp size), the first
// number of each row, and each edge's; then the numbers put into the
// incidences and the edges moved
static_assert(kRow == 32, "a row is a warp");
__global__ void k_row_firsts(const int2 *rows, int nrows, int *first) {
    const int t = tid(), r = t / kRow;
    if (r >= nrows) return;
    const unsigned m = __ballot_sync(0xffffffffu, rows[t].x >= 0);
    if (t % kRow == 0) first[r] = __popc(m);
}
// exclusive sums in place, one block
__global__ void __launch_bounds__(1024) k_scan_rows(int *first, int nrows) {
    __shared__ int part[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    for (int base = 0; base < nrows; base += 1024) {
        const int k = base + threadIdx.x;
        const int own = k < nrows ? first[k] : 0;
        int v = own;
        for (int o = 1; o < 32; o *= 2) {
            const int x = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += x;
        }
        if (lane == 31) part[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int w = part[lane];
            for (int o = 1; o < 32; o *= 2) {
                const int x = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += x;
            }
            part[lane] = w;
        }
        __syncthreads();
        const int before = carry + (warp ? part[warp - 1] : 0) + v - own;
        if (k < nrows) first[k] = before;
        __syncthreads();
        if (threadIdx.x == 0) carry += part[31];
        __syncthreads();
    }
}
__global__ void k_edge_slots(const int2 *rows, int nrows, const int *first, int *slot) {
    const int t = tid(), r = t / kRow;
    if (r >= nrows) return;
    const int e = rows[t].x;
    const unsigned m = __ballot_sync(0xffffffffu, e >= 0);
    if (e >= 0) slot[e] = first[r] + __popc(m & ((1u << (t % kRow)) - 1u));
}
__global__ void k_renumber_edges(int2 *inc, int n, const int *slot) {
    const int k = tid();
    if (k >= n) return;
    const int x = inc[k].x;
    inc[k].x = x >= 0 ? slot[x] : ~slot[~x];
}
__global__ void k_move_edges(int E, const int *slot, const int2 *in, int2 *out) {
    const int e = tid();
    if (e < E) out[slot[e]] = in[e];
}
// edge arrays from the caller's edge order (w: [3][E])
__global__ void k_put_edges(int E, const int *slot, const double *w, double *wx, double *wy, double *wz, EdgeW *ew) {
    const int e = tid();
    if (e >= E) return;
    const int q = slot ? slot[e] : e;
    const double x = w[e], y = w[(size_t)E + e], z = w[2 * (size_t)E + e];
    wx[q] = x; wy[q] = y; wz[q] = z;
    ew[q] = EdgeW{x, y, z, 0.0};
}
__global__ void k_put_edge_values(int E, const int *slot, const double *in, double *out) {
    const int e = tid();
    if (e < E) out[slot ? slot[e] : e] = in[e];
}

// FP32 incidences of the increments (w rounded once; j is ~j when the node
// is the edge's second node)
__global__ void k_make_inc32(const int2 *inc, const EdgeW *ew, int n, IncRec32 *o) {
    int k = tid();
    if (k >= n) return;
    const int2 t = inc[k];
    const EdgeW w = ew[t.x >= 0 ? t.x : ~t.x];
    o[k] = IncRec32{(float)w.wx, (float)w.wy, (float)w.wz, t.x >= 0 ? t.y : ~t.y};
}

__device__ __forceinline__ DeltaRec load_delta(const DeltaRec *q, int j) {
    const float4 *p = reinterpret_cast<const float4 *>(q + j);
    DeltaRec o;
    float4 *d = reinterpret_cast<float4 *>(&o);
    d[0] = __ldg(p); d[1] = __ldg(p + 1); d[2] = __ldg(p + 2);
    return o;
}

// increment of the one-sided flux G(u; w) of one node
__device__ __forceinline__ void delta_flux(const DeltaRec &n, float wx, float wy, float wz, float *g) {
    const float rinv = 1.f / (n.ra + n.dr);
    const float dvx = (n.dmx - n.vax * n.dr) * rinv, dvy = (n.dmy - n.vay * n.dr) * rinv;
    const float dvz = (n.dmz - n.vaz * n.dr) * rinv;
    const float vw = ((n.vax + dvx) * wx + (n.vay + dvy) * wy) + (n.vaz + dvz) * wz;
    const float dvw = (dvx * wx + dvy * wy) + dvz * wz;
    g[0] = (n.dmx * wx + n.dmy * wy) + n.dmz * wz;
    g[1] = (n.dmx * vw + (n.ra * n.vax) * dvw) + n.dp * wx;
    g[2] = (n.dmy * vw + (n.ra * n.vay) * dvw) + n.dp * wy;
    g[3] = (n.dmz * vw + (n.ra * n.vaz) * dvw) + n.dp * wz;
    g[4] = (n.dE + n.dp) * vw + n.ha * dvw;
}

// interior residual of node i as the anchor's FP64 sum plus the FP32 sum of
// the flux increments of its edges
template <int U>
__device__ __forceinline__ void gather_interior_delta(const LevelView &L, const DeltaRec *dqin, int i, double *r,
                                                      bool active, int gl, double *gs) {
    float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    const DeltaRec me = load_delta(dqin, i);
    auto terms = [&](const IncRec32 &t, float *s5, bool &first) {
        first = t.j >= 0;
        const DeltaRec nb = load_delta(dqin, first ? t.j : ~t.j);
        float g1[5], g2[5];
        delta_flux(first ? me : nb, t.wx, t.wy, t.wz, g1);
        delta_flux(first ? nb : me, t.wx, t.wy, t.wz, g2);
        for (int c = 0; c < 5; ++c) s5[c] = g1[c] + g2[c];
    };
    if constexpr (U > 1) {
        group_sum<U, 5, 1, float>(
            reinterpret_cast<float *>(gs), L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
            [&](int k, float *v) {
                bool first;
                terms(load_inc32(L.inc32, k), v, first);
                if (!first)
                    for (int c = 0; c < 5; ++c) v[c] = -v[c];  // x - y is x + (-y)
            },
            acc);
    } else {
        const int deg = L.inc_ptr[i + 1] - L.inc_ptr[i];
        const IncRec32 *row = L.rows32 + ((size_t)L.row_ptr[i / kRow] * kRow + i % kRow);
        // two incidences at a time, for the loads in flight
        auto add = [&](const float *v, bool first) {
            for (int c = 0; c < 5; ++c) acc[c] += first ? v[c] : -v[c];
        };
        int k = 0;
        IncRec32 a, b;
        if (deg > 0) a = load_inc32(row, 0);
        if (deg > 1) b = load_inc32(row, kRow);
        for (; k + 1 < deg; k += 2) {
            const IncRec32 t0 = a, t1 = b;
            row += 2 * kRow;
            if (k + 2 < deg) a = load_inc32(row, 0);
            if (k + 3 < deg) b = load_inc32(row, kRow);
            float v[5], w[5];
            bool f, g;
            terms(t0, v, f);
            terms(t1, w, g);
            add(v, f);
            add(w, g);
        }
        if (k < deg) {
            float v[5];
            bool f;
            terms(a, v, f);
            add(v, f);
        }
    }
    const int N = L.N;
    for (int c = 0; c < 5; ++c) r[c] = L.ra[c * N + i] + (double)acc[c];
}

// Interior central fluxes of node i with a thread per node, summed in edge
// order: the other nodes' records and the edges' coefficients of the next
// kPipe - 1 incidences are copied ahead into the thread's own slots of shared
// memory (asynchronous copies hold no registers, and each thread waits for
// its own only).
// What bounds it: the latency of the loads, not their bytes.  On the
// 815,425-node level one launch takes 131 us with the copies ahead, 154 us
// with plain loads from the incidence lists and 172 us with plain loads from
// the rows; kPipe 2, 3 and 4 take 154, 139 and 140 us without the prefetch
// below, 5 blocks of 128 threads per SM fit without spills, 4 and 6 take 152
// and 163 us.
constexpr int kPipe = 3, kPipeThreads = 128;
__device__ __forceinline__ void copy_ahead16(void *d, const void *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(g)
                 : "memory");
}
__device__ __forceinline__ void copy_ahead8(void *d, const void *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(g)
                 : "memory");
}
__device__ __forceinline__ void gather_central_ahead(const LevelView &L, const NodeRec *qin, int i, double *r) {
    __shared__ double2 sq[kPipe][3][kPipeThreads];
    __shared__ double sw[kPipe][3][kPipeThreads];
    const int tx = threadIdx.x;
    r[0] = r[1] = r[2] = r[3] = r[4] = 0.0;
    const int deg = L.inc_ptr[i + 1] - L.inc_ptr[i];
    const int2 *row = L.rows + ((size_t)L.row_ptr[i / kRow] * kRow + i % kRow);
    const NodeRec si = load_node(qin, i);
    int side[kPipe];
    auto issue = [&](const int2 t, int d) {
        const int e = t.x >= 0 ? t.x : ~t.x;
        const double2 *q = reinterpret_cast<const double2 *>(qin + t.y);
        copy_ahead16(&sq[d][0][tx], q);
        copy_ahead16(&sq[d][1][tx], q + 1);
        copy_ahead16(&sq[d][2][tx], q + 2);
        copy_ahead8(&sw[d][0][tx], L.wx + e);
        copy_ahead8(&sw[d][1][tx], L.wy + e);
        copy_ahead8(&sw[d][2][tx], L.wz + e);
        side[d] = t.x;
    };
#pragma unroll
    for (int d = 0; d < kPipe - 1; ++d) {
        if (d < deg) issue(__ldg(row + d * kRow), d);
        asm volatile("cp.async.commit_group;");
    }
    int2 t = make_int2(0, 0);
    if (kPipe - 1 < deg) t = __ldg(row + (kPipe - 1) * kRow);
    for (int k0 = 0; k0 < deg; k0 += kPipe) {
#pragma unroll
        for (int d = 0; d < kPipe; ++d) {
            const int k = k0 + d, kn = k + kPipe - 1;
            if (k >= deg) break;
            if (kn < deg) issue(t, (d + kPipe - 1) % kPipe);
            asm volatile("cp.async.commit_group;");
            if (kn + 1 < deg) t = __ldg(row + (size_t)(kn + 1) * kRow);
            asm volatile("cp.async.wait_group %0;" ::"n"(kPipe - 1) : "memory");
            const double2 a = sq[d][0][tx], b = sq[d][1][tx], c = sq[d][2][tx];
            const NodeRec n = {a.x, a.y, b.x, b.y, c.x, c.y};
            const double wx = sw[d][0][tx], wy = sw[d][1][tx], wz = sw[d][2][tx];
            double f[5];
            if (side[d] >= 0) {
                central_flux_rec(si, n, wx, wy, wz, f);
                r[0] = r[0] + f[0]; r[1] = r[1] + f[1]; r[2] = r[2] + f[2]; r[3] = r[3] + f[3]; r[4] = r[4] + f[4];
            } else {
                central_flux_rec(n, si, wx, wy, wz, f);
                r[0] = r[0] - f[0]; r[1] = r[1] - f[1]; r[2] = r[2] - f[2]; r[3] = r[3] - f[3]; r[4] = r[4] - f[4];
            }
        }
    }
}
// The block's incidence rows (one contiguous run) on their way to L2 before
// the walk asks for them row by row: 16-byte aligned, whole rows of 256 bytes.
__device__ __forceinline__ void prefetch_rows(const LevelView &L) {
    if (threadIdx.x) return;
    const int i0 = blockIdx.x * blockDim.x;
    const int s0 = i0 / kRow, s1 = min(i0 + (int)blockDim.x, L.N) / kRow;
    const int r0 = L.row_ptr[s0], r1 = s1 * kRow < L.N ? L.row_ptr[s1] : r0;
    if (r1 > r0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(L.rows + (size_t)r0 * kRow),
                     "r"((unsigned)(r1 - r0) * (unsigned)(kRow * sizeof(int2))));
}

// the same sums with a group of lanes per node
template <int U>
__device__ __forceinline__ void gather_interior_central(const LevelView &L, const NodeRec *qin, int i, double *r,
                                                        bool active, int gl, double *gs) {
    r[0] = r[1] = r[2] = r[3] = r[4] = 0.0;
    const NodeRec si = load_node(qin, i);
    group_sum<U, 5, 1, double>(
        gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
        [&](int k, double *g) {
            const int2 t = L.inc[k];
            const EdgeW w = load_edgew(L.ew, t.x >= 0 ? t.x : ~t.x);
            const NodeRec n = load_node(qin, t.y);
            if (t.x >= 0) {
                central_flux_rec(si, n, w.wx, w.wy, w.wz, g);
            } else {  // this node's sign: x - y is x + (-y)
                double f[5];
                central_flux_rec(n, si, w.wx, w.wy, w.wz, f);
                for (int c = 0; c < 5; ++c) g[c] = -f[c];
            }
        },
        r);
}

// interior edges of node i from the FP64 edge buffer, in edge order
template <int U>
__device__ __forceinline__ void gather_interior(const LevelView &L, int i, double *r, bool active, int gl,
                                                double *gs) {
    r[0] = r[1] = r[2] = r[3] = r[4] = 0.0;
    auto terms = [&](const int2 t, double *g) {
        const int s = t.x;
        const double *f = L.flux + (size_t)(s >= 0 ? s : ~s) * 5;
        for (int c = 0; c < 5; ++c) g[c] = s >= 0 ? f[c] : -f[c];  // x - y is x + (-y)
    };
    auto add = [&](const double *g) {
        r[0] = r[0] + g[0]; r[1] = r[1] + g[1]; r[2] = r[2] + g[2]; r[3] = r[3] + g[3]; r[4] = r[4] + g[4];
    };
    if constexpr (U > 1) {
        group_sum<U, 5, 1, double>(gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl,
                                        [&](int k, double *v) { terms(L.inc[k], v); }, r);
    } else {
        walk<2, 5>(L, i, terms, add);
    }
}

// boundary edges of node i (FP64).  On a moving mesh each boundary edge
// first subtracts its GCL terms from both its nodes, then adds its fluxes
// (def_par:2124-2177): per node -t, +g; an edge with both ends at node i (a
// coarse level's self-edge) gives -t1, -t2, +g1, +g2, its second end's
// entry following its first in the node's list
template <int U>
__device__ __forceinline__ void gather_boundary(const LevelView &L, int i, double *r, bool active = true,
                                                int gl = 0, double *gs = nullptr) {
    auto terms = [&](int k, double *g) {
        const int v = L.binc[k];
        const double *b = L.bflux + (size_t)(v >> 1) * 10 + (v & 1) * 5;
        for (int c = 0; c < 5; ++c) g[c] = b[c];
    };
    auto add = [&](const double *g) {
        r[0] = r[0] + g[0]; r[1] = r[1] + g[1]; r[2] = r[2] + g[2]; r[3] = r[3] + g[3]; r[4] = r[4] + g[4];
    };
    // g[0..4] the GCL term, g[5..9] the flux, g[10] 0 (an edge between two
    // nodes), 1 or 2 (first or second end of a self-edge)
    auto terms_gcl = [&](int k, double *g) {
        const int v = L.binc[k];
        const size_t o = (size_t)(v >> 1) * 10 + (v & 1) * 5;
        for (int c = 0; c < 5; ++c) { g[c] = L.bgterm[o + c]; g[5 + c] = L.bflux[o + c]; }
        const int2 nd = L.bedge[v >> 1];
        g[10] = nd.x == nd.y ? (double)(1 + (v & 1)) : 0.0;
    };
    double pend[5];  // the flux of a self-edge's first end, added after its second GCL term
    auto add_gcl = [&](const double *g) {
        if (g[10] == 1.0) {
            for (int c = 0; c < 5; ++c) { r[c] = r[c] - g[c]; pend[c] = g[5 + c]; }
        } else if (g[10] == 2.0) {
            for (int c = 0; c < 5; ++c) r[c] = ((r[c] - g[c]) + pend[c]) + g[5 + c];
        } else {
            for (int c = 0; c < 5; ++c) r[c] = (r[c] - g[c]) + g[5 + c];
        }
    };
    if constexpr (U > 1) {
        if (L.bgterm) {
            // two terms per entry: -t, +g; a self-edge's entries, which follow
            // one another, give -t1, -t2 and +g1, +g2
            group_sum<U, 5, 2, double>(
                gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl,
                [&](int k, double *g) {
                    const int v = L.binc[k];
                    const size_t o = (size_t)(v >> 1) * 10, own = o + (v & 1) * 5;
                    const int2 nd = L.bedge[v >> 1];
                    const bool self = nd.x == nd.y;
                    const double *t = self ? ((v & 1) ? L.bflux + o : L.bgterm + o) : L.bgterm + own;
                    const double *f = self ? t + 5 : L.bflux + own;
                    const bool plus0 = self && (v & 1), minus1 = self && !(v & 1);
                    for (int c = 0; c < 5; ++c) {
                        g[2 * c] = plus0 ? t[c] : -t[c];
                        g[2 * c + 1] = minus1 ? -f[c] : f[c];
                    }
                },
                r);
        } else {
            group_sum<U, 5, 1, double>(gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl, terms, r);
        }
    } else if (L.bgterm) {
        for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
            double v[11];
            terms_gcl(k, v);
            add_gcl(v);
        }
    } else {
        for (int k = L.binc_ptr[i]; k < L.binc_ptr[i + 1]; ++k) {
            double v[5];
            terms(k, v);
            add(v);
        }
    }
}

// boundary edges of node i evaluated by its group (a static mesh's): lane by
// lane, the edge's flux to this node from the states in uin and the pressures
// of the records, the numbers k_bnd_flux leaves in bflux
template <int U>
__device__ __forceinline__ void gather_boundary_inline(const Params &P, const LevelView &L, const double *uin,
                                                       const NodeRec *qin, int i, double *r, bool active, int gl,
                                                       double *gs) {
    const int N = L.N;
    auto state = [&](int j) {
        NodeState s;
        s.r = uin[j]; s.ru = uin[N + j]; s.rv = uin[2 * N + j]; s.rw = uin[3 * N + j]; s.E = uin[4 * N + j];
        s.p = qin[j].p;
        return s;
    };
    group_sum<U, 5, 1, double>(
        gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl,
        [&](int k, double *v) {
            const int b = L.binc[k];
            double g1[5], g2[5];
            boundary_flux(P, L, b >> 1, state, g1, g2);
            for (int c = 0; c < 5; ++c) v[c] = (b & 1) ? g2[c] : g1[c];
        },
        r);
}

// the FP64 evaluation becomes the new anchor of node i
__device__ __forceinline__ void store_anchor(const LevelView &L, int i, const double *rint) {
    const int N = L.N;
    double u[5];
    for (int c = 0; c < 5; ++c) {
        u[c] = L.u[c * N + i];
        L.ua[c * N + i] = u[c];
        L.ra[c * N + i] = rint[c];
    }
    const double p = L.p[i];
    L.pa[i] = p;
    const double rinv = 1.0 / u[0];
    L.a32[i] = (float)u[0];
    L.a32[N + i] = (float)(u[1] * rinv);
    L.a32[2 * N + i] = (float)(u[2] * rinv);
    L.a32[3 * N + i] = (float)(u[3] * rinv);
    L.a32[4 * N + i] = (float)(u[4] + p);
}

// the node part of a stage after the residual r of node i is summed:
// time differences, dissipation, solveSystem, the increment conditions, the
// clipped update and the solution and outer conditions, or the restrictGrid
// one-step forms (modes as in k_node_update)
// LEAN: a run without engine conditions and without explicit time stepping
// (the branches for those are left out of the code)
// the state a node pass reads
__device__ __forceinline__ const double *io_in(const LevelView &L, int io) {
    return (io & IO_UIN) == 0 ? L.u : (io & IO_UIN) == 1 ? L.uprev : L.ub;
}
struct TailIn {  // what the tail reads of its node, loaded ahead by the group gathers
    double diss[5], up[5], dt, V, p;
    unsigned char cls;
};
__device__ __forceinline__ TailIn load_tail(const LevelView &L, int i) {
    const int N = L.N;
    TailIn t;
    t.dt = L.dt[i];
    t.V = L.V[i];
    t.p = L.p[i];
    t.cls = L.bc[i];
    for (int c = 0; c < 5; ++c) { t.diss[c] = L.diss[c * N + i]; t.up[c] = L.uprev[c * N + i]; }
    return t;
}
// PREC names the records an IO_EMIT pass leaves for the next stage (none for
// the edge buffer's fluxes)
template <int PREC>
__device__ __forceinline__ void node_tail(const Params &P, const LevelView &L, int i, double *r, int mode, int stage,
                                          int io, const TailIn *in) {
    constexpr bool LEAN = PREC == GATHER_LEAN;
    const int N = L.N;
    if (mode == MODE_RESID) {
        for (int c = 0; c < 5; ++c) L.rhs[c * N + i] = r[c];
        return;
    }
    if (P.addts && mode == MODE_STAGE)  // addTimeDifferences (def_par:1184-1241)
        for (int c = 0; c < 5; ++c) r[c] = r[c] + time_difference(P, L, io_in(L, io), i, c);
    for (int c = 0; c < 5; ++c) r[c] = r[c] + (in ? in->diss[c] : L.diss[c * N + i]);
    double dt = in ? in->dt : L.dt[i];
    const double V = in ? in->V : L.V[i];
    // solveSystem's dual-time step, or the explicit global step (def_par:1427-1442)
    if (P.unsteady) dt = (!LEAN && P.explicit_) ? *L.ptsg : dt / (1.0 + 1.5 * dt / P.dtp);
    for (int c = 0; c < 5; ++c) r[c] = dt * r[c] / V;  // solveSystem
    const unsigned char cls = in ? in->cls : L.bc[i];
    double n0 = 0, n1 = 0, n2 = 0;
    if (cls != BC_NONE) { n0 = L.nx[i]; n1 = L.ny[i]; n2 = L.nz[i]; }
    bc_increment<!LEAN>(P, cls, n0, n1, n2, r);
    // nullifyOuterBoundary (coarse levels): zeroes the far-field (indicator
    // 3) and engine increments for the SA model and is a no-op otherwise
    if (P.sa && L.grid > 1 && (cls == BC_FAR3 || (!LEAN && is_engine(cls)))) r[0] = r[1] = r[2] = r[3] = r[4] = 0.0;
    const double dtJ = stage > 0 ? P.CFL * P.RK[stage - 1] : P.CFL;
    double d[5], up[5], un[5];
    for (int c = 0; c < 5; ++c) { d[c] = dtJ * r[c]; up[c] = in ? in->up[c] : L.uprev[c * N + i]; }
    clipped_update(P, up, d, un);
    if (mode == MODE_RFINE) {
        // the density floor of updateSolutionVector acts on grp%u, which is
        // not the array being updated in this call (def_par:1398-1403)
        // (IO_LATER: other lanes of this launch still read it; k_restrict_incr
        // floors it)
        if (!(io & IO_LATER) && L.u[i] < P.minRho) L.u[i] = P.minRho;
    } else {
        if (un[0] < P.minRho) un[0] = P.minRho;
    }
    double cm0 = 0, cm1 = 0, cm2 = 0;
    if (cls == BC_WALL && P.viscous) { cm0 = L.cmx[i]; cm1 = L.cmy[i]; cm2 = L.cmz[i]; }
    bc_solution(P, cls, n0, n1, n2, cm0, cm1, cm2, relax_param(P, *L.cyc), un);
    if (!LEAN && is_exhaust(cls)) {
        // the exhaust pressure matters on level 1 only: coarse pressures are
        // recomputed before anything reads them
        const double pex = bc_exhaust(P, cls, eo_relax(P, *L.cyc), un);
        if (L.eng.f) L.eng.pbc[i] = pex;
    }
    if (!LEAN && L.eng.f && mode != MODE_RCOARSE && (P.eftype == 2 || is_engine(cls))) {
        // level 1: the engine inlet terms need every node's state first;
        // k_engine_finish completes the node (the candidate state of
        // restrictGrid's fine step goes to rhs)
        double *T = mode == MODE_RFINE ? L.rhs : L.u;
        for (int c = 0; c < 5; ++c) T[c * N + i] = un[c];
        return;
    }
    const double p_in = in ? in->p : L.p[i];
    if (mode == MODE_STAGE) {
        if (L.grid > 1) {
            const double a = P.RK[stage - 1];
            for (int c = 0; c < 5; ++c) un[c] = un[c] - a * L.src[c * N + i];
        }
        un[0] = dmax(un[0], P.minRho);  // limitDensity
        bc_outer(P, cls, n0, n1, n2, p_in, un);
        double *uo = io & IO_UOUT_B ? L.ub : L.u;
        for (int c = 0; c < 5; ++c) uo[c * N + i] = un[c];
        if (io & IO_EMIT) {  // makePressureField of the next stage
            const double p = pressure(P, un[0], un[1], un[2], un[3], un[4]);
            L.p[i] = p;
            if (L.saprim) store_saprim(L, i, un[0], un[1], un[2], un[3]);
            if constexpr (PREC == GATHER_BUFFER)
                if (L.hprim) {
                    L.hprim[i] = un[1] / un[0]; L.hprim[N + i] = un[2] / un[0]; L.hprim[2 * N + i] = un[3] / un[0];
                }
            if constexpr (PREC == GATHER_ANCHOR || PREC == GATHER_DELTA)
                store_delta(L, io & IO_REC_B ? L.dq : L.dqb, i, un, p);
            else if constexpr (PREC != GATHER_BUFFER)
                store_node(io & IO_REC_B ? L.q : L.qb, i, un[0], un[1], un[2], un[3], un[4], p);
        }
    } else if (mode == MODE_RCOARSE) {
        bc_outer(P, cls, n0, n1, n2, p_in, un);
        for (int c = 0; c < 5; ++c) L.src[c * N + i] = un[c] - up[c];
    } else {  // MODE_RFINE
        if (L.grid > 1)
            for (int c = 0; c < 5; ++c) un[c] = un[c] - L.src[c * N + i];
        bc_outer(P, cls, n0, n1, n2, p_in, un);
        for (int c = 0; c < 5; ++c) L.rhs[c * N + i] = un[c] - up[c];
    }
}

// ---- the node part of one RK stage (def_par:1069-1178), fused -------------
// mode STAGE:   u <- update of stage `stage`
// mode RCOARSE: restrictGrid coarse one-step (def_par:12244-12263): src
// mode RFINE:   restrictGrid fine increment (def_par:12356-12383): rhs
// mode RESID:   rhs <- makeRHS only
// PREC: GATHER_BUFFER (FP64 edge buffer of the upwind fluxes),
// GATHER_CENTRAL (central fluxes computed in the gather), GATHER_ANCHOR (the
// same, stored as the new mixed-precision anchor), GATHER_DELTA (anchor +
// FP32 increments)
template <int PREC, int U, int PRE, bool B>
__global__ void __launch_bounds__(node_threads(PREC, U), U > 1 ? 2 : (central_ahead(PREC) ? 5 : (PREC == GATHER_DELTA ? 4 : 3)))
    k_node_update(CaseArg<B, Params> P_, CaseArg<B, LevelView> L_, int mode, int stage, int io) {
    static_assert(PRE == PRE_NONE || U > 1, "the dissipation part takes lanes per node");
    FLITE_CASE_P(B, P, L);
    FLITE_CASE_L(B, L);
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;  // lane in the node's group
    const int i_raw = U > 1 ? tid() / U : tid();
    if (U == 1 && i_raw >= L.N) return;
    const bool active = i_raw < L.N;
    const int i = active ? i_raw : L.N - 1;  // idle groups read a valid node
    if constexpr (U == 1 && central_ahead(PREC)) prefetch_rows(L);
    double r[5];
    FLITE_GROUP_SLAB(double, 10);
    // a node's own operands are read before the chain of its gather starts
    TailIn in;
    if constexpr (U > 1) in = load_tail(L, i);
    if constexpr (PRE == PRE_JST) {
        jflux_group<U>(P, L, io_in(L, io), i, active, gl, gs, in.diss);
    } else if constexpr (PRE == PRE_VISC) {
        double v[4];
        vflux_group<U>(L, i, active, gl, gs, v);
        for (int c = 0; c < 4; ++c) in.diss[1 + c] = in.diss[1 + c] - v[c];
    }
    if constexpr (PRE != PRE_NONE)
        if (active && gl == 0)
            for (int c = 0; c < 5; ++c) L.diss[c * L.N + i] = in.diss[c];
    const NodeRec *qin = io & IO_REC_B ? L.qb : L.q;
    if constexpr (PREC == GATHER_DELTA) {
        gather_interior_delta<U>(L, io & IO_REC_B ? L.dqb : L.dq, i, r, active, gl, gs);
    } else if constexpr (PREC == GATHER_BUFFER) {
        gather_interior<U>(L, i, r, active, gl, gs);
    } else if constexpr (U == 1) {
        gather_central_ahead(L, qin, i, r);
    } else {
        gather_interior_central<U>(L, qin, i, r, active, gl, gs);
    }
    double rint[5];
    if constexpr (PREC == GATHER_ANCHOR)
        for (int c = 0; c < 5; ++c) rint[c] = r[c];
    if constexpr (U > 1 && PREC == GATHER_CENTRAL) {
        if (io & IO_BND) gather_boundary_inline<U>(P, L, io_in(L, io), qin, i, r, active, gl, gs);
        else gather_boundary<U>(L, i, r, active, gl, gs);
    } else {
        gather_boundary<U>(L, i, r, active, gl, gs);
    }
    // with a group per node every lane holds the same sums; one lane goes on
    if constexpr (U > 1)
        if (!active || gl) return;
    if constexpr (PREC == GATHER_ANCHOR) store_anchor(L, i, rint);
    node_tail<PREC>(P, L, i, r, mode, stage, io, U > 1 ? &in : nullptr);
}
#define FLITE_BOTH(kern, targs, ...)                                               \
    template __global__ void kern<FLITE_ARGS targs false> FLITE_SINGLE(__VA_ARGS__); \
    template __global__ void kern<FLITE_ARGS targs true> FLITE_GROUPED(__VA_ARGS__);
#define FLITE_ARGS(...) __VA_ARGS__
#define FLITE_SINGLE(...) (Params, LevelView __VA_ARGS__)
#define FLITE_GROUPED(...) (CaseTab<Params>, CaseTab<LevelView> __VA_ARGS__)
#define FLITE_NODE_INST(PREC, U, PRE)                                                                          \
    template __global__ void k_node_update<PREC, U, PRE, false>(Params, LevelView, int, int, int);              \
    template __global__ void k_node_update<PREC, U, PRE, true>(CaseTab<Params>, CaseTab<LevelView>, int, int, int);
#define FLITE_GATHER_INST(U)                                                                 \
    FLITE_BOTH(k_timestep, (U, ))                                                            \
    FLITE_BOTH(k_jst_lap, (U, ))                                                             \
    FLITE_BOTH(k_jst_flux, (U, ))                                                            \
    FLITE_BOTH(k_visc_grad, (U, ))                                                           \
    FLITE_BOTH(k_visc_flux, (U, ))                                                           \
    FLITE_BOTH(k_visc2_grad, (U, ))                                                          \
    FLITE_BOTH(k_visc2_flux, (U, ))                                                          \
    FLITE_BOTH(k_ts_lap, (U, ))                                                              \
    FLITE_BOTH(k_jflux_vgrad, (U, ))                                                         \
    template __global__ void k_node_update<GATHER_BUFFER, U>(Params, LevelView, int, int, int); \
    FLITE_NODE_INST(GATHER_CENTRAL, U, PRE_NONE)                                             \
    FLITE_NODE_INST(GATHER_ANCHOR, U, PRE_NONE)                                              \
    FLITE_NODE_INST(GATHER_DELTA, U, PRE_NONE)
#define FLITE_GROUP_INST(U)                          \
    FLITE_GATHER_INST(U)                             \
    FLITE_NODE_INST(GATHER_CENTRAL, U, PRE_JST)      \
    FLITE_NODE_INST(GATHER_CENTRAL, U, PRE_VISC)
FLITE_GATHER_INST(1)
FLITE_NODE_INST(GATHER_LEAN, 1, PRE_NONE)
FLITE_GROUP_INST(4)
FLITE_GROUP_INST(8)
FLITE_GROUP_INST(16)
FLITE_GROUP_INST(32)
template __global__ void k_first_order_diss<1>(Params, LevelView);
template __global__ void k_state_pass<false, false>(Params, LevelView, int, const int *);
template __global__ void k_state_pass<false, true>(CaseTab<Params>, CaseTab<LevelView>, int, const int *);
template __global__ void k_state_pass<true, false>(Params, LevelView, int, const int *);
template __global__ void k_state_pass<true, true>(CaseTab<Params>, CaseTab<LevelView>, int, const int *);
template __global__ void k_prolong<false>(Params, LevelView, LevelView);
template __global__ void k_prolong<true>(CaseTab<Params>, CaseTab<LevelView>, CaseTab<LevelView>);
template __global__ void k_bnd_flux<false>(Params, LevelView);
template __global__ void k_bnd_flux<true>(CaseTab<Params>, CaseTab<LevelView>);
template __global__ void k_delta_state<false>(LevelView);
template __global__ void k_delta_state<true>(CaseTab<LevelView>);
template __global__ void k_restrict_u<false>(LevelView, LevelView);
template __global__ void k_restrict_u<true>(CaseTab<LevelView>, CaseTab<LevelView>);
template __global__ void k_restrict_state<false>(Params, LevelView, LevelView);
template __global__ void k_restrict_state<true>(CaseTab<Params>, CaseTab<LevelView>, CaseTab<LevelView>);
template __global__ void k_restrict_incr<false>(Params, LevelView, LevelView, int);
template __global__ void k_restrict_incr<true>(CaseTab<Params>, CaseTab<LevelView>, CaseTab<LevelView>, int);
template __global__ void k_prolong_coarse<false>(Params, LevelView, LevelView);
template __global__ void k_prolong_coarse<true>(CaseTab<Params>, CaseTab<LevelView>, CaseTab<LevelView>);
template __global__ void k_prolong_fine<false>(Params, LevelView, LevelView);
template __global__ void k_prolong_fine<true>(CaseTab<Params>, CaseTab<LevelView>, CaseTab<LevelView>);
template __global__ void k_inject_u<false>(LevelView, LevelView);
template __global__ void k_inject_u<true>(CaseTab<LevelView>, CaseTab<LevelView>);

// mapFineToCoarse (def_par:12572-12596) as a gather over each coarse node's
// children in increasing fine order: the same additions in the same order as
// the reference's scatter over fine nodes.  kChildLanes lanes take a coarse
// node's children (8 to 9 on the agglomerated levels) and add the sums'
// terms as group_sum does: with a thread per coarse node the transfers of the
// 203,401-node mesh take 15 to 23 us each, bound by one thread's chain of
// child -> value loads.
template <int M>
__device__ __forceinline__ void restrict_group(const LevelView &C, int c, bool active, int gl, double *gs,
                                               const double *const (&fine)[M], double *out) {
#pragma unroll
    for (int k = 0; k < M; ++k) out[k] = 0.0;
    group_sum<kChildLanes, M, 1, double>(
        gs, C.child_ptr[c], C.child_ptr[c + 1], active, gl,
        [&](int q, double *v) {
            const int f = C.child[q];
            const double w = C.rweight[f];
#pragma unroll
            for (int k = 0; k < M; ++k) v[k] = w * fine[k][f];
        },
        out);
}
// the coarse node and lane of a transfer kernel's thread
#define FLITE_CHILD_LANES(M)                                                          \
    constexpr int U = kChildLanes;                                                     \
    FLITE_GROUP_SLAB(double, M);                                                       \
    const int gl = (int)(threadIdx.x % U), c_raw = tid() / U;                          \
    const bool active = c_raw < C.N;                                                   \
    const int c = active ? c_raw : C.N - 1

// C.u = R(F.u) (plain mapFineToCoarse of the solution)
template <bool B>
__global__ void k_restrict_u(CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_) {
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    FLITE_CHILD_LANES(6);
    const size_t n = F.N;
    // (without nu~ the sixth sum repeats the first and is dropped)
    const double *const src[6] = {F.u, F.u + n, F.u + 2 * n, F.u + 3 * n, F.u + 4 * n, C.nvar == 6 ? F.u + 5 * n : F.u};
    double v[6];
    restrict_group<6>(C, c, active, gl, gs, src, v);
    if (!active || gl) return;
    for (int k = 0; k < 5; ++k) C.u[k * C.N + c] = v[k];
    if (C.nvar == 6) C.u[5 * C.N + c] = v[5];
}

// mapFineToCoarse of another array (def_par:12572-12679)
__global__ void k_restrict_arr(LevelView C, LevelView F, const double *fsrc, double *cdst, int ncomp) {
    int c = tid();
    if (c >= C.N) return;
    for (int k = 0; k < ncomp; ++k) {
        double v = 0.0;
        for (int q = C.child_ptr[c]; q < C.child_ptr[c + 1]; ++q) {
            const int f = C.child[q];
            v = v + C.rweight[f] * fsrc[(size_t)k * F.N + f];
        }
        cdst[k * C.N + c] = v;
    }
}

// the nu~ solution conditions: zero on walls (def_par:4416-4418, 4446-4448,
// 4469-4471), the ramped exhaust value on engine exhausts (:4507-4530), 0.1
// on the far field (def_par:4076-4140); rp is the exhaust ramp
__device__ __forceinline__ double sa_bc_solution(const Params &P, unsigned char cls, double rp, double v) {
    if (cls == BC_WALL || cls == BC_IWALL) return 0.0;
    if (is_exhaust(cls)) return sa_exhaust(P, cls, rp);
    if (cls == BC_FAR3 || cls == BC_FAR4) return 0.1;
    return v;
}
// the nu~ increment conditions (def_par:4978-5125)
__device__ __forceinline__ double sa_bc_increment(const Params &P, unsigned char cls, double r) {
    if (cls == BC_WALL || cls == BC_IWALL || is_exhaust(cls)) return 0.0;
    if (is_inlet(cls)) return P.engRelax * r;
    return r;
}

// restrictGrid head (def_par:12159-12185): C.u = R(F.u), C.mu = R(F.mu),
// pressure, boundary conditions, uprev = u, pressure again
template <bool B>
__global__ void k_restrict_state(CaseArg<B, Params> P_, CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_) {
    FLITE_CASE_P(B, P, C);
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    FLITE_CHILD_LANES(7);
    const int N = C.N;
    const size_t n = F.N;
    const double *const src[7] = {F.u, F.u + n, F.u + 2 * n, F.u + 3 * n, F.u + 4 * n, F.mu, P.sa ? F.u + 5 * n : F.u};
    double v[7];
    restrict_group<7>(C, c, active, gl, gs, src, v);
    if (!active || gl) return;
    C.mu[c] = v[5];
    double p0 = pressure(P, v[0], v[1], v[2], v[3], v[4]);
    const unsigned char cls = C.bc[c];
    double n0 = 0, n1 = 0, n2 = 0;
    if (cls != BC_NONE) { n0 = C.nx[c]; n1 = C.ny[c]; n2 = C.nz[c]; }
    bc_solution(P, cls, n0, n1, n2, 0.0, 0.0, 0.0, relax_param(P, *C.cyc), v);
    const double rp = eo_relax(P, *C.cyc);
    if (is_exhaust(cls)) bc_exhaust(P, cls, rp, v);
    bc_outer(P, cls, n0, n1, n2, p0, v);
    for (int k = 0; k < 5; ++k) { C.u[k * N + c] = v[k]; C.uprev[k * N + c] = v[k]; }
    if (P.sa) {
        const double t = sa_bc_solution(P, cls, rp, v[6]);
        C.u[5 * N + c] = t;
        C.uprev[5 * N + c] = t;
    }
    const double p = fabs(pressure(P, v[0], v[1], v[2], v[3], v[4]));
    C.p[c] = p;
    store_node(C.q, c, v[0], v[1], v[2], v[3], v[4], p);
    if (C.saprim) store_saprim(C, c, v[0], v[1], v[2], v[3]);
    if (C.prim) {  // the viscous primitives (k_state_pass)
        const double gOg = P.gamma / (P.gamma - 1.0);
        C.prim[c] = v[1] / v[0];
        C.prim[N + c] = v[2] / v[0];
        C.prim[2 * N + c] = v[3] / v[0];
        C.prim[3 * N + c] = gOg * p / v[0];
    }
}

// restrictGrid tail (def_par:12385-12427): C.rhs = R(F.rhs), increment
// conditions, src -= rhs, u += rhs
template <bool B>
__global__ void k_restrict_incr(CaseArg<B, Params> P_, CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_,
                                int floor_fine) {
    FLITE_CASE_P(B, P, C);
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    FLITE_CHILD_LANES(6);
    const int N = C.N;
    // the density floor that the fine node pass left (IO_LATER)
    if (floor_fine && active)
        for (int q = C.child_ptr[c] + gl; q < C.child_ptr[c + 1]; q += U) {
            const int f = C.child[q];
            if (F.u[f] < P.minRho) F.u[f] = P.minRho;
        }
    const size_t n = F.N;
    const double *const in[6] = {F.rhs,         F.rhs + n,     F.rhs + 2 * n,
                                 F.rhs + 3 * n, F.rhs + 4 * n, P.sa ? F.rhs + 5 * n : F.rhs};
    double r[6];
    restrict_group<6>(C, c, active, gl, gs, in, r);
    if (!active || gl) return;
    const unsigned char cls = C.bc[c];
    double n0 = 0, n1 = 0, n2 = 0;
    if (cls != BC_NONE) { n0 = C.nx[c]; n1 = C.ny[c]; n2 = C.nz[c]; }
    bc_increment(P, cls, n0, n1, n2, r);
    for (int k = 0; k < 5; ++k) {
        C.rhs[k * N + c] = r[k];
        C.src[k * N + c] = C.src[k * N + c] - r[k];
        C.u[k * N + c] = C.u[k * N + c] + r[k];
    }
    if (P.sa) {
        const double t = sa_bc_increment(P, cls, r[5]);
        C.rhs[5 * N + c] = t;
        C.src[5 * N + c] = C.src[5 * N + c] - t;
        C.u[5 * N + c] = C.u[5 * N + c] + t;
    }
}

// prolongateGrid coarse part (def_par:12445-12468): uprev = R(F.u) with the
// solution conditions, rhs = u - uprev with the increment conditions
// v: the restricted solution (and nu~); r: the correction (and nu~'s)
__device__ __forceinline__ void prolong_coarse(const Params &P, const LevelView &C, int c, double *v, double *r,
                                               bool store) {
    const int N = C.N;
    const unsigned char cls = C.bc[c];
    double n0 = 0, n1 = 0, n2 = 0;
    if (cls != BC_NONE) { n0 = C.nx[c]; n1 = C.ny[c]; n2 = C.nz[c]; }
    bc_solution(P, cls, n0, n1, n2, 0.0, 0.0, 0.0, relax_param(P, *C.cyc), v);
    const double rp = eo_relax(P, *C.cyc);
    if (is_exhaust(cls)) bc_exhaust(P, cls, rp, v);
    bc_outer(P, cls, n0, n1, n2, C.p[c], v);
    for (int k = 0; k < 5; ++k) {
        if (store) C.uprev[k * N + c] = v[k];
        r[k] = C.u[k * N + c] - v[k];
    }
    double r6 = 0.0;
    if (P.sa) {
        const double t = sa_bc_solution(P, cls, rp, v[5]);
        if (store) C.uprev[5 * N + c] = t;
        r6 = C.u[5 * N + c] - t;
        // nullifyOuterBoundary, then the increment conditions
        if (cls == BC_FAR3 || is_engine(cls)) { r[0] = r[1] = r[2] = r[3] = r[4] = 0.0; r6 = 0.0; }
        r6 = sa_bc_increment(P, cls, r6);
    }
    bc_increment(P, cls, n0, n1, n2, r);
    r[5] = r6;
    if (!store) return;
    for (int k = 0; k < 5; ++k) C.rhs[k * N + c] = r[k];
    if (P.sa) C.rhs[5 * N + c] = r6;
}
template <bool B>
__global__ void k_prolong_coarse(CaseArg<B, Params> P_, CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_) {
    FLITE_CASE_P(B, P, C);
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    FLITE_CHILD_LANES(6);
    const size_t n = F.N;
    const double *const src[6] = {F.u, F.u + n, F.u + 2 * n, F.u + 3 * n, F.u + 4 * n, P.sa ? F.u + 5 * n : F.u};
    double v[6], r[6];
    restrict_group<6>(C, c, active, gl, gs, src, v);
    if (active && gl == 0) prolong_coarse(P, C, c, v, r, true);
}

// prolongateGrid fine part (def_par:12470-12567): injection, relaxation,
// u += correction, boundary conditions, floors
// corr: the parent's correction (and nu~'s)
__device__ __forceinline__ void prolong_fine(const Params &P, const LevelView &F, int i, const double *corr) {
    const int N = F.N;
    const unsigned char cls = F.bc[i];
    // nullifyOuterBoundary of the injected correction (SA runs only)
    const bool nul = P.sa && (cls == BC_FAR3 || is_engine(cls));
    double un[5];
    for (int k = 0; k < 5; ++k) un[k] = F.u[k * N + i];
    for (int k = 0; k < 5; ++k) {
        double r = corr[k];
        if (nul) r = 0.0;
        r = P.prolRelax * r;
        if (i < F.Nb) r = P.mgBCRelax * r;
        F.rhs[k * N + i] = r;
        un[k] = un[k] + r;
    }
    double un6 = 0.0;
    if (P.sa) {
        double r = corr[5];
        if (nul) r = 0.0;
        r = P.turbProlRelax * r;
        F.rhs[5 * N + i] = r;
        un6 = F.u[5 * N + i];
        // the nu~ correction reaches the levels finer than
        // numberOfTurbulenceGrids (def_par:12540-12552)
        if (F.grid < P.nTurbGrids) un6 = un6 + r;
        un6 = sa_bc_solution(P, cls, eo_relax(P, *F.cyc), un6);
        un6 = dmax(un6, 0.0);
        F.u[5 * N + i] = un6;
    }
    double n0 = 0, n1 = 0, n2 = 0;
    if (cls != BC_NONE) { n0 = F.nx[i]; n1 = F.ny[i]; n2 = F.nz[i]; }
    double cm0 = 0, cm1 = 0, cm2 = 0;
    if (cls == BC_WALL && P.viscous && F.grid == 1) { cm0 = F.cmx[i]; cm1 = F.cmy[i]; cm2 = F.cmz[i]; }
    bc_solution(P, cls, n0, n1, n2, cm0, cm1, cm2, relax_param(P, *F.cyc), un);
    if (is_exhaust(cls)) {
        const double pex = bc_exhaust(P, cls, eo_relax(P, *F.cyc), un);
        if (F.eng.f) F.eng.pbc[i] = pex;
    }
    if (F.eng.f && (P.eftype == 2 || is_engine(cls))) {  // completed by k_engine_finish
        for (int k = 0; k < 5; ++k) F.u[k * N + i] = un[k];
        return;
    }
    bc_outer(P, cls, n0, n1, n2, F.p[i], un);
    un[0] = dmax(un[0], P.minRho);
    for (int k = 0; k < 5; ++k) F.u[k * N + i] = un[k];
}
template <bool B>
__global__ void k_prolong_fine(CaseArg<B, Params> P_, CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_) {
    FLITE_CASE_P(B, P, C);
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    const int i = tid();
    if (i >= F.N) return;
    const int pc = C.parent[i];
    double corr[6] = {0, 0, 0, 0, 0, 0};
    for (int k = 0; k < F.nvar; ++k) corr[k] = pc >= 0 ? C.rhs[k * C.N + pc] : F.rhs[k * F.N + i];
    prolong_fine(P, F, i, corr);
}
// both parts in one launch where every fine node has a parent: a coarse
// node's lanes gather its children for the coarse part, then correct them.
// No other group reads or writes these children.
template <bool B>
__global__ void k_prolong(CaseArg<B, Params> P_, CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_) {
    FLITE_CASE_P(B, P, C);
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    FLITE_CHILD_LANES(6);
    const size_t n = F.N;
    const double *const src[6] = {F.u, F.u + n, F.u + 2 * n, F.u + 3 * n, F.u + 4 * n, P.sa ? F.u + 5 * n : F.u};
    double v[6], r[6];
    restrict_group<6>(C, c, active, gl, gs, src, v);
    if (!active) return;
    // every lane forms the correction; one stores the coarse arrays
    prolong_coarse(P, C, c, v, r, gl == 0);
    for (int q = C.child_ptr[c] + gl; q < C.child_ptr[c + 1]; q += U) prolong_fine(P, F, C.child[q], r);
}

// mapCoarseToFine of the solution (injection, def_par:12694-12700)
template <bool B>
__global__ void k_inject_u(CaseArg<B, LevelView> C_, CaseArg<B, LevelView> F_) {
    FLITE_CASE_L(B, C);
    FLITE_CASE_L(B, F);
    int i = tid();
    if (i >= F.N) return;
    int pc = C.parent[i];
    if (pc < 0) return;
    for (int k = 0; k < F.nvar; ++k) F.u[k * F.N + i] = C.u[k * C.N + pc];
}

// setBCsOnSolutionField on a level's solution (start-up, def_par:3994)
__global__ void k_bc_solution(Params P, LevelView L) {
    int i = tid();
    if (i >= L.N) return;
    const unsigned char cls = L.bc[i];
    if (cls == BC_NONE) return;
    const int N = L.N;
    double un[5];
    for (int k = 0; k < 5; ++k) un[k] = L.u[k * N + i];
    double cm0 = 0, cm1 = 0, cm2 = 0;
    if (cls == BC_WALL && P.viscous) { cm0 = L.cmx[i]; cm1 = L.cmy[i]; cm2 = L.cmz[i]; }
    bc_solution(P, cls, L.nx[i], L.ny[i], L.nz[i], cm0, cm1, cm2, relax_param(P, *L.cyc), un);
    if (is_exhaust(cls)) {
        const double rp = eo_relax(P, *L.cyc);
        const double pex = bc_exhaust(P, cls, rp, un);
        if (L.eng.f) L.eng.pbc[i] = pex;
        if (P.sa) L.u[5 * N + i] = sa_exhaust(P, cls, rp);
    }
    for (int k = 0; k < 5; ++k) L.u[k * N + i] = un[k];
    if (P.sa && (cls == BC_WALL || cls == BC_IWALL)) L.u[5 * N + i] = 0.0;
}

__global__ void k_set_int(int *dst, const int *src) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *dst = *src;
}

// ivd%physicalTimeStep = the smallest local time step of the level
// (makeTimeSteps under explicit time stepping, def_par:13598-13607): the
// minimum of positive doubles as the minimum of their bit patterns, which
// integer atomics take in any order to the same value.  k_min_dt_init
// starts it at the reference's 9999999.9.
__global__ void k_min_dt_init(LevelView L) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *L.ptsg = 9999999.9;
}
__global__ void k_min_dt(LevelView L) {
    __shared__ unsigned long long m[256];
    unsigned long long v = __double_as_longlong(9999999.9);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.N; i += gridDim.x * blockDim.x) {
        const double d = L.dt[i];
        if (d < __longlong_as_double((long long)v)) v = (unsigned long long)__double_as_longlong(d);
    }
    m[threadIdx.x] = v;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w && m[threadIdx.x + w] < m[threadIdx.x]) m[threadIdx.x] = m[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicMin(reinterpret_cast<unsigned long long *>(L.ptsg), m[0]);
}

// The same steps of the multigrid cycle on a level's view, so that a case
// group runs them for every case in one launch: the level's cycle number
// (doTimeIterations), uprev = u over n = nvar N values, and the zeroed
// dissipation (which 0) or FAS source (which 1) over n values.
template <bool B>
__global__ void k_case_cycle(CaseArg<B, LevelView> L_, const int *src) {
    FLITE_CASE_L(B, L);
    if (threadIdx.x == 0 && blockIdx.x == 0) *L.cyc = *src;
}
template <bool B>
__global__ void k_case_save_u(CaseArg<B, LevelView> L_, size_t n) {
    FLITE_CASE_L(B, L);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) L.uprev[i] = L.u[i];
}
template <bool B>
__global__ void k_case_zero(CaseArg<B, LevelView> L_, int which, size_t n) {
    FLITE_CASE_L(B, L);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) (which ? L.src : L.diss)[i] = 0.0;
}
template __global__ void k_case_cycle<false>(LevelView, const int *);
template __global__ void k_case_cycle<true>(CaseTab<LevelView>, const int *);
template __global__ void k_case_save_u<false>(LevelView, size_t);
template __global__ void k_case_save_u<true>(CaseTab<LevelView>, size_t);
template __global__ void k_case_zero<false>(LevelView, int, size_t);
template __global__ void k_case_zero<true>(CaseTab<LevelView>, int, size_t);

// ---- block sums -----------------------------------------------------------
// The sum of v[0..255] by halving (v[t] += v[t + w], w = 128, 64, ..., 1), by
// one warp: the pairs of the first three halvings are added from shared
// memory, the rest by shuffles, with one barrier before instead of eight.
__device__ __forceinline__ double sum256(const double *v, int lane) {
    const double a = (v[lane] + v[lane + 128]) + (v[lane + 64] + v[lane + 192]);
    const double b = (v[lane + 32] + v[lane + 160]) + (v[lane + 96] + v[lane + 224]);
    double s = a + b;
    for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
    return s;  // lane 0's
}

// ---- residual norms (writeResiduals mg_par:1299-1443) ---------------------
// per block: sum (u-uprev)^2 and max |u-uprev| with its first index; a batch
// takes all its cases in one launch (the case in blockIdx.y)
template <bool B>
__global__ void __launch_bounds__(256, 2) k_resid_partial(CaseArg<B, LevelView> L_, double *part) {
    FLITE_CASE_L(B, L);
    __shared__ double ss[6][256];
    __shared__ double sm[6][256];
    __shared__ int si[6][256];
    const int N = L.N, nv = L.nvar;
    double s[6] = {0, 0, 0, 0, 0, 0}, m[6] = {0, 0, 0, 0, 0, 0};
    int mi[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff};
    // the loads of two nodes at a time, all before the first sum: with a node's
    // components read one after another the pass took 97 us on 815,425 nodes,
    // with the loads of two nodes together 32 us (2 to 4 nodes: the same)
    const int step = gridDim.x * blockDim.x;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < N; i0 += 2 * step) {
        double d[2][6];
        int oi[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = i0 + q * step;
            if (i >= N) break;
            // the first node in the caller's numbering wins a tie (mg_par:1387-1396)
            oi[q] = L.perm ? L.perm[i] : i;
#pragma unroll
            for (int k = 0; k < 5; ++k) d[q][k] = L.u[(size_t)k * N + i] - L.uprev[(size_t)k * N + i];
            d[q][5] = nv == 6 ? L.u[5 * (size_t)N + i] - L.uprev[5 * (size_t)N + i] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (i0 + q * step >= N) break;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const double a = fabs(d[q][k]);
                s[k] = s[k] + a * a;
                if (a > m[k] || (a == m[k] && a > 0.0 && oi[q] < mi[k])) { m[k] = a; mi[k] = oi[q]; }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) { ss[k][threadIdx.x] = s[k]; sm[k][threadIdx.x] = m[k]; si[k][threadIdx.x] = mi[k]; }
    __syncthreads();
    // a warp per component
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= 6) return;
    const double sum = sum256(ss[k], lane);
    double v = 0.0;
    int iv = 0x7fffffff;
#pragma unroll
    for (int t = lane; t < 256; t += 32)
        if (sm[k][t] > v || (sm[k][t] == v && si[k][t] < iv)) { v = sm[k][t]; iv = si[k][t]; }
    for (int w = 16; w > 0; w >>= 1) {
        const double b = __shfl_down_sync(0xffffffffu, v, w);
        const int ib = __shfl_down_sync(0xffffffffu, iv, w);
        if (b > v || (b == v && ib < iv)) { v = b; iv = ib; }
    }
    if (lane == 0) {
        double *o = part + ((size_t)blockIdx.y * kResidBlocks + blockIdx.x) * 18;
        o[k] = sum;
        o[6 + k] = v;
        o[12 + k] = (double)iv;
    }
}
template __global__ void k_resid_partial<false>(LevelView, double *);
template __global__ void k_resid_partial<true>(CaseTab<LevelView>, double *);

// one warp per component (blockDim.x = 192), a block per case; each lane folds
// the block partials b = lane, lane+32, ... and the warp combines the lanes in
// a fixed tree, so the result does not depend on timing
__global__ void k_resid_final(const double *part, double *out) {
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= 6) return;
    part += (size_t)blockIdx.x * kResidBlocks * 18;
    out += (size_t)blockIdx.x * 18;
    double s = 0, m = 0;
    int mi = 0x7fffffff;
#pragma unroll
    for (int b0 = 0; b0 < kResidBlocks; b0 += 32) {
        const int b = b0 + lane;
        if (b >= kResidBlocks) break;
        s += part[b * 18 + k];
        double v = part[b * 18 + 6 + k];
        int iv = (int)part[b * 18 + 12 + k];
        if (v > m || (v == m && iv < mi)) { m = v; mi = iv; }
    }
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, off);
        double v = __shfl_down_sync(0xffffffffu, m, off);
        int iv = __shfl_down_sync(0xffffffffu, mi, off);
        if (v > m || (v == m && iv < mi)) { m = v; mi = iv; }
    }
    if (lane == 0) {
        out[k] = sqrt(s);
        out[6 + k] = m;
        out[12 + k] = (double)(mi == 0x7fffffff ? 0 : mi);
    }
}

// ---- forces (calculateLiftAndDrag def_par:14710-14805): block partials ---
// part[6*block + k]; k_forces_final sums the partials in block order
__global__ void k_forces(Params P, LevelView L, const int *wall, int nwall, double alphaR, double betaR,
                         double ground, double d0, double d1, double d2, double *part) {
    __shared__ double red[6][256];
    double ft[3] = {cos(alphaR) * cos(betaR), sin(betaR), sin(alphaR)};
    double fn1[3] = {-ft[2], 0.0, ft[0]}, fn2[3] = {-ft[1], ft[0], 0.0};
    double acc[6] = {0, 0, 0, 0, 0, 0};
    const double pinf = 1. / (P.gamma * P.mach * P.mach);
    const int N = L.N;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nwall; q += gridDim.x * blockDim.x) {
        int ip = wall[q];
        double h = L.cz[ip];
        if (!(h > (ground + 0.01))) continue;
        double xd = L.cx[ip] - d0, yd = L.cy[ip] - d1, zd = L.cz[ip] - d2;
        double n[3] = {L.nx[ip], L.ny[ip], L.nz[ip]};
        double A = L.wallArea[ip], dp = L.p[ip] - pinf;
        double dn1 = (n[0] * fn1[0] + n[1] * fn1[1]) + n[2] * fn1[2];
        double dn2 = (n[0] * fn2[0] + n[1] * fn2[1]) + n[2] * fn2[2];
        double dt = (n[0] * ft[0] + n[1] * ft[1]) + n[2] * ft[2];
        acc[0] -= A * dp * dn1;
        acc[1] -= A * dp * dt;
        acc[2] -= A * dp * dn2;
        acc[4] += xd * A * dp * dn2 - yd * A * dp * dt;
        acc[5] += xd * A * dp * dn1 - zd * A * dp * dt;
        if (P.viscous) {
            double s0 = L.wstress[ip], s1 = L.wstress[N + ip], s2 = L.wstress[2 * N + ip];
            double sn1 = (s0 * fn1[0] + s1 * fn1[1]) + s2 * fn1[2];
            double sn2 = (s0 * fn2[0] + s1 * fn2[1]) + s2 * fn2[2];
            double st = (s0 * ft[0] + s1 * ft[1]) + s2 * ft[2];
            acc[0] += A * sn1;
            acc[2] += A * sn2;
            acc[1] += A * st;
            acc[3] += A * st;
            acc[4] += -xd * A * sn2 + yd * A * st;
            acc[5] += -xd * A * sn1 + zd * A * st;
        }
    }
    for (int k = 0; k < 6; ++k) red[k][threadIdx.x] = acc[k];
    __syncthreads();
    const int kw = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (kw >= 6) return;
    const double sum = sum256(red[kw], lane);
    if (lane == 0) part[6 * blockIdx.x + kw] = sum;
}

__global__ void k_permute_nodes(double *dst, const double *src, const int *map, int N, int ncomp) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)N * ncomp) return;
    const int c = (int)(t / N), i = (int)(t - (size_t)c * N);
    dst[t] = src[(size_t)c * N + map[i]];
}

// ---- forces of forceCalcType 3 (calculateLiftAndDrag3 def_par:15129-15313)
// Per wall node (indicator register -20..-19) the face loads of its wall and
// inviscid-wall faces (codes 1, 9) with a node above the ground plane, in
// boundary-edge order as the reference's scatter adds them: 4 w_b (p - p_inf)
// and, in viscous runs on code-1 faces, 4 tau_w |w_b|.  Then the seven sums
// part[7*block + k] = (lift, drag, latF, latM, longMl, longMd, rollM).
__global__ void k_forces3(Params P, LevelView L, const int *wall, int nwall, double alphaR, double betaR,
                          double ground, double d0, double d1, double d2, double *part) {
    __shared__ double red[7][256];
    double ft[3] = {cos(alphaR) * cos(betaR), sin(betaR), sin(alphaR)};
    double fn1[3] = {-ft[2], 0.0, ft[0]}, fn2[3] = {-ft[1], ft[0], 0.0};
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    const double pinf = 1. / (P.gamma * P.mach * P.mach);
    const int N = L.N;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nwall; q += gridDim.x * blockDim.x) {
        const int ip = wall[q];
        double h0 = 0.0, h1 = 0.0, h2 = 0.0;
        for (int k = L.binc_ptr[ip]; k < L.binc_ptr[ip + 1]; ++k) {
            const int b = L.binc[k] >> 1;
            const int code = L.bind[b];
            if (!(code == 1 || code == 9)) continue;
            const int2 nd = L.bedge[b];
            if (!((L.cz[nd.x] > (ground + 0.01)) || (L.cz[nd.y] > (ground + 0.01)))) continue;
            const double pp = L.p[ip] - pinf;
            const double wx = L.bwx[b], wy = L.bwy[b], wz = L.bwz[b];
            h0 = h0 + 4.0 * wx * pp;
            h1 = h1 + 4.0 * wy * pp;
            h2 = h2 + 4.0 * wz * pp;
            if (P.viscous && code == 1) {
                const double area = sqrt((wx * wx + wy * wy) + wz * wz);
                h0 = h0 + 4.0 * L.wstress[ip] * area;
                h1 = h1 + 4.0 * L.wstress[N + ip] * area;
                h2 = h2 + 4.0 * L.wstress[2 * N + ip] * area;
            }
        }
        const double xd = L.cx[ip] - d0, yd = L.cy[ip] - d1, zd = L.cz[ip] - d2;
        const double hn1 = (h0 * fn1[0] + h1 * fn1[1]) + h2 * fn1[2];
        const double hn2 = (h0 * fn2[0] + h1 * fn2[1]) + h2 * fn2[2];
        const double ht = (h0 * ft[0] + h1 * ft[1]) + h2 * ft[2];
        acc[0] += hn1;
        acc[1] += ht;
        acc[2] += hn2;
        acc[3] += -xd * hn2 + yd * ht;
        acc[4] += -xd * hn1;
        acc[5] += zd * ht;
        acc[6] += -yd * hn1 + zd * hn2;
    }
    for (int k = 0; k < 7; ++k) red[k][threadIdx.x] = acc[k];
    __syncthreads();
    const int kw = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (kw >= 7) return;
    const double sum = sum256(red[kw], lane);
    if (lane == 0) part[7 * blockIdx.x + kw] = sum;
}

// out[k] = sum over blocks of part[nval*block + k], in block order
__global__ void k_forces_final(const double *part, int nval, double *out) {
    if (threadIdx.x >= nval) return;
    const int k = threadIdx.x;
    double s = 0.0;
#pragma unroll 16
    for (int b = 0; b < kForceBlocks; ++b) s += part[nval * b + k];
    out[k] = s;
}
}  // namespace flite
