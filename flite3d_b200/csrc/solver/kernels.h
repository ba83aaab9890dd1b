// Kernel declarations shared by the host orchestration.
#pragma once
#include "device.cuh"

namespace flite {

// node passes: an RK stage, restrictGrid's coarse and fine one-step updates,
// makeRHS alone; MODE_PROLONG and MODE_START name prolongateGrid's fine part
// and the start-up conditions for the engine pass that follows them
enum { MODE_STAGE = 0, MODE_RCOARSE = 1, MODE_RFINE = 2, MODE_RESID = 3, MODE_PROLONG = 4, MODE_START = 5 };

// the pass over a level's state before its gathers: pressure and node records
// (STATE_REC), the velocities of the HLLC gradients (STATE_HPRIM), with
// STATE_PRIM the viscous primitives, with STATE_STEP the
// start of a relaxation step (cycle number from src, uprev = u); BND adds the
// boundary edges' fluxes (threads N.. of the grid, one edge each)
enum { STATE_PRIM = 1, STATE_STEP = 2, STATE_REC = 4, STATE_HPRIM = 8 };
template <bool BND, bool B = false>
__global__ void k_state_pass(CaseArg<B, Params> P, CaseArg<B, LevelView> L, int what, const int *src);
template <int U, bool B = false>
__global__ void k_timestep(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_jst_lap(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_jst_flux(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U>
__global__ void k_first_order_diss(Params P, LevelView L);
template <int U, bool B = false>
__global__ void k_visc_grad(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_visc_flux(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_ts_lap(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_jflux_vgrad(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_visc2_grad(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
template <int U, bool B = false>
__global__ void k_visc2_flux(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
__global__ void k_fill(double *a, size_t n, double v);
template <bool MINMAX>
__global__ void k_gradient(Params P, LevelView L);
__global__ void k_jst_flux_matrix(Params P, LevelView L);
__global__ void k_lp_sums(Params P, LevelView L);
__global__ void k_lp_flux(Params P, LevelView L);
__global__ void k_prim_rec(LevelView L);
__global__ void k_gradient_rec(LevelView L);
constexpr int kMusclThreads = 128;
__global__ void k_edge_flux_muscl(Params P, LevelView L);
__global__ void k_ls_gradient(Params P, LevelView L);
__global__ void k_minmax(Params P, LevelView L);
constexpr int edge_threads(int ft, bool o2) { return ft == 4 && o2 ? 128 : 256; }
template <int FT, bool O2>
__global__ void k_edge_flux(Params P, LevelView L);
template <bool B = false>
__global__ void k_bnd_flux(CaseArg<B, Params> P, CaseArg<B, LevelView> L);
// GATHER_LEAN: GATHER_CENTRAL for runs without engine conditions and
// without explicit time stepping, whose node tail leaves those branches out
// (they cost the thread-per-node form its last free registers)
enum { GATHER_BUFFER = 0, GATHER_CENTRAL = 1, GATHER_ANCHOR = 2, GATHER_DELTA = 3, GATHER_LEAN = 5 };
// the gathers that copy ahead with a thread per node run blocks of at most
// 128 threads
constexpr bool central_ahead(int prec) { return prec == GATHER_CENTRAL || prec == GATHER_ANCHOR || prec == GATHER_LEAN; }
constexpr int node_threads(int prec, int u) { return u == 1 && central_ahead(prec) ? 128 : 256; }
// What a node pass computes of the dissipation before its residual (lanes per
// node only): nothing, the scalar JST flux, or the viscous fluxes, both
// otherwise their own launches
enum { PRE_NONE = 0, PRE_JST = 1, PRE_VISC = 2 };
// Which copies of the state a node pass reads and writes (a word of flags).
// The stages of a step alternate them, so that a stage can write its node's
// new state, pressure and records in the launch whose other nodes still read
// the old ones: no pressure pass between the stages, and with lanes per node
// (which evaluate the boundary edges themselves, IO_BND) one launch a stage.
//   stage    1               2            3            (4 as 2, 5 as 3)
//   u        uprev -> u      u -> ub      ub -> u      with IO_BND, else u -> u
//   records  q -> qb         qb -> q      q            (none after the last)
enum {
    IO_UIN = 3,      // 0 u, 1 uprev, 2 ub
    IO_UOUT_B = 4,   // the new state goes to ub, else to u
    IO_REC_B = 8,    // records read from qb (dqb), else from q (dq)
    IO_EMIT = 16,    // the new pressure, and the records to the other copy
    IO_BND = 32,     // boundary edges evaluated in the pass, else from bflux
    IO_LATER = 64    // restrictGrid's fine pass leaves the density floor to k_restrict_incr
};
constexpr int stage_io(int stage, int nstage, bool bnd, bool emit) {
    return (bnd ? (stage == 1 ? 1 : stage % 2 ? 2 : 0) | (stage % 2 ? 0 : IO_UOUT_B) | IO_BND : 0) |
           (emit ? (stage % 2 ? 0 : IO_REC_B) | (stage < nstage ? IO_EMIT : 0) : 0);
}
template <int PREC, int U, int PRE = PRE_NONE, bool B = false>
__global__ void k_node_update(CaseArg<B, Params> P, CaseArg<B, LevelView> L, int mode, int stage, int io);
// gathers: U lanes per node (1 = a thread per node); by default the widest
// group with at most this many threads on the level (flite_ctx::lanes_of)
constexpr size_t kLaneThreads = 98304;
constexpr int kSharedWalkNodes = 220000;
constexpr int kMaxLevels = 16;
template <bool B = false>
__global__ void k_delta_state(CaseArg<B, LevelView> L);
// the turbulent time step (ts) and the nu~ gradient in one walk
template <int U>
__global__ void k_sa_grad(Params P, LevelView L, int ts);
template <int U>
__global__ void k_sa_diff(Params P, LevelView L);
template <int U>
__global__ void k_sa_conv(Params P, LevelView L, int td);
__global__ void k_sa_stage(Params P, LevelView L, int mode, int stage, int turb);
// set-up of a level's edges on the device (kernels.cu)
__global__ void k_make_rows(LevelView L, int nrows, int2 *rows);
__global__ void k_row_firsts(const int2 *rows, int nrows, int *first);
__global__ void __launch_bounds__(1024) k_scan_rows(int *first, int nrows);
__global__ void k_edge_slots(const int2 *rows, int nrows, const int *first, int *slot);
__global__ void k_renumber_edges(int2 *inc, int n, const int *slot);
__global__ void k_move_edges(int E, const int *slot, const int2 *in, int2 *out);
__global__ void k_put_edges(int E, const int *slot, const double *w, double *wx, double *wy, double *wz, EdgeW *ew);
__global__ void k_put_edge_values(int E, const int *slot, const double *in, double *out);
__global__ void k_make_inc32(const int2 *inc, const EdgeW *ew, int n, IncRec32 *o);
template <bool B = false>
__global__ void k_restrict_u(CaseArg<B, LevelView> C, CaseArg<B, LevelView> F);
__global__ void k_restrict_arr(LevelView C, LevelView F, const double *fsrc, double *cdst, int ncomp);
template <bool B = false>
__global__ void k_restrict_state(CaseArg<B, Params> P, CaseArg<B, LevelView> C, CaseArg<B, LevelView> F);
template <bool B = false>
__global__ void k_restrict_incr(CaseArg<B, Params> P, CaseArg<B, LevelView> C, CaseArg<B, LevelView> F, int floor_fine);
template <bool B = false>
__global__ void k_prolong(CaseArg<B, Params> P, CaseArg<B, LevelView> C, CaseArg<B, LevelView> F);
template <bool B = false>
__global__ void k_prolong_coarse(CaseArg<B, Params> P, CaseArg<B, LevelView> C, CaseArg<B, LevelView> F);
template <bool B = false>
__global__ void k_prolong_fine(CaseArg<B, Params> P, CaseArg<B, LevelView> C, CaseArg<B, LevelView> F);
template <bool B = false>
__global__ void k_inject_u(CaseArg<B, LevelView> C, CaseArg<B, LevelView> F);
__global__ void k_bc_solution(Params P, LevelView L);
// level-1 engine inlet terms after a node pass (engine.cu)
constexpr int kEngineLanes = 256;
__global__ void __launch_bounds__(kEngineLanes) k_engine_sums(Params P, LevelView L, int mode);
__global__ void k_engine_finish(Params P, LevelView L, int mode, int all);
__global__ void k_set_int(int *dst, const int *src);
// the explicit time step: the level's smallest local time step (256 threads a block)
__global__ void k_min_dt_init(LevelView L);
__global__ void k_min_dt(LevelView L);
// steps of the cycle on a level view (group form: every case of a group)
// lanes per coarse node of the transfers that gather its children
constexpr int kChildLanes = 8;
template <bool B = false>
__global__ void k_case_cycle(CaseArg<B, LevelView> L, const int *src);
template <bool B = false>
__global__ void k_case_save_u(CaseArg<B, LevelView> L, size_t n);
template <bool B = false>
__global__ void k_case_zero(CaseArg<B, LevelView> L, int which, size_t n);
constexpr int kResidBlocks = 296;  // 2 x 148 SMs, of 256 threads
template <bool B = false>
__global__ void k_resid_partial(CaseArg<B, LevelView> L, double *part);
__global__ void k_resid_final(const double *part, double *out);
__global__ void k_forces(Params P, LevelView L, const int *wall, int nwall, double alphaR, double betaR,
                         double ground, double d0, double d1, double d2, double *part);
// dst[c*N + i] = src[c*N + map[i]] for c < ncomp (node arrays between the
// caller's numbering and the device's)
__global__ void k_permute_nodes(double *dst, const double *src, const int *map, int N, int ncomp);
__global__ void k_forces3(Params P, LevelView L, const int *wall, int nwall, double alphaR, double betaR,
                          double ground, double d0, double d1, double d2, double *part);
__global__ void k_forces_final(const double *part, int nval, double *out);
constexpr int kForceBlocks = 64;
// transposed residual Jacobian at the state x (adjoint.cu)
template <int U>
__global__ void k_vjp_node(Params P, LevelView L, const double *x, const double *rbar, const double *bvjp,
                           const double *pbar, double *ubar, int add);

}  // namespace flite
