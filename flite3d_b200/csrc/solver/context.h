// Device context of one solve: the per-level device layout and the host
// orchestration that mirrors the reference's solver routines.  Shared by the
// single-solve ABI (flite_gpu.cu) and the batched one (batch.cu).
#pragma once
#include <cuda_runtime.h>

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "flite_gpu.h"
#include "kernels.h"

using namespace flite;

namespace flite {
// buffers of the steady adjoint (steady_adjoint.cu), made on its first call
struct SteadyAdjoint;
void destroy_steady_adjoint(SteadyAdjoint *a);
}  // namespace flite

namespace flite_detail {

struct cuda_error : std::runtime_error {
    using std::runtime_error::runtime_error;
};

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t _e = (call);                                                              \
        if (_e != cudaSuccess)                                                                \
            throw cuda_error(std::string(#call) + ": " + cudaGetErrorString(_e));             \
    } while (0)

constexpr int kBlock = 256;

// Pinned buffers for results to pageable arrays, shared by the process's
// contexts: taken for one call and returned (any thread, any device), at most
// kKeep kept, all freed with the last context.  Pinning 2 MB takes 1.4 to 3.3
// ms, as long as ten such results save.
class StagePool {
public:
    static constexpr size_t kBytes = (size_t)2 << 20;
    static StagePool &get() {
        static StagePool p;
        return p;
    }
    void enter() {
        std::lock_guard<std::mutex> g(m);
        ++users;
    }
    void leave() {
        std::lock_guard<std::mutex> g(m);
        if (--users > 0) return;
        for (char *b : free_) cudaFreeHost(b);
        free_.clear();
    }
    char *take() {
        {
            std::lock_guard<std::mutex> g(m);
            if (!free_.empty()) {
                char *b = free_.back();
                free_.pop_back();
                return b;
            }
        }
        void *b = nullptr;
        CK(cudaHostAlloc(&b, kBytes, cudaHostAllocPortable));
        return (char *)b;
    }
    void give(char *b) {
        {
            std::lock_guard<std::mutex> g(m);
            if (users > 0 && free_.size() < kKeep) {
                free_.push_back(b);
                return;
            }
        }
        cudaFreeHost(b);
    }

private:
    static constexpr size_t kKeep = 4;
    std::mutex m;
    std::vector<char *> free_;
    int users = 0;
};

struct DevLevel {
    int N = 0, E = 0, B = 0, Nb = 0;
    int nrows = 0;           // incidence rows
    bool orphans = false;    // coarse level: some finer node has no parent here
    LevelView v{};
    std::vector<int> wall;  // level-1 wall nodes in register order (forces)
    int *d_wall = nullptr;
};

}  // namespace flite_detail

using namespace flite_detail;

#define FLITE_UNPAREN(...) __VA_ARGS__
// a launch of kernel template `kern` (its other template arguments `targs`,
// parenthesised with a trailing comma, or ()) for this context, or in group
// form for every case of its group: the same grid for each case, the case
// in blockIdx.y
#define FLITE_LAUNCH(kern, targs, grid, block, smem, ...)                                                     \
    do {                                                                                                       \
        if (group) launch_group(kern<FLITE_UNPAREN targs true>, dim3((grid), group), (block), (smem), __VA_ARGS__); \
        else kern<FLITE_UNPAREN targs false><<<(grid), (block), (smem), s>>>(__VA_ARGS__);                     \
    } while (0)

// a gather kernel template launched with the lanes per node of level l
#define FLITE_GATHER(kern, l, ...)                                                       \
    do {                                                                                 \
        switch (lanes_of(l)) {                                                           \
            case 4: FLITE_LAUNCH(kern, (4,), gblk(l, 4), nb, 0, __VA_ARGS__); break;     \
            case 8: FLITE_LAUNCH(kern, (8,), gblk(l, 8), nb, 0, __VA_ARGS__); break;     \
            case 16: FLITE_LAUNCH(kern, (16,), gblk(l, 16), nb, 0, __VA_ARGS__); break;  \
            case 32: FLITE_LAUNCH(kern, (32,), gblk(l, 32), nb, 0, __VA_ARGS__); break;  \
            default: FLITE_LAUNCH(kern, (1,), gblk(l, 1), nb, 0, __VA_ARGS__);           \
        }                                                                                \
    } while (0)

// an adjoint gather with the lanes per node of level l of context X (blocks of
// at most 128 threads: its slabs hold up to 24 terms a lane)
#define FLITE_ADJ_GATHER(kern, X, l, ...)                                                                        \
    do {                                                                                                          \
        const int u_ = X.lanes_of(l), t_ = std::min(X.nb, 128);                                                    \
        const unsigned g_ = (unsigned)((u_ * (size_t)X.V(l).N + t_ - 1) / t_);                                     \
        switch (u_) {                                                                                              \
            case 4: kern<4><<<g_, t_, 0, X.s>>>(__VA_ARGS__); break;                                               \
            case 8: kern<8><<<g_, t_, 0, X.s>>>(__VA_ARGS__); break;                                               \
            case 16: kern<16><<<g_, t_, 0, X.s>>>(__VA_ARGS__); break;                                             \
            case 32: kern<32><<<g_, t_, 0, X.s>>>(__VA_ARGS__); break;                                             \
            default: kern<1><<<g_, t_, 0, X.s>>>(__VA_ARGS__);                                                     \
        }                                                                                                          \
    } while (0)

struct flite_ctx {
    flite_controls c{};
    Params P{};
    std::vector<DevLevel> lv;
    std::vector<void *> allocs;
    cudaStream_t s = nullptr;
    // Launches that do not depend on each other go to further streams (in a
    // captured cycle: branches of the graph): beside(k, f) runs f's launches
    // on stream k after what s holds now, join(k) makes s wait for them.
    // Streams: 0 restrictGrid's coarse part; 1 and 2 boundary fluxes and the
    // nu~ part of a pass; 3 and 4 those of the coarse part.
    static constexpr int kBranches = 5;
    cudaStream_t branch[kBranches] = {};
    cudaEvent_t forked[kBranches] = {}, done[kBranches] = {}, coarse_ready = nullptr;
    int pass_branch = 1;  // 3 within the coarse part
    template <class F>
    void beside(int k, F &&f) {
        struct On {  // s is the branch's stream in its scope
            cudaStream_t &a, &b;
            ~On() { std::swap(a, b); }
        };
        CK(cudaEventRecord(forked[k], s));
        CK(cudaStreamWaitEvent(branch[k], forked[k], 0));
        std::swap(s, branch[k]);
        On on{s, branch[k]};
        f();
        CK(cudaEventRecord(done[k], s));
    }
    void join(int k) { CK(cudaStreamWaitEvent(s, done[k], 0)); }
    int *d_cycle = nullptr;
    int *d_cyc = nullptr;  // per-level cycle numbers
    double *d_part = nullptr;
    double *d_ptsg = nullptr;  // ivd%physicalTimeStep (explicit time stepping)
    int *h_cycle = nullptr;    // pinned
    double *h_out = nullptr;  // pinned: the last kernel of a reduction writes here (kOut values)
    static constexpr int kOut = 2048;
    // a GMRES iteration leaves two passes of restart + 1 dot products and a norm there
    static constexpr int kMaxRestart = 500;
    static_assert(2 * (kMaxRestart + 1) + 1 <= kOut, "the GMRES results fit the pinned buffer");
    cudaGraphExec_t graph = nullptr;
    int64_t launches = 0;
    bool counting = false;
    // a case group (batch cases on one mesh, advanced together): while
    // `group` > 0 the cycle's launches run in group form for that many
    // cases, with every case's parameters and level views (gP, gV) in the
    // kernel's parameter bank.  Paths without a group form refuse it.
    int group = 0;
    CaseTab<Params> gP{};
    std::vector<CaseTab<LevelView>> gV;
    const CaseTab<Params> &to_group(const Params &) const { return gP; }
    const CaseTab<LevelView> &to_group(const LevelView &v) const {
        for (size_t l = 0; l < lv.size(); ++l)
            if (&lv[l].v == &v) return gV[l];
        throw std::runtime_error("a group launch argument is not one of the context's level views");
    }
    template <class T>
    const T &to_group(const T &x) const { return x; }
    template <class... KP, class... A>
    void launch_group(void (*k)(KP...), dim3 g, unsigned b, size_t sm, const A &...a) {
        k<<<g, b, sm, s>>>(to_group(a)...);
    }
    struct no_group_error : std::runtime_error {
        using std::runtime_error::runtime_error;
    };
    void no_group(const char *what) const {
        if (group) throw no_group_error(std::string(what) + " has no case-group form");
    }
    // threads per block of the edge kernels and of the node kernels (the
    // batch autotuner may change them; kernels with launch bounds take <= 256)
    // by default node kernels take blocks of 128: the separate gathers of the
    // 2.1-million-node level run 1736 us a step with 128 and 1821 with 256
    int eb = kBlock, nb = 128;
    // calculateTurbulence of the cycle being run or captured (Spalart-
    // Allmaras: cycleNo <= numberOfTurbulenceSteps, mg_par:922-926), and the
    // value the instantiated graph was captured with
    bool calcTurb = true, graphTurb = true;
    int nvar() const { return c.turbulenceModel == 1 ? 6 : 5; }
    bool sa() const { return c.turbulenceModel == 1; }
    bool turb() const { return sa() && calcTurb; }
    // set calcTurb for cycle `cyc`, dropping a graph captured with the other value
    void select_cycle(int cyc) {
        const bool t = !sa() || cyc <= c.numberOfTurbulenceSteps;
        if (graph && graphTurb != t) drop_graph();
        calcTurb = t;
    }
    // adjoint buffers (allocated on the first flite_residual_vjp)
    double *adj_rbar = nullptr, *adj_ubar = nullptr, *adj_b = nullptr;
    size_t adj_n = 0;
    void vjp_kernels(int l);
    flite::SteadyAdjoint *sadj = nullptr;
    // node numbering of the device (renumber.h): perm[l][new] = the caller's
    // number, iperm[l] its inverse; d_perm/d_iperm on the device (shared with
    // contexts that share this mesh); a scratch array for the permutations
    bool renumbered = false;
    // the mesh arrays are another context's (a batch case on a shared mesh)
    bool shares_mesh = false;
    std::vector<std::vector<int>> perm, iperm;
    std::vector<int *> d_perm, d_iperm;
    double *d_io = nullptr;
    size_t io_n = 0;
    double *io_buffer(size_t n) {
        if (io_n < n) {
            if (d_io) CK(cudaFree(d_io));
            d_io = nullptr;
            io_n = 0;
            CK(cudaMalloc(&d_io, n * sizeof(double)));
            io_n = n;
        }
        return d_io;
    }
    // ---- results to the caller's arrays ---------------------------------
    // A pageable array of more than kStageMin bytes whose pages are not there
    // yet is filled from the two halves of a pinned buffer (StagePool), one
    // emptied while the other is under way: 2.1 ms to 8.1 MB of fresh pages
    // where the driver's own path takes 3.5 (from pinned memory 0.16; the rest
    // is the page faults).  An array written before keeps the driver's path
    // where it is longer than a piece: 0.48 against 0.53 ms at 8.1 MB, 1.8
    // against 2.0 at 33 MB, 134 against 152 us at 2 MB; but 81 against 70 us at
    // 1 MB.  More threads for the copy cost more to start than they save, and
    // in the other direction the driver's path is the faster one (0.45 against
    // 0.54 ms).
    static constexpr size_t kStageMin = (size_t)1 << 18, kStagePiece = StagePool::kBytes / 2;
    cudaEvent_t staged[2] = {nullptr, nullptr};
    static bool pageable(const void *p, size_t n) {
        if (n < kStageMin) return false;
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }
    // whether the middle page of the n bytes at p (several pages) is there
    static bool touched(const void *p, size_t n) {
        const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
        unsigned char there = 1;
        return mincore((void *)(((uintptr_t)p + n / 2) & ~(page - 1)), page, &there) != 0 || (there & 1);
    }
    void to_host(void *dst, const void *src, size_t n) {
        if (!pageable(dst, n) || (n > kStagePiece && touched(dst, n))) {
            CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, s));
            return;
        }
        for (cudaEvent_t &e : staged)
            if (!e) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        struct Taken {
            cudaStream_t s;
            char *b;
            bool idle = false;  // no transfer into the buffer is under way
            ~Taken() {
                if (!idle) cudaStreamSynchronize(s);  // (an error on the way)
                StagePool::get().give(b);
            }
        } taken{s, StagePool::get().take()};
        char *stage = taken.b;
        const size_t pieces = (n + kStagePiece - 1) / kStagePiece;
        for (size_t j = 0; j <= pieces; ++j) {
            if (j < pieces) {  // on its way while the piece before is emptied
                const size_t k = j & 1, at = j * kStagePiece;
                CK(cudaMemcpyAsync(stage + k * kStagePiece, (const char *)src + at, std::min(kStagePiece, n - at),
                                   cudaMemcpyDeviceToHost, s));
                CK(cudaEventRecord(staged[k], s));
            }
            if (j > 0) {
                const size_t k = (j - 1) & 1, at = (j - 1) * kStagePiece;
                CK(cudaEventSynchronize(staged[k]));
                std::memcpy((char *)dst + at, stage + k * kStagePiece, std::min(kStagePiece, n - at));
            }
        }
        taken.idle = true;
    }
    // host [ncomp][N] in the caller's numbering -> device array in the
    // device's numbering (stream-ordered on s)
    void put_nodes(int l, double *dst, const double *host, int ncomp) {
        const size_t n = (size_t)lv[l].v.N * ncomp;
        if (!renumbered) {
            CK(cudaMemcpyAsync(dst, host, n * sizeof(double), cudaMemcpyHostToDevice, s));
            return;
        }
        double *t = io_buffer(n);
        CK(cudaMemcpyAsync(t, host, n * sizeof(double), cudaMemcpyHostToDevice, s));
        k_permute_nodes<<<blocks(n), kBlock, 0, s>>>(dst, t, d_perm[l], lv[l].v.N, ncomp);
        CK(cudaGetLastError());
    }
    // device array -> host [ncomp][N] in the caller's numbering (the copy is
    // stream-ordered on s: the caller synchronises before reading host)
    void get_nodes(int l, double *host, const double *src, int ncomp) {
        const size_t n = (size_t)lv[l].v.N * ncomp;
        if (!renumbered) {
            to_host(host, src, n * sizeof(double));
            return;
        }
        double *t = io_buffer(n);
        k_permute_nodes<<<blocks(n), kBlock, 0, s>>>(t, src, d_iperm[l], lv[l].v.N, ncomp);
        CK(cudaGetLastError());
        to_host(host, t, n * sizeof(double));
    }
    int adj_method = 1, adj_restart = 50;  // flite_set_adjoint_method (GMRES(50))
    std::string err;

    template <class T>
    T *alloc(size_t n) {
        void *p = nullptr;
        if (n == 0) n = 1;
        cudaError_t e = cudaMalloc(&p, n * sizeof(T));
        if (e != cudaSuccess) throw cuda_error(std::string("cudaMalloc: ") + cudaGetErrorString(e));
        allocs.push_back(p);
        return (T *)p;
    }
    template <class T>
    T *upload(const std::vector<T> &h) {
        T *d = alloc<T>(h.size());
        if (!h.empty()) CK(cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
        return d;
    }
    flite_ctx() { StagePool::get().enter(); }
    flite_ctx(const flite_ctx &) = delete;
    flite_ctx &operator=(const flite_ctx &) = delete;
    ~flite_ctx() {
        StagePool::get().leave();
        if (graph) cudaGraphExecDestroy(graph);
        if (adj_rbar) { cudaFree(adj_rbar); cudaFree(adj_ubar); cudaFree(adj_b); }
        if (sadj) flite::destroy_steady_adjoint(sadj);
        if (d_io) cudaFree(d_io);
        for (void *p : allocs) cudaFree(p);
        if (h_cycle) cudaFreeHost(h_cycle);
        if (h_out) cudaFreeHost(h_out);
        for (cudaEvent_t e : staged)
            if (e) cudaEventDestroy(e);
        for (int k = 0; k < kBranches; ++k) {
            if (forked[k]) cudaEventDestroy(forked[k]);
            if (done[k]) cudaEventDestroy(done[k]);
            if (branch[k]) cudaStreamDestroy(branch[k]);
        }
        if (coarse_ready) cudaEventDestroy(coarse_ready);
        if (s) cudaStreamDestroy(s);
    }

    static unsigned blocks(size_t n) { return (unsigned)((n + kBlock - 1) / kBlock); }
    unsigned nblk(size_t n) const { return (unsigned)((n + nb - 1) / nb); }
    unsigned eblk(size_t n) const { return (unsigned)((n + eb - 1) / eb); }
    void counted() {
        if (counting) ++launches;
    }

    // ---- single-grid building blocks ------------------------------------
    LevelView &V(int l) { return lv[l].v; }
    // lanes per node of each level's gathers (1, 4, 8, 16 or 32).  By
    // default the widest group that keeps the level's threads within
    // kLaneThreads: below that a thread per node leaves SMs idle and each
    // thread waits on a long chain of dependent loads, above it the extra
    // lanes only add instructions.  Kernels of one relaxation step (laminar,
    // flite_profile_kernels, us, lanes 1/4/8/16/32) on the bump channel's
    // agglomerated levels: 1,908 nodes 170/94/66/56/54, 21,972
    // 185/128/121/140/184, 237,662 313/555/738/1027/1623; on generated level-1
    // meshes 4,225 nodes 88/61/53/53/59, 14,161 90/67/70/82/113, 33,327
    // 92/94/108/143/214.  Whole cycles order them alike (four levels, 2,099,065
    // nodes: 6.39/6.22/6.21/6.38/6.84 ms by the lanes of the 21,972-node level).
    // A case group's cases share the launch.
    int lanes[kMaxLevels] = {0};
    int lanes_of(int l) const {
        if (l < kMaxLevels && lanes[l] > 0) return lanes[l];
        const size_t n = (size_t)lv[l].v.N * std::max(group, 1);
        for (int u = 32; u > 2; u /= 2)
            if (u * n <= kLaneThreads) return u;
        return 1;
    }
    unsigned gblk(int l, int g) const { return (unsigned)((g * (size_t)lv[l].v.N + nb - 1) / nb); }
    // levels whose gathers that walk the same incidence list share one walk
    // (k_ts_lap, k_jflux_vgrad) where a thread serves a node
    // (flite_set_gather_fusion: 1 on; 0 off, held as -1).  By default up to
    // kSharedWalkNodes nodes: there the walks are short of work and one launch
    // less pays; above, the separate kernels' smaller register counts do (one
    // step's kernels, shared/separate: 99,099 nodes 137/150 us, 206,400 nodes
    // 233/241, 242,219 nodes 283/271, 2,099,065 nodes 1661/1633)
    int fuse_mode[kMaxLevels] = {0};
    bool fuse_walks(int l) const {
        if (lanes_of(l) != 1) return false;
        if (l < kMaxLevels && fuse_mode[l] != 0) return fuse_mode[l] > 0;
        return lv[l].v.N <= kSharedWalkNodes;
    }

    // pass over the state of level l (STATE_*), with the boundary edges' fluxes
    // where `bnd`
    void state_pass(int l, int what, bool bnd = false) {
        const LevelView &L = V(l);
        if (fused()) what |= STATE_REC;  // only the central gathers read the records
        if (L.hprim) what |= STATE_HPRIM;
        counted();
        if (bnd)
            FLITE_LAUNCH(k_state_pass, (true,), nblk((size_t)L.N + L.B), nb, 0, P, L, what, (const int *)d_cycle);
        else
            FLITE_LAUNCH(k_state_pass, (false,), nblk(L.N), nb, 0, P, L, what, (const int *)d_cycle);
    }
    void pressure(int l) { state_pass(l, 0); }
    bool visc() const { return c.ReynoldsNumber > 0.0; }
    // passes of a level with lanes per node take their boundary fluxes from
    // the state pass or evaluate them in the node pass: the launch of the
    // boundary kernel costs these levels more than its work
    bool group_level(int l) const { return lanes_of(l) > 1; }
    // the node pass leaves the pressure (and records) of the next stage; with
    // engines the pass of the inlet nodes ends later (k_engine_finish)
    bool emits() const { return !P.engines; }
    // runs whose levels with lanes per node alternate the copies of the state:
    // the FP64 central flux of a static mesh without engines (the
    // Spalart-Allmaras kernels between the stages read the state in u)
    bool alternates() const { return fused() && !mixed() && !sa() && emits(); }
    // the node pass evaluates the boundary edges
    bool inline_bnd(int l) const { return group_level(l) && alternates(); }
    // makeTimeSteps's ivd%physicalTimeStep under explicit time stepping
    // (unsteady runs read it; steady ones never do)
    void explicit_step(int l) {
        if (!(P.explicit_ && P.unsteady)) return;
        no_group("explicit time stepping");
        counted();
        k_min_dt_init<<<1, 1, 0, s>>>(V(l));
        counted();
        k_min_dt<<<(unsigned)std::min<size_t>((V(l).N + 255) / 256, kResidBlocks), 256, 0, s>>>(V(l));
    }
    void timesteps(int l) {
        timestep_kernels(l);
        explicit_step(l);
    }
    void timestep_kernels(int l) {
        counted();
        FLITE_GATHER(k_timestep, l, P, V(l));
    }
    void zero_diss(int l) {
        counted();
        FLITE_LAUNCH(k_case_zero, (), nblk(5 * (size_t)V(l).N), nb, 0, V(l), 0, 5 * (size_t)V(l).N);
    }
    // makeArtificialDissipation2 (def_par:11484-11993), scalar form
    void jst(int l) {
        if (!jst_gathers(l)) {
            zero_diss(l);
            return;
        }
        jst_lap(l);
        jst_flux(l);
    }
    // the JST kernels run (not the zero dissipation of jst)
    bool jst_gathers(int l) {
        return !((c.fluxType == 4 && V(l).grid == 1) ||
                 (c.fourthOrderDissipationFactor == 0 && c.secondOrderDissipationFactor == 0));
    }
    void jst_lap(int l) {
        counted();
        FLITE_GATHER(k_jst_lap, l, P, V(l));
    }
    void jst_flux(int l) {
        counted();
        if (P.matrixDiss) {
            no_group("the matrix dissipation");
            k_jst_flux_matrix<<<nblk(V(l).N), nb, 0, s>>>(P, V(l));
        } else {
            FLITE_GATHER(k_jst_flux, l, P, V(l));
        }
    }
    // the walks that the scalar dissipation's passes of level l share: 0 none;
    // 1 time step and Laplacian (k_ts_lap); 2 also JST flux and viscous
    // gradients (k_jflux_vgrad).  With lanes per node they are always shared.
    int shared_walks(int l) {
        if (!(group_level(l) || fuse_walks(l)) || !jst_gathers(l)) return 0;
        return visc() && !P.matrixDiss && c.viscosityScheme == 1 ? 2 : 1;
    }
    // the part of the dissipation that is left to the node pass where it
    // evaluates the boundary edges (and so does not write the state it reads)
    int folded(int l, int walks) {
        if (!inline_bnd(l)) return PRE_NONE;
        return walks == 2 ? PRE_VISC : walks == 1 && !visc() && !P.matrixDiss ? PRE_JST : PRE_NONE;
    }
    void ts_lap(int l) {
        counted();
        FLITE_GATHER(k_ts_lap, l, P, V(l));
    }
    void jflux_vgrad(int l) {
        counted();
        FLITE_GATHER(k_jflux_vgrad, l, P, V(l));
    }
    // whether a relaxation step of level l takes its dissipation from
    // ts_jst_viscous (else from the separate kernels of `dissipation`)
    bool step_jst(int l) {
        return !((c.dissipationScheme == 1 && V(l).grid == 1) || c.dissipationScheme == 3);
    }
    // whether the state pass at the head of a relaxation step leaves the
    // boundary fluxes of its first stage
    bool step_bnd(int l) const { return group_level(l) && !inline_bnd(l) && c.flowType != 2; }
    // the time step (ts), the JST dissipation (or its zero) and the viscous
    // terms of a level, in the order of singleIteration and restrictGrid; the
    // viscous primitives, which only the gradients read, go before the JST
    // flux.  `prim`: they are there already.  With `fold` the last part may be
    // left to the node pass that follows (the PRE_* returned).
    int ts_jst_viscous(int l, bool ts, bool prim, bool fold) {
        const int walks = shared_walks(l);
        if (!walks) {
            if (ts) timesteps(l);
            jst(l);
            viscous(l, prim);
            return PRE_NONE;
        }
        if (ts) {
            ts_lap(l);
            explicit_step(l);
        } else {
            jst_lap(l);
        }
        if (visc() && !prim) viscous_prim(l);
        const int pre = fold ? folded(l, walks) : PRE_NONE;
        if (walks == 2) {
            jflux_vgrad(l);
            if (pre) return pre;
        } else {
            if (pre) return pre;
            jst_flux(l);
            if (visc()) {
                counted();
                visc_grad(l);
            }
        }
        if (visc()) {
            counted();
            visc_flux(l);
        }
        return PRE_NONE;
    }
    void first_order_diss(int l) {
        no_group("dissipation scheme 3");
        counted();
        k_first_order_diss<1><<<nblk(V(l).N), nb, 0, s>>>(P, V(l));
    }
    // dissipation choice of singleIteration (def_par:1030-1036)
    void dissipation(int l) {
        if (c.dissipationScheme == 1 && V(l).grid == 1) lp_diss(l);
        else if (c.dissipationScheme == 3) first_order_diss(l);
        else jst(l);
    }
    // makeArtificialDissipation1 (def_par:10706-11482), level 1 only
    void lp_diss(int l) {
        no_group("dissipation scheme 1");
        counted();
        k_lp_sums<<<nblk(V(l).N), nb, 0, s>>>(P, V(l));
        counted();
        k_lp_flux<<<nblk(V(l).N), nb, 0, s>>>(P, V(l));
    }
    void viscous_prim(int l) { state_pass(l, STATE_PRIM); }
    // makeViscosityTerm (def_par:5198-5893), subtracted from the dissipation
    void viscous(int l, bool prim = false) {
        if (!visc()) return;
        if (!prim) viscous_prim(l);
        counted();
        visc_grad(l);
        counted();
        visc_flux(l);
    }
    void visc_grad(int l) {
        if (c.viscosityScheme == 2) {  // makeViscosityTerm2 (def_par:5896-6807)
            FLITE_GATHER(k_visc2_grad, l, P, V(l));
            return;
        }
        FLITE_GATHER(k_visc_grad, l, P, V(l));
    }
    void visc_flux(int l) {
        if (c.viscosityScheme == 2) {
            FLITE_GATHER(k_visc2_flux, l, P, V(l));
            return;
        }
        FLITE_GATHER(k_visc_flux, l, P, V(l));
    }
    // ---- Spalart-Allmaras ----------------------------------------------
#define FLITE_SA(kern, l, ...)                                                           \
    do {                                                                                 \
        counted();                                                                       \
        switch (lanes_of(l)) {                                                           \
            case 4: kern<4><<<gblk(l, 4), nb, 0, s>>>(__VA_ARGS__); break;               \
            case 8: kern<8><<<gblk(l, 8), nb, 0, s>>>(__VA_ARGS__); break;               \
            case 16: kern<16><<<gblk(l, 16), nb, 0, s>>>(__VA_ARGS__); break;            \
            case 32: kern<32><<<gblk(l, 32), nb, 0, s>>>(__VA_ARGS__); break;            \
            default: kern<1><<<gblk(l, 1), nb, 0, s>>>(__VA_ARGS__);                     \
        }                                                                                \
    } while (0)
    // the turbulent time steps (ts), and the diffusion
    void sa_diffusion(int l, bool ts) {
        no_group("the Spalart-Allmaras model");
        FLITE_SA(k_sa_grad, l, P, V(l), ts ? 1 : 0);
        FLITE_SA(k_sa_diff, l, P, V(l));
    }
    // the nu~ part of a stage or one-step update; before the mean-flow node
    // update, which overwrites the density the source term reads
    void sa_stage(int l, int mode, int stage) {
        if (!sa()) return;
        no_group("the Spalart-Allmaras model");
        if (turb()) {
            FLITE_SA(k_sa_conv, l, P, V(l), P.addts && mode == MODE_STAGE ? 1 : 0);
        }
        counted();
        k_sa_stage<<<nblk(V(l).N), nb, 0, s>>>(P, V(l), mode, stage, turb() ? 1 : 0);
    }
    // makeRHS up to the node gather (def_par:1587-1607 and the edge loops);
    // with FLITE_MIXED, `anchor` selects the FP64 evaluation that refreshes
    // the anchor state, otherwise the FP32 increments over it
    // `delta`: the increments' records are there already, `bnd`: so are the
    // boundary fluxes, or the node pass evaluates them
    void rhs_terms(int l, bool anchor = true, bool delta = false, bool bnd = false) {
        const LevelView &L = V(l);
        if (c.reconstruction == FLITE_RECON_VAN_ALBADA && L.grid == 1) {
            // the extension reconstructs from the Galerkin gradients, through
            // the primitive and gradient records
            no_group("the reconstruction extension");
            counted();
            k_prim_rec<<<nblk(L.N), nb, 0, s>>>(L);
            counted();
            k_gradient_rec<<<nblk(L.N), nb, 0, s>>>(L);
        } else if (c.fluxType == 4 && c.HLLCFluxOrder > 1 && L.grid == 1) {
            no_group("the HLLC order-2 gradients");
            counted();
            if (c.GradientMethod == 1) {
                if (c.Automaticlipping == 1) k_gradient<true><<<nblk(L.N), nb, 0, s>>>(P, L);
                else k_gradient<false><<<nblk(L.N), nb, 0, s>>>(P, L);
            } else {
                k_ls_gradient<<<nblk(L.N), nb, 0, s>>>(P, L);
                if (c.Automaticlipping == 1) {
                    counted();
                    k_minmax<<<nblk(L.N), nb, 0, s>>>(P, L);
                }
            }
        }
        if (L.E > 0) {
            if (mixed() && !anchor && delta) {
            } else if (mixed() && !anchor) {
                // FP32 records of the increments over the anchor
                counted();
                FLITE_LAUNCH(k_delta_state, (), nblk(L.N), nb, 0, L);
            } else if (!fused()) {
                no_group("the upwind fluxes");
                counted();
                edge_flux_launch(L);
            }
        }
        if (!bnd) bnd_flux(l);
    }
    void bnd_flux(int l) {
        const LevelView &L = V(l);
        if (L.B <= 0) return;
        counted();
        FLITE_LAUNCH(k_bnd_flux, (), eblk(L.B), eb, 0, P, L);
    }
    // The residual's terms of a pass with their node update: the boundary
    // fluxes (where the pass neither has nor evaluates them) beside the edge
    // fluxes, and with Spalart-Allmaras the diffusion (`diff`: 0 none, 1, 2
    // with the turbulent time steps) and the nu~ part beside both.  With
    // `bnd_forked` the boundary fluxes are under way already.  The branches
    // pay where launches are short, the RANS cycle's four coarse levels, and
    // cost at the graph's instantiation: the boundary branches of the upwind
    // cycle on 14,161 nodes take 0.096 ms off each cycle (0.576 -> 0.480) and
    // put 1.15 ms on the first (1.32 -> 2.47), won back in twelve cycles; on
    // 203,401 nodes (W-cycle) 0.123 and 1.87 ms, fifteen.
    void residual_pass(int l, int mode, int stage, bool anchor, bool delta, bool bnd, bool bnd_forked, int diff, int pre,
                       int io) {
        const int kb = pass_branch, ks = pass_branch + 1;
        const bool fork_bnd = !bnd && !bnd_forked && !fused() && V(l).B > 0;
        if (fork_bnd) beside(kb, [&] { bnd_flux(l); });
        if (sa())
            beside(ks, [&] {
                if (turb() && diff) sa_diffusion(l, diff == 2);
                sa_stage(l, mode, stage);
            });
        rhs_terms(l, anchor, delta, bnd || bnd_forked || fork_bnd);
        if (fork_bnd || bnd_forked) join(kb);
        if (sa()) join(ks);
        node_update(l, mode, stage, anchor, pre, io);
        engine_pass(l, mode);
    }
    // the boundary fluxes beside the dissipation that precedes the pass
    bool bnd_beside(int l, bool bnd) {
        if (bnd || V(l).B <= 0) return false;
        beside(pass_branch, [&] { bnd_flux(l); });
        return true;
    }
    bool mixed() const { return c.precision == FLITE_MIXED; }
    // the central flux (and FLITE_MIXED, which only takes it) is computed
    // inside the node gather; the upwind fluxes, and every flux of a moving
    // mesh (with its GCL term), go through the edge buffer
    bool fused() const { return c.fluxType == 1 && c.flowType != 2; }
    // the flux kernel instance of this run's fluxType (and HLLC order; the
    // reconstruction only acts on level 1, where coordinates exist)
    void edge_flux_launch(const LevelView &L) {
        const unsigned ng = eblk(L.E);
        switch (c.fluxType) {
            case 2: k_edge_flux<2, false><<<ng, eb, 0, s>>>(P, L); break;
            case 3:
                // the extension: MUSCL on level 1, upwind first order below
                if (P.recon == FLITE_RECON_VAN_ALBADA && L.grid == 1)
                    k_edge_flux_muscl<<<(unsigned)((L.E + kMusclThreads - 1) / kMusclThreads), kMusclThreads, 0, s>>>(P, L);
                else if (P.recon == FLITE_RECON_VAN_ALBADA) k_edge_flux<3, true><<<ng, eb, 0, s>>>(P, L);
                else k_edge_flux<3, false><<<ng, eb, 0, s>>>(P, L);
                break;
            case 4:
                if (c.HLLCFluxOrder > 1) {
                    const int nt = std::min(eb, edge_threads(4, true));
                    k_edge_flux<4, true><<<(unsigned)((L.E + nt - 1) / nt), nt, 0, s>>>(P, L);
                }
                else k_edge_flux<4, false><<<ng, eb, 0, s>>>(P, L);
                break;
            default: k_edge_flux<1, false><<<ng, eb, 0, s>>>(P, L);
        }
    }
    void node_update(int l, int mode, int stage, bool anchor = true, int pre = PRE_NONE, int io = 0) {
        counted();
        launch_node_update(l, mode, stage, anchor, pre, io);
    }
    // the level-1 engine inlet terms after a node pass of `mode` (engine.cu)
    void engine_pass(int l, int mode) {
        const LevelView &L = V(l);
        if (l != 0 || !L.eng.f) return;
        no_group("the engine conditions");
        counted();
        k_engine_sums<<<1, kEngineLanes, 0, s>>>(P, L, mode);
        const bool all = P.eftype == 2;
        const int n = all ? L.N : L.eng.nnode;
        if (n > 0) {
            counted();
            k_engine_finish<<<nblk(n), nb, 0, s>>>(P, L, mode, all ? 1 : 0);
        }
    }
    void launch_node_update(int l, int mode, int stage, bool anchor, int pre = PRE_NONE, int io = 0) {
        switch (lanes_of(l)) {
            case 4: launch_node_update_u<4>(l, mode, stage, anchor, pre, io); break;
            case 8: launch_node_update_u<8>(l, mode, stage, anchor, pre, io); break;
            case 16: launch_node_update_u<16>(l, mode, stage, anchor, pre, io); break;
            case 32: launch_node_update_u<32>(l, mode, stage, anchor, pre, io); break;
            default: launch_node_update_u<1>(l, mode, stage, anchor, pre, io);
        }
    }
    template <int U>
    void launch_node_update_u(int l, int mode, int stage, bool anchor, int pre, int io) {
        // blocks of nt threads (nb, or less where the kernel's own bound is)
        const auto blk = [&](int prec) { return (unsigned)std::min(nb, node_threads(prec, U)); };
        const auto grid = [&](unsigned nt) { return (unsigned)((U * (size_t)V(l).N + nt - 1) / nt); };
#define FLITE_NODE(PREC, PRE)                                                                        \
    do {                                                                                              \
        const unsigned nt = blk(PREC);                                                                \
        FLITE_LAUNCH(k_node_update, (PREC, U, PRE,), grid(nt), nt, 0, P, V(l), mode, stage, io);      \
    } while (0)
        if (mixed()) {
            if (anchor) FLITE_NODE(GATHER_ANCHOR, PRE_NONE);
            else FLITE_NODE(GATHER_DELTA, PRE_NONE);
        } else if (fused()) {
            if constexpr (U == 1) {
                if (!P.engines && !(P.unsteady && P.explicit_)) {
                    FLITE_NODE(GATHER_LEAN, PRE_NONE);
                    return;
                }
            }
            if constexpr (U > 1) {
                if (pre == PRE_JST) {
                    FLITE_NODE(GATHER_CENTRAL, PRE_JST);
                    return;
                }
                if (pre == PRE_VISC) {
                    FLITE_NODE(GATHER_CENTRAL, PRE_VISC);
                    return;
                }
            }
            FLITE_NODE(GATHER_CENTRAL, PRE_NONE);
        } else {
            no_group("the edge buffer's fluxes");
            const unsigned nt = blk(GATHER_BUFFER);
            k_node_update<GATHER_BUFFER, U><<<grid(nt), nt, 0, s>>>(P, V(l), mode, stage, io);
        }
#undef FLITE_NODE
    }

    // ---- singleIteration (def_par:1002-1181) -----------------------------
    // after the step's state pass (pressure, records, primitives and, with
    // `bnd`, boundary fluxes of stage 1)
    void singleIteration(int l, bool calcDiss, bool bnd) {
        int pre = PRE_NONE;
        const bool own = inline_bnd(l), emit = emits();
        bool early = false;
        if (calcDiss) {
            early = bnd_beside(l, own || bnd);
            if (!step_jst(l)) {
                timesteps(l);
                dissipation(l);
                viscous(l, true);
            } else {
                pre = ts_jst_viscous(l, true, true, true);
            }
        }
        for (int st = 1; st <= P.nstage; ++st) {
            // u == uprev at stage 1: the FP64 evaluation there is the anchor
            // of the mixed-precision increments of the later stages
            const bool one = st == 1;
            if (!one && !emit) pressure(l);
            residual_pass(l, MODE_STAGE, st, one, !one && emit, own || (one && bnd), one && early,
                          one && calcDiss ? 2 : 0, one ? pre : PRE_NONE, stage_io(st, P.nstage, own, emit));
        }
    }
    // ---- doTimeIterations (def_par:966-1000) -----------------------------
    void doTimeIterations(int l, int nsteps, bool calcDiss) {
        if (nsteps <= 0) {
            counted();
            FLITE_LAUNCH(k_case_cycle, (), 1, 1, 0, V(l), d_cycle);
        }
        for (int i = 0; i < nsteps; ++i) {
            const bool bnd = step_bnd(l);
            state_pass(l, STATE_STEP | (calcDiss && visc() ? STATE_PRIM : 0), bnd);
            singleIteration(l, calcDiss, bnd);
        }
    }
    // ---- restrictGrid (def_par:12141-12430) ------------------------------
    // the coarse level's one-step update and the fine level's increment do not
    // depend on each other: the coarse part runs on the side stream (a branch
    // of the captured graph), where the small level's chain of launches hides
    // behind the fine level's.  The fine part waits for the coarse state
    // before it writes what that was restricted from.  Under explicit time
    // stepping the fine part reads the coarse level's step: no branch.
    void restrictGrid(int fl) {
        const int cl = fl + 1;
        const bool parallel = !(P.explicit_ && P.unsteady);
        auto coarse_state = [&] {
            counted();
            FLITE_LAUNCH(k_restrict_state, (), nblk(kChildLanes * (size_t)V(cl).N), nb, 0, P, V(cl), V(fl));
        };
        auto coarse = [&] {
            int pre = PRE_NONE;
            const bool mine = inline_bnd(cl);
            const bool early = bnd_beside(cl, mine);
            if (c.coarseGridDissipationScheme == 2) {
                pre = ts_jst_viscous(cl, true, true, true);
            } else {
                timesteps(cl);
                if (c.coarseGridDissipationScheme == 3) first_order_diss(cl);
                viscous(cl, true);
            }
            residual_pass(cl, MODE_RCOARSE, 0, true, false, mine, early, 2, pre, mine ? IO_BND : 0);
        };
        // with lanes per node the fine pass reads its neighbours' state (the
        // folded JST flux, the boundary edges), so the density floor it would
        // write there waits for k_restrict_incr, which visits the nodes with a
        // parent
        const bool own = inline_bnd(fl) && !lv[cl].orphans;
        const bool bnd = group_level(fl) && !own && c.flowType != 2;
        auto fine_head = [&] { state_pass(fl, visc() ? STATE_PRIM : 0, bnd); };
        auto fine = [&] {
            int pre = PRE_NONE;
            const bool early = bnd_beside(fl, bnd || own);
            // the fine part uses scheme 1 on level 1 under dissipationScheme 1,
            // scheme 2 otherwise (def_par:12269-12273)
            if (c.dissipationScheme == 1 && V(fl).grid == 1) {
                lp_diss(fl);
                viscous(fl, true);
            } else {
                pre = ts_jst_viscous(fl, false, true, own);
            }
            // the fine level keeps its turbulent time steps
            residual_pass(fl, MODE_RFINE, 0, false, false, bnd || own, early, 1, pre, own ? IO_BND | IO_LATER : 0);
        };
        if (parallel) {
            beside(0, [&] {
                coarse_state();
                CK(cudaEventRecord(coarse_ready, s));
                pass_branch = 3;
                try {
                    coarse();
                } catch (...) {
                    pass_branch = 1;
                    throw;
                }
                pass_branch = 1;
            });
            fine_head();
            CK(cudaStreamWaitEvent(s, coarse_ready, 0));
            fine();
            join(0);
        } else {
            coarse_state();
            coarse();
            fine_head();
            fine();
        }
        counted();
        FLITE_LAUNCH(k_restrict_incr, (), nblk(kChildLanes * (size_t)V(cl).N), nb, 0, P, V(cl), V(fl), own ? 1 : 0);
    }
    // ---- prolongateGrid (def_par:12432-12570) ----------------------------
    void prolongateGrid(int cl) {
        const int fl = cl - 1;
        const unsigned g = nblk(kChildLanes * (size_t)V(cl).N);
        counted();
        if (!lv[cl].orphans) {
            FLITE_LAUNCH(k_prolong, (), g, nb, 0, P, V(cl), V(fl));
        } else {
            FLITE_LAUNCH(k_prolong_coarse, (), g, nb, 0, P, V(cl), V(fl));
            counted();
            FLITE_LAUNCH(k_prolong_fine, (), nblk(V(fl).N), nb, 0, P, V(cl), V(fl));
        }
        engine_pass(fl, MODE_PROLONG);
    }
    // the head of a physical time step (mg_par:586-602): laminar viscosity
    // 1/Re on every level, u (and in unsteady runs uold) restricted to every
    // coarse level
    void physical_step_start() {
        const double mu = c.ReynoldsNumber > 0.0 ? 1. / c.ReynoldsNumber : 0.0;
        for (size_t l = 0; l < lv.size(); ++l) {
            k_fill<<<blocks(V(l).N), kBlock, 0, s>>>(V(l).mu, V(l).N, mu);
            if (l > 0) {
                mapFineToCoarse((int)l - 1);
                if (P.unsteady)
                    k_restrict_arr<<<nblk(V(l).N), nb, 0, s>>>(V(l), V(l - 1), V(l - 1).uold, V(l).uold, nvar());
            }
        }
    }
    void mapFineToCoarse(int fl) {
        counted();
        FLITE_LAUNCH(k_restrict_u, (), nblk(kChildLanes * (size_t)V(fl + 1).N), nb, 0, V(fl + 1), V(fl));
    }
    // ---- oneCycle (mg_par:907-1196) --------------------------------------
    void oneCycle() {
        const int G = (int)lv.size();
        const int nr = c.numberOfRelaxationSteps;
        auto relax = [&](int j1, int steps, bool calc) { doTimeIterations(j1 - 1, steps, calc); };
        const int sch = c.multigridScheme;
        if (sch <= 0) {
            for (int i = 1; i <= G - 1; ++i) {
                counted();
                FLITE_LAUNCH(k_case_save_u, (), nblk(nvar() * (size_t)V(i - 1).N), nb, 0, V(i - 1),
                             nvar() * (size_t)V(i - 1).N);
                mapFineToCoarse(i - 1);
            }
            counted();
            FLITE_LAUNCH(k_case_zero, (), nblk(nvar() * (size_t)V(G - 1).N), nb, 0, V(G - 1), 1,
                         nvar() * (size_t)V(G - 1).N);
            relax(G, nr, true);
            for (int i = G; i >= 2; --i) {
                counted();
                FLITE_LAUNCH(k_inject_u, (), nblk(V(i - 2).N), nb, 0, V(i - 1), V(i - 2));
            }
        } else if (sch == 1) {
            for (int i = 1; i <= G - 1; ++i) {
                relax(i, nr, i == 1);
                restrictGrid(i - 1);
                mapFineToCoarse(i - 1);
            }
            relax(G, nr, G == 1);
            for (int i = G; i >= 2; --i) {
                prolongateGrid(i - 1);
                relax(i - 1, nr, (i - 1) == 1);
            }
        } else if (sch == 2 || sch == 5) {
            int nsw = G <= 2 ? 1 : 2 * G - 4;
            int fsl = 1;
            for (int i = 1; i <= nsw; ++i) {
                for (int j = fsl; j <= G - 1; ++j) {
                    relax(j, sch == 5 ? j : nr, j == fsl);
                    restrictGrid(j - 1);
                }
                relax(G, sch == 5 ? G : nr, G == 1);
                if (fsl == 1) fsl = G > 2 ? G - 1 : G;
                else if (i <= nsw / 2) fsl = fsl - 1;
                else fsl = fsl + 1;
                for (int j = G; j >= fsl + 1; --j) {
                    prolongateGrid(j - 1);
                    relax(j - 1, nr, (j - 1) == 1);
                }
            }
            for (int j = G; j >= 2; --j) {
                prolongateGrid(j - 1);
                relax(j - 1, nr, (j - 1) == 1);
            }
        } else if (sch == 3 || sch == 7) {
            int nsw = G == 1 ? 1 : G - 1;
            int fsl = 1;
            for (int i = 1; i <= nsw; ++i) {
                for (int j = fsl; j <= G - 1; ++j) {
                    relax(j, nr, j == fsl);
                    restrictGrid(j - 1);
                }
                relax(G, nr, G == 1);
                if (fsl == 1) fsl = G >= 2 ? G - 1 : G;
                else fsl = fsl - 1;
                for (int j = G; j >= fsl + 1; --j) {
                    prolongateGrid(j - 1);
                    if (sch == 7) relax(j - 1, nr, (j - 1) == 1);
                }
            }
        } else if (sch == 4) {
            int nsw = G == 1 ? 1 : G - 1;
            int fsl = 1;
            for (int i = 1; i <= nsw; ++i) {
                for (int j = fsl; j <= G - 1; ++j) {
                    relax(j, nr, j == fsl);
                    restrictGrid(j - 1);
                }
                relax(G, nr, G == 1);
                fsl = fsl + 1;
                for (int j = G; j >= fsl + 1; --j) {
                    prolongateGrid(j - 1);
                    relax(j - 1, nr, (j - 1) == 1);
                }
            }
            for (int j = G; j >= 2; --j) {
                prolongateGrid(j - 1);
                relax(j - 1, nr, (j - 1) == 1);
            }
        }
    }

    void set_cycle(int cyc) {
        *h_cycle = cyc;
        CK(cudaMemcpyAsync(d_cycle, h_cycle, sizeof(int), cudaMemcpyHostToDevice, s));
    }

    // capture one oneCycle into a graph (not instantiated)
    void capture_cycle(cudaGraph_t *g) {
        *g = nullptr;
        CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        launches = 0;
        counting = true;
        try {
            oneCycle();
        } catch (...) {
            counting = false;
            cudaStreamEndCapture(s, g);
            if (*g) cudaGraphDestroy(*g);
            *g = nullptr;
            cudaGetLastError();  // an unfinished branch's
            throw;
        }
        counting = false;
        CK(cudaStreamEndCapture(s, g));
    }
    void drop_graph() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
    }
    // a launch option was set: the context's graph goes, and a batch that
    // holds the context sees by the number that its own is out of date
    unsigned options = 0;
    void options_changed() {
        ++options;
        drop_graph();
    }

    void ensure_graph() {
        if (graph) return;
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        launches = 0;
        counting = true;
        try {
            oneCycle();
        } catch (...) {
            counting = false;
            cudaStreamEndCapture(s, &g);
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();  // an unfinished branch's
            throw;
        }
        counting = false;
        CK(cudaStreamEndCapture(s, &g));
        graphTurb = calcTurb;
        cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
        cudaGraphDestroy(g);
        CK(e);
    }
};

namespace flite {
int create_context(const flite_controls *c, int nlevels, const flite_level_desc *levels, const flite_ctx *donor,
                   flite_ctx **out);
// far-field edges' part of the transposed Jacobian's product (adjoint.cu)
void vjp_farfield(flite_ctx &X, const LevelView &L, const double *x, const double *rbar, double *bvjp);
// the geometry arrays of level l from its descriptor (allocated when create)
void put_geometry(flite_ctx &X, int l, const flite_level_desc &d, bool create);
}  // namespace flite
