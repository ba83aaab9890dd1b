// Node gathers with a group of lanes per node, for kernels that sum terms over
// a node's incidences.
#pragma once
#include "device.cuh"

namespace flite {

// Group-per-node gathers (small levels): U lanes (a power of two up to 32)
// serve one node, M sums of the node take R terms each from every incidence.
// Lane l of the group evaluates the M*R terms of incidence k0 + l and leaves
// them in the warp's shared slab gs[term][lane] (rows of 33 values: the lanes
// that read different terms of one incidence hit different banks); lane m of
// the group then adds sum m's terms in incidence order, so the sums are those
// of the serial loop bit for bit (lanes past the last incidence leave zeros,
// and x + 0 is x).  `out` holds the sums so far on entry and the new ones, in
// every lane, on return.  Groups past the last node stay in the loop (the
// warp's barriers need every lane) but add nothing.
// What bounds it: the latency of one node's chain.  The serial part is one
// add per term on M lanes at once; broadcasting every term to every lane
// instead takes 2 M R shuffles and M R adds per incidence of the warp.
constexpr int kSlabRow = 33;
template <int U, int M, int R, class T, class Terms>
__device__ __forceinline__ void group_sum(T *gs, int beg, int end, bool active, int gl, Terms &&terms, T *out) {
    constexpr int C = (M + U - 1) / U;  // sums per lane
    constexpr int S = U < 8 ? U : 8;    // incidences added per step
    const int lane = (int)(threadIdx.x & 31), g0 = lane - gl;
    T acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = T(0);
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (m % U == gl) acc[m / U] = out[m];
    const int span = active ? end - beg : 0;
    const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)span);
    for (int t = 0; t < longest; t += U) {
        T v[M * R];
#pragma unroll
        for (int c = 0; c < M * R; ++c) v[c] = T(0);
        if (t + gl < span) terms(beg + t + gl, v);
#pragma unroll
        for (int c = 0; c < M * R; ++c) gs[c * kSlabRow + lane] = v[c];
        __syncwarp();
        const int n = min(U, longest - t);
        for (int q = 0; q < n; q += S) {
            T x[C][S][R];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int m = gl + c * U < M ? gl + c * U : 0;
#pragma unroll
                for (int k = 0; k < S; ++k)
#pragma unroll
                    for (int r = 0; r < R; ++r) x[c][k][r] = gs[(m * R + r) * kSlabRow + g0 + q + k];
            }
#pragma unroll
            for (int k = 0; k < S; ++k)
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int c = 0; c < C; ++c) acc[c] = acc[c] + x[c][k][r];
        }
        __syncwarp();
    }
#pragma unroll
    for (int m = 0; m < M; ++m) out[m] = __shfl_sync(0xffffffffu, acc[m / U], m % U, U);
}
// the calling warp's slab of K terms out of the block's (blocks of at most
// 256 threads; 128 with more than 16 terms)
#define FLITE_GROUP_SLAB(T, K)                                            \
    __shared__ T gslab_[U > 1 ? ((K) > 16 ? 4 : 8) * (K)*kSlabRow : 1];   \
    T *gs = gslab_ + (U > 1 ? (threadIdx.x >> 5) * (K)*kSlabRow : 0)

// Node i's incidences with a thread per node, Q at a time: the M terms of all
// Q are evaluated (terms(t, v)) before the first is added (add(v)), in order.
// What bounds such a walk is the latency of its loads; Q incidences have Q
// times the loads in flight, for as many registers as their terms take, so
// each kernel takes the Q and the resident blocks that measured best together
// (815,425 nodes, one at a time before, us): time step 148 -> 105 with two and
// four blocks of 64 registers (three incidences 126, four 144), Laplacian and
// JST flux 215 -> 158, viscous gradients 110 -> 104, viscous flux 150 -> 139.
template <int Q, int M, class Terms, class Add>
__device__ __forceinline__ void walk(const LevelView &L, int i, Terms &&terms, Add &&add) {
    const int deg = L.inc_ptr[i + 1] - L.inc_ptr[i];
    const int2 *row = L.rows + ((size_t)L.row_ptr[i / kRow] * kRow + i % kRow);
    int2 t[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (q < deg) t[q] = __ldg(row + q * kRow);
    int k = 0;
    for (; k + Q <= deg; k += Q) {
        int2 now[Q];
        double v[Q][M];
        row += Q * kRow;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            now[q] = t[q];
            if (k + Q + q < deg) t[q] = __ldg(row + q * kRow);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) terms(now[q], v[q]);
#pragma unroll
        for (int q = 0; q < Q; ++q) add(v[q]);
    }
#pragma unroll
    for (int q = 0; q < Q - 1; ++q)
        if (k + q < deg) {
            double v[M];
            terms(t[q], v);
            add(v);
        }
}
// the node i, lane gl and idle groups of a gather kernel templated on U
#define FLITE_NODE_LANES(L)                                          \
    const int gl = U > 1 ? (int)(threadIdx.x % U) : 0;               \
    const int i_raw = (int)(blockIdx.x * blockDim.x + threadIdx.x) / U; \
    if (U == 1 && i_raw >= L.N) return;                              \
    const bool active = i_raw < L.N;                                 \
    const int i = active ? i_raw : L.N - 1
// M sums of node i over its incidences (terms(t, v): one term per sum) and
// boundary entries (bterms(q, v)), with a thread or a group per node, both in
// order.  gs: the group's slab of M terms (unused with a thread).
template <int U, int M, class Terms>
__device__ __forceinline__ void sum_incidences(const LevelView &L, int i, bool active, int gl, double *gs,
                                               Terms &&terms, double *out) {
    if constexpr (U > 1) {
        group_sum<U, M, 1, double>(
            gs, L.inc_ptr[i], L.inc_ptr[i + 1], active, gl, [&](int q, double *v) { terms(L.inc[q], v); }, out);
    } else {
        walk<2, M>(
            L, i,
            [&](const int2 t, double *v) {
#pragma unroll
                for (int m = 0; m < M; ++m) v[m] = 0.0;
                terms(t, v);
            },
            [&](const double *v) {
#pragma unroll
                for (int m = 0; m < M; ++m) out[m] = out[m] + v[m];
            });
    }
}
template <int U, int M, class Terms>
__device__ __forceinline__ void sum_boundary(const LevelView &L, int i, bool active, int gl, double *gs,
                                             Terms &&terms, double *out) {
    if constexpr (U > 1) {
        group_sum<U, M, 1, double>(gs, L.binc_ptr[i], L.binc_ptr[i + 1], active, gl, terms, out);
    } else {
        for (int q = L.binc_ptr[i]; q < L.binc_ptr[i + 1]; ++q) {
            double v[M];
#pragma unroll
            for (int m = 0; m < M; ++m) v[m] = 0.0;
            terms(q, v);
#pragma unroll
            for (int m = 0; m < M; ++m) out[m] = out[m] + v[m];
        }
    }
}

}  // namespace flite
