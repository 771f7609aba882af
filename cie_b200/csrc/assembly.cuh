// Shared by the assembly kernels: the assembly plan, the 1-D rules and bases,
// the integrand conventions and the finite-cell geometry.
#pragma once

#include "ciecu_assembly.h"
#include "space.cuh"
#include "spmv.cuh"

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <vector>

struct ciecu_assembly_s {
    ciecu_csr_s* csr = nullptr;
    int dim = 0, order = 0, nb = 0, nq = 0;
    long ncells = 0;
    const int* d_dofmap = nullptr;
    // Incidences (cell e, local row a) grouped by matrix row and sorted by colour
    // within a row: d_inc[i] = e * nb + a for i in [d_incStart[row], d_incStart[row + 1]),
    // and for every b the position of column dof[b] within that row, d_pos[i * nb + b],
    // in the smallest integer type that holds the longest row (posBytes).
    int* d_incStart = nullptr;        // rows + 1
    int* d_inc = nullptr;             // ncells * nb
    void* d_pos = nullptr;            // ncells * nb * nb
    int posBytes = 1;
    int maxRow = 0;                   // longest row of the pattern
    int colors = 0;
    double* d_gtab = nullptr;         // nq * dim * nb parametric gradients
    double* d_wq = nullptr;           // nq weights
    // nb * nb: the reference element's sums of the call that holds the lock while it submits
    // what writes and reads them; the next call's come after them on the stream.
    double* d_unit = nullptr;
    std::mutex unitMutex;
    int q1 = 0;                       // 1-D quadrature points (nq = q1^dim)
    std::vector<double> gn, gw;       // 1-D Gauss-Legendre rule on [-1, 1]
};

namespace ciecu {

// Gauss-Legendre nodes and weights by Newton iteration on P_n from the
// Tricomi initial guess (the method of GaussLegendreQuadrature.cpp:82-175).
int gauss_legendre(int order, std::vector<double>& nodes, std::vector<double>& weights);

// Lagrange basis on equispaced nodes -1 + 2i/p and its derivative at x.
__host__ __device__ inline void lagrange(int p, double x, double* v, double* dv) {
    const int n = p + 1;
    double nodes[16];
    for (int i = 0; i < n; ++i) nodes[i] = -1.0 + 2.0 * i / p;
    for (int i = 0; i < n; ++i) {
        double value = 1.0, deriv = 0.0;
        for (int j = 0; j < n; ++j) {
            if (j == i) continue;
            const double f = (x - nodes[j]) / (nodes[i] - nodes[j]);
            deriv = deriv * f + value / (nodes[i] - nodes[j]);
            value *= f;
        }
        v[i] = value;
        dv[i] = deriv;
    }
}

// Scale and per-axis factors of the two stiffness conventions:
//   reference (0): scale = prod_d 2/h_d, f_d = 1
//   physical  (1): scale = prod_d h_d/2, f_d = (2/h_d)^2
inline void convention_factors(int dim, const double* h, int convention, double& scale, double f[3]) {
    scale = 1.0;
    for (int d = 0; d < 3; ++d) f[d] = 1.0;
    for (int d = 0; d < dim; ++d) {
        if (convention == 1) {
            scale *= 0.5 * h[d];
            f[d] = (2.0 / h[d]) * (2.0 / h[d]);
        } else {
            scale *= 2.0 / h[d];
        }
    }
}

// The standard-rule element matrix with kappa = 1, scale * sum_q w_q sum_d f_d
// G_q[d][a] G_q[d][b], into d_out (nb * nb doubles) on stream st.
int unit_element(const ciecu_assembly_s* P, double scale, const double f[3], double* d_out, cudaStream_t st);

// ---- row-gather scatter ----------------------------------------------------------
//
// Adds element matrices into the CSR values row by row.  A group of `lanes` lanes
// (the power of two >= nb, at most 32) owns a matrix row: it walks the row's
// incidences in colour order, lane b adding entry (a, b) of the incident cell's
// matrix at its position of the row in shared memory, and writes the finished row
// once.  Every entry is summed in colour order, as a launch per colour that adds
// into global memory would sum it.
//   What bounds it: the bytes of the values (written once), the incidence list and
// the positions (1 byte per element entry for rows of up to 256 entries).  A launch
// per colour read a 4-byte slot and read and wrote an 8-byte value in scattered
// order for every element entry, and integrated that entry again for every cell:
// 3D Q1 128^3, 134 M element entries: 3.43 ms with the zero fill, this kernel
// 0.38 ms for the 700 MB of values, lists and positions.  What holds it there is
// the shared-memory pipe (a read-modify-write, a matrix entry and three shuffles
// for every 32 element entries), not memory.
//   SRC: coef(e) = the cell's coefficient, matrix(e) its nb x nb matrix, adds(e)
// whether the cell takes part in this pass.  `base` (nb x nb) is staged in shared
// memory when it fits (stagedBase) and handed to matrix().
template <typename POS>
struct GatherArgs {
    int rows, nb, lanes, rowStride;   // rowStride: values of shared memory per row, 0: sum in global memory
    int stagedBase, accumulate;
    const int* __restrict__ rowptr;
    const int* __restrict__ incStart;
    const int* __restrict__ inc;
    const POS* __restrict__ pos;
};

constexpr int kGatherThreads = 256;
constexpr size_t kGatherBaseBytes = 32 * 1024;   // the base matrix is staged up to this size
constexpr size_t kGatherRowBytes = 64 * 1024;    // a block's rows are summed in shared memory up to this size

// Lanes of a row for nb element columns.
constexpr int gather_lanes(int nb) {
    int lanes = 1;
    while (lanes < nb && lanes < 32) lanes <<= 1;
    return lanes;
}

// NB: the element columns when they are known at compile time (0: G.nb).
template <typename V, typename POS, int NB, typename SRC>
__global__ void __launch_bounds__(kGatherThreads)
    row_gather_kernel(GatherArgs<POS> G, SRC src, const V* __restrict__ base, V* __restrict__ val) {
    extern __shared__ __align__(16) unsigned char gather_smem[];
    V* s_base = reinterpret_cast<V*>(gather_smem);
    const int nb = NB ? NB : G.nb, nb2 = nb * nb;
    const int L = NB ? gather_lanes(NB) : G.lanes, perWarp = 32 / L;
    const V* K = base;
    int used = 0;
    if (G.stagedBase) {
        for (int k = threadIdx.x; k < nb2; k += kGatherThreads) s_base[k] = base[k];
        K = s_base;
        used = nb2;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = lane / L, l = lane - group * L;
    V* s_row = s_base + used + (warp * perWarp + group) * G.rowStride;
    const long warps = static_cast<long>(gridDim.x) * (kGatherThreads / 32);
    const long tasks = (static_cast<long>(G.rows) + perWarp - 1) / perWarp;
    // Incidences whose positions are loaded a row ahead, and the columns of each a lane holds.
    constexpr int kAhead = NB == 0 ? 2 : (gather_lanes(NB) < 8 ? gather_lanes(NB) : (NB > 32 ? 4 : 8));
    constexpr int kCols = NB > 32 ? (NB + 31) / 32 : 1;
    // A row is a chain of dependent loads (extents, incidences and positions, cells),
    // each a trip to memory of its own; the chain of the next two rows is in flight
    // while this one is summed (without it the kernel was latency-bound: 0.40 ms).
    struct Extents {
        int k0, len, i0, count;
    };
    auto extents = [&](long task) {
        Extents x{0, 0, 0, 0};
        const long row = task * perWarp + group;
        if (row < G.rows) {
            x.k0 = G.rowptr[row];
            x.len = G.rowptr[row + 1] - x.k0;
            x.i0 = G.incStart[row];
            x.count = G.incStart[row + 1] - x.i0;
        }
        return x;
    };
    auto incidence = [&](const Extents& x, int first) { return first + l < x.count ? G.inc[x.i0 + first + l] : -1; };
    auto positions = [&](const Extents& x, POS (&at)[kAhead][kCols]) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                at[u][j] = u < x.count && l + 32 * j < nb ? G.pos[static_cast<long>(x.i0 + u) * nb + l + 32 * j] : POS(0);
    };
    // coefficient and matrix row of an incidence (null: takes no part)
    auto resolve = [&](int ea, V& c, const V*& M) {
        c = V(0);
        M = nullptr;
        if (ea < 0) return;
        const int e = ea / nb;
        if (!src.adds(e)) return;
        c = src.coef(e);
        M = src.matrix(e, K) + (ea - e * nb) * nb;
    };
    auto from = [&](const V* M, int u) {
        return reinterpret_cast<const V*>(
            __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(M), u, L));
    };
    long task = static_cast<long>(blockIdx.x) * (kGatherThreads / 32) + warp;
    Extents x = extents(task), xn = extents(task + warps);
    POS at[kAhead][kCols];
    V c;
    const V* M;
    positions(x, at);
    resolve(incidence(x, 0), c, M);
    for (; task < tasks; task += warps) {
        const Extents xnn = extents(task + 2 * warps);
        const int nextInc = incidence(xn, 0);
        POS nextAt[kAhead][kCols];
        positions(xn, nextAt);
        V* acc = G.rowStride ? s_row : val + x.k0;
        if (G.rowStride || !G.accumulate)
            for (int j = l; j < x.len; j += L) acc[j] = G.accumulate ? val[x.k0 + j] : V(0);
        __syncwarp();
        const int most = __reduce_max_sync(0xffffffffu, x.count);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (u >= most || u >= L) break;
            const V cu = __shfl_sync(0xffffffffu, c, u, L);
            const V* Mu = from(M, u);
            if (Mu && l < nb) {
#pragma unroll
                for (int j = 0; j < kCols; ++j)
                    if (l + 32 * j < nb) acc[at[u][j]] = fma(cu, Mu[l + 32 * j], acc[at[u][j]]);
                if (NB == 0)
                    for (int b = l + L; b < nb; b += L) {
                        const int to = static_cast<int>(G.pos[static_cast<long>(x.i0 + u) * nb + b]);
                        acc[to] = fma(cu, Mu[b], acc[to]);
                    }
            }
            __syncwarp();
        }
        for (int first = 0; first < most; first += L) {  // the incidences past those held
            if (first > 0) resolve(incidence(x, first), c, M);
            const int end = min(most - first, L);
            for (int u = first == 0 ? kAhead : 0; u < end; ++u) {
                const V cu = __shfl_sync(0xffffffffu, c, u, L);
                const V* Mu = from(M, u);
                if (Mu)
                    for (int b = l; b < nb; b += L) {
                        const int to = static_cast<int>(G.pos[static_cast<long>(x.i0 + first + u) * nb + b]);
                        acc[to] = fma(cu, Mu[b], acc[to]);
                    }
                __syncwarp();
            }
        }
        resolve(nextInc, c, M);
        if (G.rowStride) {
            for (int j = l; j < x.len; j += L) val[x.k0 + j] = acc[j];
            __syncwarp();
        }
        x = xn;
        xn = xnn;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int j = 0; j < kCols; ++j) at[u][j] = nextAt[u][j];
    }
}

template <typename V, typename POS, int NB, typename SRC>
int launch_row_gather_nb(const ciecu_assembly_s* P, const SRC& src, const V* base, int accumulate, V* val,
                         cudaStream_t st) {
    GatherArgs<POS> G{};
    G.rows = P->csr->rows;
    G.nb = P->nb;
    G.lanes = gather_lanes(P->nb);
    G.accumulate = accumulate;
    G.rowptr = P->csr->rowptr;
    G.incStart = P->d_incStart;
    G.inc = P->d_inc;
    G.pos = static_cast<const POS*>(P->d_pos);
    const size_t baseBytes = sizeof(V) * P->nb * P->nb;
    G.stagedBase = baseBytes <= kGatherBaseBytes ? 1 : 0;
    const int rowsPerBlock = (kGatherThreads / 32) * (32 / G.lanes);
    const size_t rowBytes = sizeof(V) * static_cast<size_t>(rowsPerBlock) * static_cast<size_t>(P->maxRow);
    G.rowStride = rowBytes <= kGatherRowBytes ? std::max(P->maxRow, 1) : 0;
    const size_t smem = (G.stagedBase ? baseBytes : 0) +
                        (G.rowStride ? sizeof(V) * static_cast<size_t>(rowsPerBlock) * G.rowStride : 0);
    auto kernel = row_gather_kernel<V, POS, NB, SRC>;
    CIECU_TRY(allow_shared(kernel));
    const long blocks = (static_cast<long>(G.rows) + rowsPerBlock - 1) / rowsPerBlock;
    kernel<<<fit_grid(kernel, kGatherThreads, blocks, smem), kGatherThreads, smem, st>>>(G, src, base, val);
    count_launch();
    CIECU_CHECK_LAUNCH("row_gather_kernel");
    return CIECU_OK;
}

// Compile-time element sizes of the Q1, Q2 and Q3 cells of two and three axes.
template <typename V, typename POS, typename SRC>
int launch_row_gather_pos(const ciecu_assembly_s* P, const SRC& src, const V* base, int accumulate, V* val,
                          cudaStream_t st) {
    switch (P->nb) {
        case 4: return launch_row_gather_nb<V, POS, 4>(P, src, base, accumulate, val, st);
        case 8: return launch_row_gather_nb<V, POS, 8>(P, src, base, accumulate, val, st);
        case 9: return launch_row_gather_nb<V, POS, 9>(P, src, base, accumulate, val, st);
        case 16: return launch_row_gather_nb<V, POS, 16>(P, src, base, accumulate, val, st);
        case 27: return launch_row_gather_nb<V, POS, 27>(P, src, base, accumulate, val, st);
        case 64: return launch_row_gather_nb<V, POS, 64>(P, src, base, accumulate, val, st);
        default: return launch_row_gather_nb<V, POS, 0>(P, src, base, accumulate, val, st);
    }
}

// val (+)= the element matrices of `src`; rows without an incidence become zero
// unless `accumulate`.
template <typename V, typename SRC>
int launch_row_gather(const ciecu_assembly_s* P, const SRC& src, const V* base, int accumulate, V* val,
                      cudaStream_t st) {
    if (P->csr->rows == 0) return CIECU_OK;
    if (P->posBytes == 1) return launch_row_gather_pos<V, uint8_t>(P, src, base, accumulate, val, st);
    if (P->posBytes == 2) return launch_row_gather_pos<V, uint16_t>(P, src, base, accumulate, val, st);
    return launch_row_gather_pos<V, int>(P, src, base, accumulate, val, st);
}

// ---- finite-cell geometry -------------------------------------------------------

struct EmbeddedArgs {
    int dim, order, nb, q1, nq, maxDepth;
    int cells[3];
    double gn[16], gw[16];
    double origin[3], h[3], center[3];
    double radius2, alpha, scale;
    double f[3];
};

// Inside test of the sphere domain at the parametric point xi of a cell.
__device__ __forceinline__ bool embedded_inside(const EmbeddedArgs& P, const double* corg, const double* xi) {
    double r2 = 0.0;
    for (int d = 0; d < P.dim; ++d) {
        const double x = corg[d] + 0.5 * (xi[d] + 1.0) * P.h[d];
        r2 += (x - P.center[d]) * (x - P.center[d]);
    }
    return r2 < P.radius2;
}

// Parametric position and base weight of point q of a tree node (first index fastest).
__device__ __forceinline__ double embedded_point(const EmbeddedArgs& P, const double* base, double length, int q,
                                                 double* xi) {
    int rest = q;
    double w = 1.0;
    for (int d = 0; d < P.dim; ++d) {
        const int i = rest % P.q1;
        rest /= P.q1;
        xi[d] = base[d] + 0.5 * length * (P.gn[i] + 1.0);
        w *= P.gw[i];
    }
    return w;
}

}  // namespace ciecu
