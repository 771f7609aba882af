// Finite-cell stiffness: the cut-cell quadrature of KDTreeQuadraturePointFactory
// (fem/packages/numeric/inc/KDTreeQuadraturePointFactory.hpp:67-173) with the
// material scaling of ScaledMultiMaterialIntegrand (integrands/impl/
// ScaledMultiMaterialIntegrand_impl.hpp:33-60) and the stiffness integrand
// (LinearIsotropicStiffnessIntegrand_impl.hpp:62-75), load-balanced and with the
// element matrices formed from moments.
//
// The element matrix of a cut cell is a Gram matrix over its kept quadrature
// points, K = sum_{p,d} w_p s_p f_d G_p[d] G_p[d]^T.  Products of two basis
// functions (or of two derivatives) of one axis are polynomials of degree 2 p, so
//   phi_i phi_j = sum_a c0[ij][a] P_a,   phi_i' phi_j' = sum_a c1[ij][a] P_a
// in Legendre polynomials, and the points enter only through the (2p + 1)^dim
// moments of the cell, mu[abc] = sum_p w_p s_p P_a(x_p) P_b(y_p) P_c(z_p):
//   K = sum_axis f_axis sum_abc mu[abc] c[..][a] c[..][b] c[..][c].
// Three passes:
//   1. classify every cell by its base points (one warp per cell); a prefix sum
//      numbers the cut cells in cell order;
//   2. one CTA per cut cell (fc_cell_kernel): a warp per depth-1 tree node walks
//      that node's subtree with the keep / refine rules and adds the kept points'
//      moments, plane by plane and axis by axis; the warps' moments are summed in
//      node order and contracted with c0 and c1 axis by axis;
//   3. the row gather (assembly.cuh) adds every cell's matrix into the CSR values:
//      regular cells s K1 (s = 1 inside, alpha outside, K1 the standard-rule
//      matrix), cut cells their own, in colour order.
// Everything is in FP64 (the FP32 copy for inner / preconditioner operators rounds
// the finished FP64 element matrices), and no sum depends on the schedule.
#include "assembly.cuh"
#include "sortscan.cuh"
#include "space.cuh"

#include <algorithm>
#include <string>
#include <type_traits>

namespace ciecu {
namespace {

// One warp per cell: number of the cell's base points inside the domain.
// cut[e] = 1 for a cell with points on both sides; side[e] = 1 for a cell fully
// inside.
__global__ void fc_classify_kernel(EmbeddedArgs P, long ncells, int* __restrict__ cut, signed char* __restrict__ side) {
    const int lane = threadIdx.x & 31;
    const long warps = static_cast<long>(gridDim.x) * (blockDim.x >> 5);
    for (long e = static_cast<long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); e < ncells; e += warps) {
        double corg[3] = {0.0, 0.0, 0.0};
        long rest = e;
        for (int d = 0; d < P.dim; ++d) {
            corg[d] = P.origin[d] + static_cast<double>(rest % P.cells[d]) * P.h[d];
            rest /= P.cells[d];
        }
        const double root[3] = {-1.0, -1.0, -1.0};
        int inside = 0;
        for (int q = lane; q < P.nq; q += 32) {
            double xi[3];
            embedded_point(P, root, 2.0, q, xi);
            inside += embedded_inside(P, corg, xi) ? 1 : 0;
        }
        inside = __reduce_add_sync(0xffffffffu, inside);
        if (lane == 0) {
            cut[e] = (inside > 0 && inside < P.nq) ? 1 : 0;
            side[e] = inside == P.nq ? 1 : 0;
        }
    }
}

__global__ void fc_compact_kernel(long ncells, const int* __restrict__ cut, const int* __restrict__ index,
                                  int* __restrict__ cutCells) {
    for (long e = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; e < ncells;
         e += static_cast<long>(gridDim.x) * blockDim.x)
        if (cut[e]) cutCells[index[e]] = static_cast<int>(e);
}

// Sizes of a cell's moment form: axis d < dim has q1 points, order + 1 functions,
// m1 = 2 order + 1 Legendre polynomials and `pairs` unordered function pairs; an
// absent axis has one of each.  DIM and ORDER are compile-time for the common
// elements (0: taken from the arguments).
template <int DIM, int ORDER>
struct FcShape {
    int dim, n1, m1, pairs, q1;
    __device__ FcShape(const EmbeddedArgs& P) {
        dim = DIM ? DIM : P.dim;
        n1 = (ORDER ? ORDER : P.order) + 1;
        m1 = 2 * n1 - 1;
        pairs = n1 * (n1 + 1) / 2;
        q1 = P.q1;
    }
    __device__ __forceinline__ int q(int d) const { return d < dim ? q1 : 1; }
    __device__ __forceinline__ int m(int d) const { return d < dim ? m1 : 1; }
    __device__ __forceinline__ int p(int d) const { return d < dim ? pairs : 1; }
};

constexpr int kFcMoments = 343;                      // most moments of a cell: 7^3 (nb <= 64)
constexpr int kFcPerLane = (kFcMoments + 31) / 32;

// Shared memory of a CTA in doubles: each warp's tables and planes, then the
// moments and the arrays of the contraction (the warps' moments alias the latter).
struct FcSmem {
    int warp, moments, a, b, k, total;
};
__host__ __device__ inline FcSmem fc_smem(int dim, int order, int q1, int warps) {
    const int m1 = 2 * order + 1, pairs = (order + 1) * (order + 2) / 2;
    const int mx = m1, my = dim > 1 ? m1 : 1, mz = dim > 2 ? m1 : 1;
    const int px = pairs, py = dim > 1 ? pairs : 1, pz = dim > 2 ? pairs : 1;
    FcSmem s;
    s.warp = 3 * q1 * m1 + q1 * q1 + m1 * q1 + m1 * m1;
    s.moments = mx * my * mz;
    s.a = mx * my * pz;
    s.b = mx * py * pz;
    s.k = px * py * pz;
    const int contraction = 2 * s.a + 2 * s.b + s.k, partial = warps * s.moments;
    s.total = warps * s.warp + s.moments + (contraction > partial ? contraction : partial);
    return s;
}

// One CTA per cut cell, one warp per start node: the 2^dim children of the root
// (depth 1) when maxDepth >= 1, else the root.  Each warp walks its subtree
// depth-first with the rules of KDTreeQuadraturePointFactory.hpp:156-170.
// pairTable: c0 then c1, [pair (i <= j) at j (j + 1) / 2 + i][m1].
//   What bounds it: FP64 arithmetic and the latency of its short steps.  The
// contraction of a cell is 36,000 FMAs (Q3) and a kept tree node 2,600, against
// 8,192 FMAs for every kept point of the Gram form on the tensor cores (FP64 DMMA),
// which took 17.7 ms of the 22 ms of the 32^3 Q3 sphere (2,528 cut cells); this
// kernel takes 0.62 ms of 1.46 ms.  Against a 64-bit evaluation both are 4.1e-15
// off (2-norm of the matrix).  The FP32 copy came from split-BF16 MMAs, 2.2e-6 off;
// rounded from these matrices it is 2.9e-8 off.
template <int DIM, int ORDER, typename V>
__global__ void __launch_bounds__(256) fc_cell_kernel(EmbeddedArgs P, const int* __restrict__ cutCells, int first,
                                                      const double* __restrict__ pairTable, V* __restrict__ out) {
    extern __shared__ double fc_shared[];
    const FcShape<DIM, ORDER> S(P);
    const int dim = S.dim, m1 = S.m1, q1 = S.q1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const FcSmem size = fc_smem(dim, S.n1 - 1, q1, warps);
    double* s_tab = fc_shared + warp * size.warp;  // [axis][point][polynomial]
    double* s_w = s_tab + 3 * q1 * m1;             // weights of a plane, x fastest
    double* s_t1 = s_w + q1 * q1;                  // [y point][x polynomial]
    double* s_t2 = s_t1 + m1 * q1;                 // [y polynomial][x polynomial]
    double* s_mu = fc_shared + warps * size.warp;
    double* s_part = s_mu + size.moments;          // the warps' moments, then the contraction's arrays
    const int e = cutCells[first + blockIdx.x];
    double corg[3] = {0.0, 0.0, 0.0};
    {
        long rest = e;
        for (int d = 0; d < dim; ++d) {
            corg[d] = P.origin[d] + static_cast<double>(rest % P.cells[d]) * P.h[d];
            rest /= P.cells[d];
        }
    }
    const int nq = P.nq;
    const int qx = S.q(0), qy = S.q(1), qz = S.q(2), mx = S.m(0), my = S.m(1), mz = S.m(2);
    const int mxy = mx * my;
    double acc[kFcPerLane];
#pragma unroll
    for (int j = 0; j < kFcPerLane; ++j) acc[j] = 0.0;
    const int d0 = P.maxDepth >= 1 ? 1 : 0, digit = (1 << dim) - 1;
    int depth = d0, code = d0 ? warp : 0;  // `dim` bits of the child number a level below the root
    for (;;) {
        double base[3] = {-1.0, -1.0, -1.0};
        double length = 2.0;
        for (int level = 1; level <= depth; ++level) {
            length *= 0.5;
            const int child = (code >> (dim * (depth - level))) & digit;
            for (int d = 0; d < dim; ++d)
                if ((child >> d) & 1) base[d] += length;
        }
        int inside = 0;
        for (int q = lane; q < nq; q += 32) {
            double xi[3];
            embedded_point(P, base, length, q, xi);
            inside += embedded_inside(P, corg, xi) ? 1 : 0;
        }
        inside = __reduce_add_sync(0xffffffffu, inside);
        const bool homogeneous = inside == 0 || inside == nq;
        const bool keep = inside == nq || depth == P.maxDepth || (depth == 0 && homogeneous);
        if (keep) {
            double jac = 1.0;
            for (int d = 0; d < dim; ++d) jac *= 0.5 * length;
            // P_a at the node's points of each axis, by the three-term recurrence
            for (int t = lane; t < 3 * q1; t += 32) {
                const int d = t / q1, i = t - d * q1;
                double* tab = s_tab + t * m1;
                const double x = base[d] + 0.5 * length * (P.gn[i] + 1.0);
                double p0 = 1.0, p1 = x;
                tab[0] = 1.0;
                for (int k = 1; k < m1; ++k) {
                    tab[k] = p1;
                    const double p2 = ((2.0 * k + 1.0) * x * p1 - k * p0) / (k + 1.0);
                    p0 = p1;
                    p1 = p2;
                }
            }
            __syncwarp();
            for (int z = 0; z < qz; ++z) {
                for (int t = lane; t < qx * qy; t += 32) {
                    double xi[3];
                    const double w = embedded_point(P, base, length, z * qx * qy + t, xi) * jac;
                    s_w[t] = w * (embedded_inside(P, corg, xi) ? 1.0 : P.alpha);
                }
                __syncwarp();
                for (int t = lane; t < mx * qy; t += 32) {
                    const int y = t / mx, a = t - y * mx;
                    double s = 0.0;
                    for (int x = 0; x < qx; ++x) s = fma(s_w[y * qx + x], s_tab[x * m1 + a], s);
                    s_t1[t] = s;
                }
                __syncwarp();
                for (int t = lane; t < mxy; t += 32) {
                    const int b = t / mx, a = t - b * mx;
                    double s = 0.0;
                    for (int y = 0; y < qy; ++y) s = fma(s_t1[y * mx + a], s_tab[(q1 + y) * m1 + b], s);
                    s_t2[t] = s;
                }
                __syncwarp();
                const double* pz = s_tab + (2 * q1 + z) * m1;
#pragma unroll
                for (int j = 0; j < kFcPerLane; ++j) {
                    const int t = lane + 32 * j;
                    if (t < size.moments) {
                        const int c = t / mxy;
                        acc[j] = fma(s_t2[t - c * mxy], pz[c], acc[j]);
                    }
                }
                __syncwarp();
            }
        }
        if (!homogeneous && depth < P.maxDepth) {
            code <<= dim;
            ++depth;
            continue;
        }
        while (depth > d0 && (code & digit) == digit) {
            code >>= dim;
            --depth;
        }
        if (depth == d0) break;
        ++code;
    }
#pragma unroll
    for (int j = 0; j < kFcPerLane; ++j) {
        const int t = lane + 32 * j;
        if (t < size.moments) s_part[warp * size.moments + t] = acc[j];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < size.moments; t += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < warps; ++w) s += s_part[w * size.moments + t];
        s_mu[t] = s;
    }
    __syncthreads();
    // Contraction, z then y then x.  Per axis only one of the three factors is a
    // product of derivatives, so two arrays are carried: "0" without a derivative
    // yet, "1" the sum of those with one (times their f).
    const int px = S.p(0), py = S.p(1), pz = S.p(2);
    double* s_a0 = s_part;
    double* s_a1 = s_a0 + size.a;
    double* s_b0 = s_a1 + size.a;
    double* s_b1 = s_b0 + size.b;
    double* s_k = s_b1 + size.b;
    const double* c0 = pairTable;
    const double* c1 = pairTable + S.pairs * m1;
    for (int t = threadIdx.x; t < size.a; t += blockDim.x) {
        const int p = t / mxy, ab = t - p * mxy;
        double s0 = 0.0, s1 = 0.0;
        if (dim > 2) {
            for (int c = 0; c < mz; ++c) {
                const double mu = s_mu[c * mxy + ab];
                s0 = fma(mu, c0[p * m1 + c], s0);
                s1 = fma(mu, c1[p * m1 + c], s1);
            }
        } else {
            s0 = s_mu[ab];
        }
        s_a0[t] = s0;
        s_a1[t] = s1 * P.f[2];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < size.b; t += blockDim.x) {
        const int pp = t / mx, a = t - pp * mx;  // pp = (z pair, y pair), y fastest
        const int pzi = pp / py, pyi = pp - pzi * py;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        if (dim > 1) {
            for (int b = 0; b < my; ++b) {
                const double v0 = s_a0[pzi * mxy + b * mx + a], v1 = s_a1[pzi * mxy + b * mx + a];
                s0 = fma(v0, c0[pyi * m1 + b], s0);
                s1 = fma(v0, c1[pyi * m1 + b], s1);
                s2 = fma(v1, c0[pyi * m1 + b], s2);
            }
        } else {
            s0 = s_a0[a];
        }
        s_b0[t] = s0;
        s_b1[t] = fma(s1, P.f[1], s2);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < size.k; t += blockDim.x) {
        const int pp = t / px, pxi = t - pp * px;
        double s0 = 0.0, s1 = 0.0;
        for (int a = 0; a < mx; ++a) {
            s0 = fma(s_b0[pp * mx + a], c1[pxi * m1 + a], s0);
            s1 = fma(s_b1[pp * mx + a], c0[pxi * m1 + a], s1);
        }
        s_k[t] = fma(s0, P.f[0], s1);
    }
    __syncthreads();
    const int n1 = S.n1;
    int nb = 1;
    for (int d = 0; d < dim; ++d) nb *= n1;
    V* o = out + static_cast<long>(blockIdx.x) * nb * nb;
    auto pair = [](int i, int j) { return i < j ? j * (j + 1) / 2 + i : i * (i + 1) / 2 + j; };
    for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) {
        const int a = t / nb, b = t - a * nb;
        int at = pair(a % n1, b % n1);
        if (dim > 1) at += px * pair((a / n1) % n1, (b / n1) % n1);
        if (dim > 2) at += px * py * pair(a / (n1 * n1), b / (n1 * n1));
        o[t] = static_cast<V>(s_k[at]);
    }
    (void)pz;
}

template <int DIM, int ORDER, typename V>
int launch_cells(const EmbeddedArgs& A, const int* cutCells, long first, long count, const double* pairTable, V* out,
                 cudaStream_t st) {
    const int warps = A.maxDepth >= 1 ? (1 << A.dim) : 1;
    const size_t smem = sizeof(double) * fc_smem(A.dim, A.order, A.q1, warps).total;
    auto kernel = fc_cell_kernel<DIM, ORDER, V>;
    CIECU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
    kernel<<<static_cast<unsigned>(count), 32 * warps, smem, st>>>(A, cutCells, static_cast<int>(first), pairTable, out);
    count_launch();
    CIECU_CHECK_LAUNCH("fc_cell_kernel");
    return CIECU_OK;
}

// c0 and c1 of the 1-D basis: coefficients (2a + 1)/2 int f P_a of the products f,
// by a Gauss rule that is exact for them (degree 4 order).
std::vector<double> pair_table(int order) {
    const int n1 = order + 1, m1 = 2 * order + 1, pairs = n1 * (n1 + 1) / 2;
    std::vector<double> x, w, out(static_cast<size_t>(2 * pairs * m1), 0.0);
    gauss_legendre(m1, x, w);
    for (int a = 0; a < m1; ++a)
        for (int j = 0, at = 0; j < n1; ++j)
            for (int i = 0; i <= j; ++i, ++at) {
                long double s0 = 0.0L, s1 = 0.0L;
                for (int q = 0; q < m1; ++q) {
                    double v[16], dv[16];
                    lagrange(order, x[q], v, dv);
                    long double p0 = 1.0L, p1 = x[q];
                    for (int k = 1; k <= a; ++k) {
                        const long double p2 = ((2 * k + 1) * static_cast<long double>(x[q]) * p1 - k * p0) / (k + 1);
                        p0 = p1;
                        p1 = p2;
                    }
                    s0 += static_cast<long double>(w[q]) * v[i] * v[j] * p0;
                    s1 += static_cast<long double>(w[q]) * dv[i] * dv[j] * p0;
                }
                out[static_cast<size_t>(at) * m1 + a] = static_cast<double>((2 * a + 1) * s0 / 2);
                // the products of derivatives have degree 2 order - 2
                out[static_cast<size_t>(pairs + at) * m1 + a] =
                    a <= 2 * order - 2 ? static_cast<double>((2 * a + 1) * s1 / 2) : 0.0;
            }
    return out;
}

// The row gather's cells: regular cells kappa s K1 (first batch only), the cut
// cells of the batch kappa scale times their own matrix.
template <typename V>
struct FiniteCellSource {
    const int* __restrict__ cut;
    const int* __restrict__ index;
    const signed char* __restrict__ side;
    const V* __restrict__ cutMatrix;
    const double* __restrict__ kappa;
    double alpha, scale;
    int nb2, batchFirst, batchEnd, withRegular;
    __device__ __forceinline__ bool adds(int e) const {
        return cut[e] ? index[e] >= batchFirst && index[e] < batchEnd : withRegular != 0;
    }
    __device__ __forceinline__ V coef(int e) const {
        const double kap = kappa ? kappa[e] : 1.0;
        return static_cast<V>(cut[e] ? kap * scale : kap * (side[e] ? 1.0 : alpha));
    }
    __device__ __forceinline__ const V* matrix(int e, const V* K) const {
        return cut[e] ? cutMatrix + static_cast<long>(index[e] - batchFirst) * nb2 : K;
    }
};

__global__ void to_float_kernel(int n, const double* __restrict__ a, float* __restrict__ b) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = static_cast<float>(a[i]);
}

template <bool F64>
int assemble_finite_cell(ciecu_assembly_s* P, const double* d_kappa, const double* h_cellSize, const int32_t* h_cells,
                         const double* h_origin, const double* h_center, double radius, double alpha, int maxDepth,
                         int convention, int accumulate, void* d_entries, int64_t* h_cutCells) {
    using V = typename std::conditional<F64, double, float>::type;
    CIECU_REQUIRE(P && h_cellSize && h_cells && h_origin && h_center && d_entries, "assemble_embedded: null argument");
    CIECU_REQUIRE(convention == 0 || convention == 1, "assemble_embedded: convention must be 0 or 1");
    CIECU_REQUIRE(P->nb <= 64 && P->order + 1 <= 16, "assemble_embedded: at most 64 basis functions per cell");
    CIECU_REQUIRE(P->q1 <= 16, "assemble_embedded: at most 16 quadrature points per axis");
    CIECU_REQUIRE(maxDepth >= 0 && maxDepth <= 4, "assemble_embedded: tree depth must be in [0, 4]");
    CIECU_REQUIRE(radius > 0.0, "assemble_embedded: radius must be positive");
    long cellsTotal = 1;
    for (int d = 0; d < P->dim; ++d) {
        CIECU_REQUIRE(h_cells[d] >= 1, "assemble_embedded: empty grid");
        cellsTotal *= h_cells[d];
    }
    CIECU_REQUIRE(cellsTotal == P->ncells, "assemble_embedded: grid size differs from the plan's cell count");
    cudaStream_t st = P->csr->space->stream;
    const long ncells = P->ncells;
    const int nb = P->nb, nb2 = nb * nb;
    if (ncells == 0) {
        if (!accumulate) CIECU_CUDA(cudaMemsetAsync(d_entries, 0, sizeof(V) * P->csr->nnz, st));
        if (h_cutCells) *h_cutCells = 0;
        return CIECU_OK;
    }
    EmbeddedArgs A{};
    A.dim = P->dim;
    A.order = P->order;
    A.nb = nb;
    A.q1 = P->q1;
    A.nq = P->nq;
    A.maxDepth = maxDepth;
    for (int d = 0; d < 3; ++d) {
        A.cells[d] = d < P->dim ? h_cells[d] : 1;
        A.origin[d] = d < P->dim ? h_origin[d] : 0.0;
        A.h[d] = d < P->dim ? h_cellSize[d] : 1.0;
        A.center[d] = d < P->dim ? h_center[d] : 0.0;
    }
    for (int i = 0; i < P->q1; ++i) {
        A.gn[i] = P->gn[i];
        A.gw[i] = P->gw[i];
    }
    A.radius2 = radius * radius;
    A.alpha = alpha;
    double f[3];
    convention_factors(P->dim, h_cellSize, convention, A.scale, f);
    for (int d = 0; d < 3; ++d) A.f[d] = f[d];
    // batches of cut cells whose matrices fit in 512 MB
    const long perCut = nb2 * static_cast<long>(sizeof(V));
    const long batchCap = std::max<long>(1, (512L << 20) / perCut);
    // work: K1 (FP64 and V), the pair table, cut flags, their prefix sum, cut list, sides, scan work
    const std::vector<double> pairs = pair_table(P->order);
    const long scanWork = scan_work(ncells);
    const size_t bytes = sizeof(double) * (nb2 + pairs.size()) + sizeof(V) * nb2 +
                         sizeof(int) * (3 * static_cast<size_t>(ncells) + 1 + static_cast<size_t>(scanWork)) +
                         static_cast<size_t>(ncells) + 256;
    unsigned char* work = nullptr;
    CIECU_CUDA(pool_alloc(&work, bytes, st));
    V* matrices = nullptr;
    auto done = [&](int status) {  // stream-ordered: the kernels that use them come first
        if (matrices) cudaFreeAsync(matrices, st);
        cudaFreeAsync(work, st);
        return status;
    };
    double* K1 = reinterpret_cast<double*>(work);
    double* pairTable = K1 + nb2;
    V* K1v = reinterpret_cast<V*>(pairTable + pairs.size());
    int* cut = reinterpret_cast<int*>(
        work + ((sizeof(double) * (nb2 + pairs.size()) + sizeof(V) * nb2 + 15) & ~size_t(15)));
    int* index = cut + ncells;       // ncells + 1
    int* cutCells = index + ncells + 1;
    int* scan = cutCells + ncells;
    signed char* side = reinterpret_cast<signed char*>(scan + scanWork);
    int status = unit_element(P, A.scale, f, K1, st);
    if (status != CIECU_OK) return done(status);
    if constexpr (F64) {
        cudaError_t e = cudaMemcpyAsync(K1v, K1, sizeof(double) * nb2, cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return done(cuda_fail(e, "assemble_embedded"));
    } else {
        to_float_kernel<<<(nb2 + 255) / 256, 256, 0, st>>>(nb2, K1, K1v);
        count_launch();
    }
    fc_classify_kernel<<<grid_for(ncells * 32, 256, 8), 256, 0, st>>>(A, ncells, cut, side);
    count_launch();
    status = exclusive_scan(cut, index, ncells, scan, st);
    if (status != CIECU_OK) return done(status);
    fc_compact_kernel<<<grid_for(ncells, 256, 8), 256, 0, st>>>(ncells, cut, index, cutCells);
    count_launch();
    cudaError_t e = cudaMemcpyAsync(pairTable, pairs.data(), sizeof(double) * pairs.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return done(cuda_fail(e, "assemble_embedded: pair table"));
    int ncut = 0;
    e = cudaMemcpyAsync(&ncut, index + ncells, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return done(cuda_fail(e, "assemble_embedded: classification"));
    const long batch = std::min<long>(std::max(ncut, 1), batchCap);
    if (ncut > 0) {
        e = pool_alloc(&matrices, static_cast<size_t>(batch * perCut), st);
        if (e != cudaSuccess) return done(cuda_fail(e, "assemble_embedded: cut-cell matrices"));
    }
    V* val = static_cast<V*>(d_entries);
    for (long b0 = 0; b0 < std::max<long>(ncut, 1); b0 += batch) {
        const long b1 = std::min<long>(ncut, b0 + batch);
        if (b1 > b0) {
            const int shape = A.dim * 10 + A.order;
            auto cells = [&](auto d, auto p) {
                return launch_cells<decltype(d)::value, decltype(p)::value, V>(A, cutCells, b0, b1 - b0, pairTable,
                                                                               matrices, st);
            };
            using std::integral_constant;
            if (shape == 33) status = cells(integral_constant<int, 3>{}, integral_constant<int, 3>{});
            else if (shape == 32) status = cells(integral_constant<int, 3>{}, integral_constant<int, 2>{});
            else if (shape == 31) status = cells(integral_constant<int, 3>{}, integral_constant<int, 1>{});
            else status = cells(integral_constant<int, 0>{}, integral_constant<int, 0>{});
            if (status != CIECU_OK) return done(status);
        }
        status = launch_row_gather<V>(P,
                                      FiniteCellSource<V>{cut, index, side, matrices, d_kappa, alpha, A.scale, nb2,
                                                          static_cast<int>(b0), static_cast<int>(b1), b0 == 0 ? 1 : 0},
                                      K1v, accumulate || b0 > 0 ? 1 : 0, val, st);
        if (status != CIECU_OK) return done(status);
    }
    e = cudaStreamSynchronize(st);  // part of the call's contract
    if (e != cudaSuccess) return done(cuda_fail(e, "assemble_embedded"));
    if (h_cutCells) *h_cutCells = ncut;
    return done(CIECU_OK);
}

}  // namespace
}  // namespace ciecu

using namespace ciecu;

extern "C" {

int ciecu_assemble_embedded(ciecu_assembly P, const double* d_kappa, const double* h_cellSize, const int32_t* h_cells,
                            const double* h_origin, const double* h_center, double radius, double alpha, int maxDepth,
                            int convention, int accumulate, double* d_entries, double* d_work, int64_t* h_cutCells) {
    CIECU_REQUIRE(d_work, "assemble_embedded: null argument");
    return assemble_finite_cell<true>(P, d_kappa, h_cellSize, h_cells, h_origin, h_center, radius, alpha, maxDepth,
                                      convention, accumulate, d_entries, h_cutCells);
}

int ciecu_assemble_embedded_f32(ciecu_assembly P, const double* d_kappa, const double* h_cellSize,
                                const int32_t* h_cells, const double* h_origin, const double* h_center, double radius,
                                double alpha, int maxDepth, int convention, int accumulate, float* d_entries32,
                                int64_t* h_cutCells) {
    return assemble_finite_cell<false>(P, d_kappa, h_cellSize, h_cells, h_origin, h_center, radius, alpha, maxDepth,
                                       convention, accumulate, d_entries32, h_cutCells);
}

}  // extern "C"
