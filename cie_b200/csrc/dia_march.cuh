// Row sums over the upper half of a bitwise symmetric DIA matrix of the 3D Q1 stencil,
// every entry read from memory once: for matrices past L2.
//
// The offsets are {dz S + dy N + dx}, dx, dy, dz in {-1, 0, 1} (S rows to a plane, N to a
// line).  A block owns a tile of T consecutive rows of a plane and marches through a run
// of planes, a row of the plane to a thread.  A producer warp brings, plane by plane, the
// windows of the operand and of the 14 upper diagonals that the tile's rows touch to
// shared memory, by bulk copies into two rings of slots; the warps free a slot when they
// are done with it.  The lower entries A[r][r - o] = U_o[r - o] of a row are in the same
// windows (o < S), or in those of the plane before (o >= S), which stay for one step more.
// So L2 is read about 1.3 times (the tile's halo of N + 1 rows to either side) instead of
// the two times of dia_rows_sym, whose lower entries come from L2 again.
//
// Lower terms from the farthest diagonal in, the main diagonal, the upper ones, one FMA
// each: the column order of dia_rows on the full copy, the same sums bit for bit.  Rows
// outside [0, n) hold zeros in the windows.
//
// What bounds it: HBM, 240 MB of matrix and 34 of vectors at 129^3 rows, 42 us; 52 us
// measured, 78 by dia_rows_sym, which reads 600 MB through L2.  With a copy for each diagonal
// of a triple (15 a plane instead of 7, about 250 cycles each for the producer) 56; a warp
// that takes the matrix's first or last rows fills zeros alone (100 when it went through
// whole windows).  In FP32 the row pass itself binds, 47 us, and reading the full matrix
// once (dia_rows4_triples, 41 us) is faster.
//
// Every wait is bounded.  After one has given up the warps of rows free no slot any more,
// the producer brings nothing more, all run to their end without waiting, and op.expired()
// tells.
#pragma once

#include "dia.cuh"
#include "space.cuh"

#include <algorithm>
#include <cstdint>

namespace ciecu {

constexpr int kDmAlign = 128;   // bytes that a copy starts at, in both memories
constexpr int kDmOperands = 5;  // operand windows: planes z - 1, z, z + 1 and two ahead

constexpr int kDmThreads = 736;  // 22 warps of rows and the producer, up to 88 registers
constexpr int kDmSlots = 8;      // of a triple's window each; a plane takes 5, 3 of the plane before stay

struct DmArgs {
    const double* __restrict__ triples;  // (N, S - N, S, S + N) -1, +0, +1: triple k of row r at (k ld + r) 3
    const double* __restrict__ upper;    // the main diagonal, and offset 1 at upper + ld
    long ld;
    int n, S, N;
    int T, tiles;     // rows of a tile, tiles of a plane
    int run, planes;  // planes of a block at most, planes of the matrix
    int W;            // rows of a window
    long long waitClocks;  // bound of a wait
    int withholdPlane;     // test hook: block 0 leaves out a copy in its plane of this number, from 1 (0: none)
};

constexpr long long kDmWaitClocks = 1LL << 31;  // about a second

struct DmPlan {
    DmArgs args{};
    int blocks = 0;  // 0: the matrix is none for it
    size_t smem = 0;
};

__device__ __forceinline__ unsigned dm_shared(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool dm_wait(const unsigned long long* bar, unsigned parity, long long limit,
                                        volatile int* failed) {
    unsigned ok = 0;
    for (long long begun = clock64();;) {
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(dm_shared(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*failed || clock64() - begun > limit) {
            *failed = 1;
            return false;
        }
    }
}

__device__ __forceinline__ void dm_arrive(const unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dm_shared(bar)) : "memory");
}

// Producer warp: rows [w0, w1) of PITCH values each of `count` arrays into windows W rows
// apart, a window beginning at w0 rounded down to kDmAlign bytes; zeros outside [0, n).
template <int PITCH>
__device__ __forceinline__ void dm_bring(double* to, int W, const double* from, long stride, int count, int w0, int w1, int n,
                                         const unsigned long long* bar, bool go, bool withhold = false) {
    constexpr int Q = kDmAlign / 8, R = 2;
    const int lane = threadIdx.x & 31;
    const int s0 = w0 & ~(Q - 1);
    const int lo = max(s0, 0);
    int end = (w1 + R - 1) & ~(R - 1);
    if (lo != s0 || end > n) {  // the matrix's first or last rows
        end = max(min(end, n & ~(R - 1)), lo);
        for (int k = 0; k < count; ++k) {
            double* row = to + k * W;
            for (int i = lane; i < (min(lo, w1) - s0) * PITCH; i += 32) row[i] = 0.0;
            for (int i = (end - s0) * PITCH + lane; i < (w1 - s0) * PITCH; i += 32)
                row[i] = s0 * PITCH + i < n * static_cast<long>(PITCH) ? from[k * stride + s0 * static_cast<long>(PITCH) + i]
                                                                      : 0.0;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
    }
    const int bytes = (end - lo) * PITCH * 8;
    if (lane == 0 && go)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(dm_shared(bar)), "r"(bytes * count)
                     : "memory");
    __syncwarp();
    if (lane < count && bytes > 0 && go && !withhold)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         dm_shared(to + lane * W + (lo - s0) * PITCH)),
                     "l"(from + lane * stride + lo * static_cast<long>(PITCH)), "r"(bytes), "r"(dm_shared(bar))
                     : "memory");
}

// Op: Pre pre(row), post(row, pre, sum), expired().
template <typename Op>
__device__ __forceinline__ void dm_rows(const DmArgs& A, const double* __restrict__ x, Op& op) {
    extern __shared__ __align__(128) unsigned char dm_smem[];
    constexpr int kDmBars = 2 * (kDmSlots + kDmOperands);
    __shared__ __align__(8) unsigned long long bars[kDmBars];
    __shared__ int s_failed;
    double* slots = reinterpret_cast<double*>(dm_smem);
    double* operands = slots + kDmSlots * 3 * A.W;
    unsigned long long *slotFull = bars, *slotFree = bars + kDmSlots, *opFull = bars + 2 * kDmSlots,
                       *opFree = bars + 2 * kDmSlots + kDmOperands;
    constexpr int kWarps = kDmThreads / 32 - 1;
    constexpr int Q = kDmAlign / 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_failed = 0;
        for (int k = 0; k < kDmBars; ++k) {
            const bool full = k < kDmSlots || (k >= 2 * kDmSlots && k < 2 * kDmSlots + kDmOperands);
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(dm_shared(bars + k)), "r"(full ? 1 : kWarps)
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int tile = static_cast<int>(blockIdx.x) % A.tiles, part = static_cast<int>(blockIdx.x) / A.tiles;
    const int a = tile * A.T, width = min(A.T, A.S - a);
    const int z0 = part * A.run, z1 = min(z0 + A.run, A.planes);
    const int N = A.N, S = A.S, W = A.W;
    if (z0 < z1) {
        if (warp == kWarps) {
            int slot = 0, turn = 0, opSlot = 0, opTurn = 0;
            // After a wait that gave up the lane neither arms a barrier nor copies: the slot may
            // be in use, and a barrier armed in a phase that has not ended gets an arrival too
            // many.  (Lanes keep together: the branches around them stay those of the others.)
            bool stop = false;
            auto until_free = [&](const unsigned long long* bar, int turns) {
                if (turns && !dm_wait(bar, (turns - 1) & 1, A.waitClocks, &s_failed)) stop = true;
            };
            auto slot_next = [&]() {
                if (++slot == kDmSlots) slot = 0, ++turn;
            };
            auto triple = [&](int k, int w0, int w1, bool withhold = false) {
                until_free(slotFree + slot, turn);
                dm_bring<3>(slots + slot * 3 * W, 0, A.triples + k * A.ld * 3, 0, 1, w0, w1, A.n, slotFull + slot, !stop,
                            withhold);
                slot_next();
            };
            auto operand = [&](int w0, int w1) {
                until_free(opFree + opSlot, opTurn);
                dm_bring<1>(operands + opSlot * W, 0, x, 0, 1, w0, w1, A.n, opFull + opSlot, !stop);
                if (++opSlot == kDmOperands) opSlot = 0, ++opTurn;
            };
            for (int z = z0 - 1; z < z1; ++z) {
                const int w0 = z * S + a - N - 1, own = z * S + a + width, w1 = own + N + 1;
                if (z < z0) operand(w0, w1);
                operand(w0 + S, w1 + S);
                if (z >= z0) {
                    triple(0, w0, own, blockIdx.x == 0 && z - z0 + 1 == A.withholdPlane);
                    until_free(slotFree + slot, turn);
                    dm_bring<1>(slots + slot * 3 * W, W, A.upper, A.ld, 2, w0, own, A.n, slotFull + slot, !stop);
                    slot_next();
                }
                for (int k = 1; k <= 3; ++k) triple(k, w0, w1);
            }
        } else {
            const int j = min(tid, width - 1);  // row of the plane
            int slot = 0, parity = 0, opSlot = 0, opParity = 0;
            bool dead = false;  // a wait gave up: the slots are freed no more, and the producer stops
            auto next = [&]() {  // the next slot, when it is full
                double* p = slots + slot * 3 * W;
                if (!dm_wait(slotFull + slot, parity, A.waitClocks, &s_failed)) dead = true;
                if (++slot == kDmSlots) slot = 0, parity ^= 1;
                return p;
            };
            auto next_operand = [&]() {
                double* p = operands + opSlot * W;
                if (!dm_wait(opFull + opSlot, opParity, A.waitClocks, &s_failed)) dead = true;
                if (++opSlot == kDmOperands) opSlot = 0, opParity ^= 1;
                return p;
            };
            auto at = [&](int z) {  // the row's place in the windows of plane z
                return z * S + a + j - ((z * S + a - N - 1) & ~(Q - 1));
            };
            const double* xm = next_operand();
            const double* xc = next_operand();
            const double* g[3];
            int gSlot = slot;
            for (int k = 0; k < 3; ++k) g[k] = next();
            int opFirst = 0;
            int bm = at(z0 - 1), bc = at(z0);
            auto row_of = [&](int z) { return z * S + a + j; };
            auto mine = [&](int z) { return tid < width && z < z1 && row_of(z) < A.n; };
            typename Op::Pre pre{};
            if (mine(z0)) pre = op.pre(row_of(z0));
            for (int z = z0; z < z1; ++z) {
                typename Op::Pre ahead{};
                if (mine(z + 1)) ahead = op.pre(row_of(z + 1));
                double sum = 0.0;
#pragma unroll
                for (int k = 2; k >= 0; --k)
#pragma unroll
                    for (int e = 2; e >= 0; --e) {
                        const int i = bm - (k - 1) * N - (e - 1);
                        sum = fma(g[k][3 * i + e], xm[i], sum);
                    }
                __syncwarp();
                if (lane == 0 && !dead) {
                    for (int k = 0; k < 3; ++k) dm_arrive(slotFree + (gSlot + k) % kDmSlots);
                    dm_arrive(opFree + opFirst);
                }
                if (++opFirst == kDmOperands) opFirst = 0;
                const int lineSlot = slot;
                const double* line = next();
                const double* self = next();
#pragma unroll
                for (int e = 2; e >= 0; --e) {
                    const int i = bc - N + 1 - e;
                    sum = fma(line[3 * i + e], xc[i], sum);
                }
                sum = fma(self[W + bc - 1], xc[bc - 1], sum);
                sum = fma(self[bc], xc[bc], sum);
                sum = fma(self[W + bc], xc[bc + 1], sum);
#pragma unroll
                for (int e = 0; e < 3; ++e) sum = fma(line[3 * bc + e], xc[bc + N - 1 + e], sum);
                __syncwarp();
                if (lane == 0 && !dead)
                    for (int k = 0; k < 2; ++k) dm_arrive(slotFree + (lineSlot + k) % kDmSlots);
                const double* xp = next_operand();
                const int bp = at(z + 1);
                gSlot = slot;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    g[k] = next();
#pragma unroll
                    for (int e = 0; e < 3; ++e) sum = fma(g[k][3 * bc + e], xp[bp + (k - 1) * N + e - 1], sum);
                }
                if (mine(z)) op.post(row_of(z), pre, sum);
                pre = ahead;
                xm = xc;
                xc = xp;
                bm = bc;
                bc = bp;
            }
        }
    }
    __syncthreads();
    if (s_failed) {  // no copy is in flight some milliseconds after the producer's last
        for (const long long begun = clock64(); clock64() - begun < (1LL << 24);) {
        }
        if (tid == 0) op.expired();
    }
}

// The interleaved triples of the upper half u.
__global__ void __launch_bounds__(256) dm_fill_kernel(DiaArgs<double> u, double* __restrict__ triples) {
    const int r = blockIdx.x * 256 + threadIdx.x;
    if (r >= u.ld) return;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 3; ++e) triples[(k * u.ld + r) * 3 + e] = u.val[(2 + 3 * k + e) * u.ld + r];
}

// The plan for the upper half `u` (dia_upper_view) of a bitwise symmetric matrix; blocks = 0
// when its offsets are no 3D Q1 stencil, a window does not fit, or the halo of a tile costs
// more than it saves (over five eighths of the tile).
inline DmPlan dm_plan(const DiaArgs<double>& u, int sms, size_t maxSmem) {
    DmPlan plan;
    if (u.ndiag != 14 || u.off[0] != 0 || u.off[1] != 1) return plan;
    const int N = u.off[3], S = u.off[9];
    if (N < 3 || S < 2 * N + 3) return plan;
    for (int k = 0; k < 3; ++k) {
        if (u.off[2 + k] != N - 1 + k) return plan;
        for (int e = 0; e < 3; ++e)
            if (u.off[5 + 3 * k + e] != S + (k - 1) * N + e - 1) return plan;
    }
    const long planes = (static_cast<long>(u.nrows) + S - 1) / S;
    constexpr int Q = kDmAlign / 8, R = 2;
    double best = 1e30;
    for (int tiles = 1; tiles <= sms; ++tiles) {
        const int T = (S + tiles - 1) / tiles;
        const int W = (T + 2 * N + 2 + Q + R + 15) / 16 * 16;
        const size_t smem = sizeof(double) * static_cast<size_t>(W) * (kDmSlots * 3 + kDmOperands);
        if (T > kDmThreads - 32 || smem > maxSmem) continue;
        const int used = (S + T - 1) / T;
        const long runs = std::min<long>(std::max(1, sms / used), planes), run = (planes + runs - 1) / runs;
        const double cost = (run + 1.5) * (T + 2.0 * N);  // the first plane brings its predecessor's diagonals
        if (2 * N > T / 2 + T / 8 || cost >= best) continue;
        best = cost;
        plan.args =
            DmArgs{nullptr, u.val, u.ld, u.nrows, S, N, T, used, static_cast<int>(run), static_cast<int>(planes), W,
                   kDmWaitClocks, 0};
        plan.blocks = used * static_cast<int>((planes + run - 1) / run);
        plan.smem = smem;
    }
    return plan;
}

// The plan of a solver and its copy of the triples (from the pool; not yet filled), with the
// kernels' shared memory opted in.  `operand` is the vector that they read.  None where the
// upper half is smaller than leastBytes, or where there is no room for the copy.
inline int dm_prepare(const DiaArgs<double>& u, long leastBytes, std::initializer_list<const void*> kernels, const double* operand,
               cudaStream_t st, DmPlan* out, double** copy) {
    *out = DmPlan{};
    const uintptr_t places = reinterpret_cast<uintptr_t>(operand) | reinterpret_cast<uintptr_t>(u.val);
    if (14L * u.nrows * 8 < leastBytes || u.nrows > (1 << 28) || (places & (kDmAlign - 1)))
        return CIECU_OK;
    int device = 0, optin = 0;
    CIECU_CUDA(cudaGetDevice(&device));
    CIECU_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    DmPlan plan = dm_plan(u, sm_count(), static_cast<size_t>(std::max(optin - 2048, 0)));
    if (!plan.blocks) return CIECU_OK;
    for (const void* kernel : kernels)
        CIECU_TRY(allow_shared(kernel));
    double* triples = nullptr;
    if (pool_alloc(&triples, sizeof(double) * 12 * static_cast<size_t>(u.ld), st) != cudaSuccess) {
        cudaGetLastError();
        return CIECU_OK;
    }
    plan.args.triples = triples;
    *copy = triples;
    *out = plan;
    return CIECU_OK;
}

inline int dm_fill(const DiaArgs<double>& u, double* triples, cudaStream_t st) {
    dm_fill_kernel<<<static_cast<unsigned>((u.ld + 255) / 256), 256, 0, st>>>(u, triples);
    count_launch();
    CIECU_CHECK_LAUNCH("dm_fill_kernel");
    return CIECU_OK;
}

}  // namespace ciecu
