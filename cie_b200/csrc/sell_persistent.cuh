// Conjugate-gradient iterations over sparse matrices of moderate bandwidth that are
// no DIA matrices (high-order meshes, batches of them) in ONE cooperative launch:
// the batched solver (batched.cu, many systems) and the FP64 solver (pcg.cu, one).
//
// A system is shared out to a group of blocks, R rows (a multiple of 32) to each; the
// iteration's two phases, their exchanges and decisions are those of
// dia_persistent.cuh, within the group.  Every block works through a list of
// (system, part) items in the order in which the systems were planned: the first
// unfinished system has all its blocks, so no block waits for ever; every wait is
// bounded all the same.
//
// The matrix is an FP64 copy in slices of 32 rows, two entries of a row to a lane: step
// t of a slice holds entries 2t and 2t + 1 of its rows as 16 bytes of values and two
// 16-bit column offsets (column - row) per lane, so a warp reads 512 + 128 contiguous
// bytes a step.  The rows of kSpSort consecutive rows of a system are dealt to its
// slices by length (a row's place is in `row`), so that the rows of a slice are about
// equally long: high-order meshes alternate vertex rows with much shorter ones (3D Q2:
// 36 % padding with the rows as they come) (a row of one entry per lane and 12-byte entries is bound by the
// requests, about one per 6 cycles and SM, before it is by L2).  Padding has value 0
// and offset 0.  A row is summed by one thread in column order, one FMA per entry:
// the sequential sum of CSROperator.cpp:49-56.  Up to kFewLongRows rows of more than kLongRow
// entries are summed by a warp each instead, from the matrix itself: 75,777 rows of 48 and
// two of 8,300 27 us an iteration, 190 with a thread for each; 300,000 rows and two of 3,650
// 40 and 219.  (Where all rows are long a thread for each is better: 40,000 rows of 801 66,
// 115 by warps.)  The operand entries of a block's rows
// lie in one window of R + span columns, formed in shared memory from the z and
// p_{k-1} of the owners: even columns in its first half, odd ones in its second
// (sp_place), as the rows of a slice are mostly every other row or neighbours, and
// 32 operands then fill two wavefronts.  A block's q, r and x, and p and D^-1 where they fit, stay in
// shared memory for the solve.
//
// Batches: as many rows are in flight at a time as keep the copies of their matrices in
// L2 (kSpRows to a block), where all systems at once stream every matrix from HBM in
// every iteration and run three kernels over the whole batch until its last system is
// done.
//
// What bounds it: reading the copy from L2 at 10 bytes an entry (Q2 batch, 2,816 rows a
// block: rows 15,000 of 33,000 cycles, exchanges 10,000, windows 3,600); one 3D Q2
// system of 250,047 rows and 14.8 M entries (148 MB, past L2) from HBM: 52 us an
// iteration against 65 us by the graph of three kernels over CSR (12 bytes an entry).
// Measured at 64 Q2 systems / the 3D Q2 system: natural row order 89 / 18.3 ms, rows
// dealt by length 81 / 16.5, a warp's slices back and forth 78 / 14.3, odd and even
// columns apart 68 / 13.3; threads x unroll 1024 x 4, 896 x 6, 640 x 8, 512 x 12 before
// the last step: 76 / 14.3, 82 / 13.7, 77 / 14.3, 74 / 13.2; blocks of 2,048, 2,816,
// 3,584, 4,480 rows: 68, 68, 69, 79 ms.
#pragma once

#include "dia_persistent.cuh"

#include <climits>
#include <vector>

namespace ciecu {

constexpr int kSpThreads = 512;      // at most: 16 warps of up to 128 registers
constexpr int kSpSort = 128;         // rows that share their slices; parts are multiples of it
constexpr int kSpRows = 2816;        // rows of a block at most: 148 blocks' matrices stay in L2 (Q2: 200 B a row)
constexpr int kSpUnroll = 12;        // steps of a row in flight
constexpr int kSpLongUnroll = 8;     // entries of a lane in flight in a long row

struct SpItem {
    int system, part, parts;  // part of the system's `parts` blocks
    int rowBegin, rows;       // global rows
    int sliceBegin;
    int sysBegin, sysEnd;     // rows of the system
    int lo, span;             // window: columns rowBegin + lo .. rowBegin + rows - 1 + lo + span
    int slotBase;             // words of the system start at slotBase * kSpWords
    int longBegin, longRows;  // the part's rows that are in no slice
};

constexpr int kSpWords = 2 * 2 * kDpCopies;  // words a block has: sets x values x copies

struct SpMatrix {
    const double* __restrict__ val;
    const short2* __restrict__ off;
    const int* __restrict__ sliceStep;  // first step of each slice; one past the last
    const int* __restrict__ row;        // 32 per slice: the lane's row (-1: none)
    const int* __restrict__ longRow;    // rows that are in no slice, ascending
    // the matrix itself, for these
    const int* __restrict__ rowptr;
    const int* __restrict__ col;
    const double* __restrict__ entries;
};

struct SpArgs {
    SpMatrix A;
    const SpItem* __restrict__ items;
    const int* __restrict__ itemBegin;  // per block; gridDim.x + 1
    int R, winLen;                      // capacities of the shared arrays
    int homes;                          // kDpP, kDpD
    const double* __restrict__ dinv;
    double* x;
    double* r;
    double* z;
    double* p0;
    double* p1;
    DpSlot* slots;
    int* abortFlag;
    unsigned long long epoch0;
    long long waitNs;
    unsigned long long withholdEpoch;
};

// Place of window column x in a window of `half` places a half.
__host__ __device__ __forceinline__ int sp_place(int x, int half) { return (x & 1) * half + (x >> 1); }

// Ctl: Scalars, Shared (settings of the launch), and as in dia_persistent.cuh
// start / afterProduct / afterUpdate with the settings as a further argument, and
// finish(scalars, settings) run by the system's first block after its last exchange.
// LONG: some rows are in no slice (a kernel of its own: the test alone cost 1 % of a batch).
template <bool PRECOND, bool LONG, typename Ctl>
__device__ __forceinline__ void sp_solve(const SpArgs& P, typename Ctl::Scalars* scalars, typename Ctl::Shared shared) {
    extern __shared__ __align__(16) unsigned char sp_smem[];
    __shared__ typename Ctl::Scalars s_scalars;
    __shared__ DpCommand s_cmd;
    __shared__ double s_red[64];
    __shared__ int s_ok, s_run;
    __shared__ SpItem s_item;
    __shared__ DpGroup s_group;
    const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* s_win = reinterpret_cast<double*>(sp_smem);
    double* sq = s_win + P.winLen;
    double* sr = sq + P.R;
    double* sx = sr + P.R;
    double* next = sx + P.R;
    double* sp = P.homes & kDpP ? next : nullptr;
    if (sp) next += P.R;
    double* sd = PRECOND && (P.homes & kDpD) ? next : nullptr;
    if (sd) next += P.R;
    int* s_step = reinterpret_cast<int*>(next);                     // R / 32 + 1 first steps
    short* s_row = reinterpret_cast<short*>(s_step + P.R / 32 + 1);  // R places: the row in the block, -1: none
    const SpItem& I = s_item;
    for (int it = P.itemBegin[blockIdx.x]; it < P.itemBegin[blockIdx.x + 1]; ++it) {
        __syncthreads();  // the item before is done with the shared arrays
        if (tid == 0) {
            s_item = P.items[it];
            s_group = DpGroup{P.slots + static_cast<size_t>(I.slotBase) * kSpWords, 2 * kDpCopies * I.parts,
                              kDpCopies * I.parts, I.parts, I.part, P.abortFlag, P.waitNs, P.withholdEpoch};
            s_scalars = scalars[I.system];
            s_run = *reinterpret_cast<volatile int*>(P.abortFlag) ? 2 : (Ctl::start(s_scalars, s_cmd, shared) ? 1 : 0);
        }
        __syncthreads();
        if (s_run == 2) return;
        if (s_run == 0) continue;  // the same in the whole group: scalars are written after its last exchange
        const int rb = I.rowBegin, nr = I.rows;
        for (int i = tid; i < nr; i += T) {
            sr[i] = P.r[rb + i];
            sx[i] = P.x[rb + i];
            if (sd) sd[i] = P.dinv[rb + i];
        }
        const int slices = (nr + kSpSort - 1) / kSpSort * (kSpSort / 32);
        for (int k = tid; k <= slices; k += T) s_step[k] = P.A.sliceStep[I.sliceBegin + k];
        for (int k = tid; k < 32 * slices; k += T) {
            const int row = P.A.row[static_cast<long>(I.sliceBegin) * 32 + k];
            s_row[k] = static_cast<short>(row < 0 ? -1 : row - rb);
        }
        const double* hd = sd ? sd : P.dinv + rb;
        unsigned long long epoch = P.epoch0;
        bool aborted = false;
        while (true) {
            // ---- S --------------------------------------------------------------
            const double* pprev = s_cmd.parity ? P.p0 : P.p1;
            double* pcur = s_cmd.parity ? P.p1 : P.p0;
            const double beta = s_cmd.beta;
            const bool first = s_cmd.first;
            const int len = nr + I.span;
            for (int x0 = tid; x0 < len; x0 += 4 * T) {
                double zv[4], pv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int x = x0 + u * T, c = rb + I.lo + x;
                    const bool in = x < len && c >= I.sysBegin && c < I.sysEnd;
                    zv[u] = in ? __ldcg(P.z + c) : 0.0;
                    pv[u] = in && !first ? __ldcg(pprev + c) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int x = x0 + u * T, i = x + I.lo;
                    if (x >= len) break;
                    const double p = first ? zv[u] : dp_direction(zv[u], beta, pv[u]);
                    s_win[sp_place(x, P.winLen / 2)] = p;
                    if (i >= 0 && i < nr) {
                        pcur[rb + i] = p;
                        if (sp) sp[i] = p;
                    }
                }
            }
            __syncthreads();
            double pq = 0.0;
            // A warp's slices back and forth: those of a run of kSpSort rows get shorter
            // from one to the next.
            const int warps = T / 32;
            for (int s0 = 0, k = 0; s0 < slices; s0 += warps, ++k) {
                const int s = s0 + (k & 1 ? warps - 1 - warp : warp);
                if (s >= slices) continue;
                const int row = s_row[32 * s + lane];
                const int t0 = s_step[s], t1 = s_step[s + 1];
                const double2* v = reinterpret_cast<const double2*>(P.A.val) + static_cast<long>(t0) * 32 + lane;
                const short2* o = P.A.off + static_cast<long>(t0) * 32 + lane;
                const double* operand = s_win + sp_place(max(row, 0) - I.lo, P.winLen / 2);
                double sum = 0.0;
                for (int t = t0; t < t1; t += kSpUnroll) {
                    double2 a[kSpUnroll];
                    short2 c[kSpUnroll];
#pragma unroll
                    for (int u = 0; u < kSpUnroll; ++u) {
                        const bool in = t + u < t1;
                        a[u] = in ? __ldg(v + 32 * u) : make_double2(0.0, 0.0);
                        c[u] = in ? __ldg(o + 32 * u) : make_short2(0, 0);
                    }
#pragma unroll
                    for (int u = 0; u < kSpUnroll; ++u) {
                        sum = fma(a[u].x, operand[c[u].x], sum);
                        sum = fma(a[u].y, operand[c[u].y], sum);
                    }
                    v += 32 * kSpUnroll;
                    o += 32 * kSpUnroll;
                }
                if (row >= 0) {
                    sq[row] = sum;
                    pq = fma(operand[0], sum, pq);
                }
            }
            // A long row to a warp, from the matrix itself: one thread would take 20 ns an entry.
            for (int k = warp; LONG && k < I.longRows; k += warps) {
                const int row = P.A.longRow[I.longBegin + k], k1 = P.A.rowptr[row + 1];
                const int at = -rb - I.lo, half = P.winLen / 2;
                double sum = 0.0;
                for (int e = P.A.rowptr[row] + lane; e < k1; e += 32 * kSpLongUnroll) {
                    double a[kSpLongUnroll];
                    int c[kSpLongUnroll];
#pragma unroll
                    for (int u = 0; u < kSpLongUnroll; ++u) {
                        const bool in = e + 32 * u < k1;
                        a[u] = in ? __ldg(P.A.entries + e + 32 * u) : 0.0;
                        c[u] = in ? __ldg(P.A.col + e + 32 * u) : row;
                    }
#pragma unroll
                    for (int u = 0; u < kSpLongUnroll; ++u) sum = fma(a[u], s_win[sp_place(c[u] + at, half)], sum);
                }
                sum = warp_sum(sum);
                if (lane == 0) {
                    sq[row - rb] = sum;
                    pq = fma(s_win[sp_place(row + at, half)], sum, pq);
                }
            }
            __syncthreads();
            {
                const double mine[1] = {pq};
                if (!dp_exchange<1, false>(mine, 0, ++epoch, s_group, s_red, &s_ok, [&](const double (&tot)[1]) {
                        Ctl::afterProduct(s_scalars, s_cmd, shared, tot[0]);
                    })) {
                    aborted = true;
                    break;
                }
            }
            if (!s_cmd.go) break;
            // ---- U --------------------------------------------------------------
            const double alpha = s_cmd.alpha;
            const double* hp = sp ? sp : pcur + rb;
            double rr = 0.0, rz = 0.0;
            for (int i = tid; i < nr; i += T) {
                sx[i] = fma(alpha, hp[i], sx[i]);
                const double ri = fma(-alpha, sq[i], sr[i]);
                sr[i] = ri;
                const double zi = PRECOND ? __dmul_rn(ri, hd[i]) : ri;
                P.z[rb + i] = zi;
                rr = fma(ri, ri, rr);
                if (PRECOND) rz = fma(ri, zi, rz);
            }
            {
                const double mine[2] = {rr, rz};
                if (!dp_exchange<2, true>(mine, 1, ++epoch, s_group, s_red, &s_ok, [&](const double (&tot)[2]) {
                        Ctl::afterUpdate(s_scalars, s_cmd, shared, tot[0], PRECOND ? tot[1] : tot[0]);
                    })) {
                    aborted = true;
                    break;
                }
            }
            if (!s_cmd.go) break;
        }
        if (aborted) return;
        for (int i = tid; i < nr; i += T) {
            P.r[rb + i] = sr[i];
            P.x[rb + i] = sx[i];
        }
        if (I.part == 0 && tid == 0) {
            Ctl::finish(s_scalars, shared);
            scalars[I.system] = s_scalars;
        }
    }
}

// ---- the copy and the plan (sell_persistent.cu) ---------------------------------

struct SpPlan {
    int state = 0;  // 0 not built, 1 usable, 2 the matrix does not suit this form
    int grid = 0;
    int threads = 0;
    size_t smem = 0;
    SpArgs args{};  // A, items, itemBegin, R, winLen, homes
    long slices = 0, steps = 0;
    long longestList = 0;  // items of a block
    bool longRows = false;
    // device memory (library pool)
    double* val = nullptr;
    short2* off = nullptr;
    int* sliceStep = nullptr;
    int* row = nullptr;  // 32 per slice
    int* longRow = nullptr;
    SpItem* items = nullptr;
    int* itemBegin = nullptr;
    DpSlot* slots = nullptr;
};

// Where this form is taken; the caller has another one outside.
struct SpLimits {
    long rows = LONG_MAX;      // rows of a block at most
    // This share of the copy's entries to the matrix's, at most, where a thread each sums
    // more rows of over kLongRow entries than kFewLongRows.
    double padding = 1e30;
    long window = LONG_MAX;    // window entries of a block, or ...
    long entriesPerColumn = 0; // ... this many stored entries for each of them: every block forms its own
    // parts for each block at most, by the stored entries of a part on average
    bool (*rounds)(double rounds, double entries) = nullptr;
};

// Builds the copy's layout and column offsets and the plan for the systems
// [rowOffsets[s], rowOffsets[s + 1]) of a block-diagonal FP64 CSR matrix; state 2 outside
// the limits, and when the windows do not fit in shared memory or padding takes over 60 %.
int sp_build(SpPlan& plan, const ciecu_csr_s* csr, const std::vector<long long>& rowOffsets, const SpLimits& limits,
             cudaStream_t st);
// The copy's values from the live CSR values.
int sp_fill(const SpPlan& plan, const ciecu_csr_s* csr, cudaStream_t st);
void sp_destroy(SpPlan& plan);  // waits for the device

}  // namespace ciecu
