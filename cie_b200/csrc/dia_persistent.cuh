// Conjugate-gradient iterations over a DIA matrix in ONE cooperative launch, for
// the FP64 solver (pcg.cu) and the FP32 inner iteration of the mixed solver
// (mixed.cu).
//
// Block b owns rows [bR, (b + 1)R).  An iteration has two phases, each ending in a
// grid-wide exchange of the blocks' partial sums:
//   S  p_k = z_k + beta p_{k-1} and q = A p_k for the own rows; p^T q
//   U  x += alpha p_k, r -= alpha q, z = D^-1 r on the own rows; r^T r, r^T z
// The operand entries a block needs lie in a few windows of columns (the diagonals'
// offsets, merged where they are closer than R: the three planes of the 27-point
// stencil, the one band of the 9-point stencil).  A block forms p_k for whole windows
// in shared memory from the z and p_{k-1} that the owners published, and reads every
// row sum's operands from there; p is double-buffered in global memory so that no
// block overwrites entries another one still reads.  q, r, x and, where they fit, p
// and D^-1 of the own rows stay in shared memory for the whole launch.
//   RESIDENT   all diagonals of a block's rows fit in its shared memory too: they are
//              read once per launch;
//   otherwise  they are read from L2 in every iteration, all entries of a row in flight.
//
// Row sums run over the diagonals in ascending offset order, one FMA each, as
// dia_rows and dia_rows_sym do, so they equal theirs bit for bit.  SYM: the lower
// diagonals of a bitwise symmetric matrix are read from the upper ones, so only the
// upper half crosses HBM.
//
// An exchange: every warp's sums meet in shared memory, warp 0 publishes the
// block's sums as 16-byte (value, epoch) words, in kDpCopies copies so that the readers spread over L2, polls the words of all
// blocks (16-byte loads, all in flight at once: a word whose epoch matches carries
// its value),
// sums them in block order, takes the step's decisions on the scalars in shared
// memory, and releases the block.  All blocks hold bit-identical scalars and take
// the same branches.  Every wait is bounded in time; a wait that gives up sets the
// abort flag, every block leaves, and the host reports CIECU_ERR_TIMEOUT.  Two
// alternating sets of words suffice: a block publishes exchange e + 2 only after
// it has seen every block's e + 1, which a block publishes after reading all of e.
//
// What bounds it (FP64, 1.965 GHz, cycles of one iteration): 2D Q1 256^2, 15,500: the
// two exchanges 10,700 (two crossings of the chip, a fence and a division each), the
// windows 1,900, the rows 830, U 790.  3D Q1 64^3, 30,000: the rows 11,000 (59 MB of
// matrix from L2, 11 TB/s), the windows 4,000, U 2,500, the exchanges 11,000.  Eight
// copies of the words: 2D 256^2 takes 10.4 us with one copy, 8.4 with two, 8.3 with
// four, 7.9 with eight and with sixteen.
#pragma once

#include "dia.cuh"
#include "pcg.cuh"

#include <algorithm>
#include <type_traits>

namespace ciecu {

// Threads of a block at most.
template <bool RESIDENT>
constexpr int dp_threads() {
    return RESIDENT ? 512 : 1024;
}
constexpr int kDpCopies = 8;
constexpr int kDpMaxBlocks = 160;  // 5 polled words per lane of warp 0
constexpr int kDpBatch = 4;        // rows of U a thread has in flight

struct alignas(16) DpSlot {
    double v;
    unsigned long long epoch;
};

// Slots of one solver: 2 sets x 2 values x kDpCopies x kDpMaxBlocks.
constexpr size_t kDpSlotBytes = sizeof(DpSlot) * 2 * 2 * kDpCopies * kDpMaxBlocks;

enum DpHome { kDpQ = 1, kDpR = 2, kDpX = 4, kDpP = 8, kDpD = 16 };  // vectors kept in shared memory

// The blocks that take part in an exchange and their words: value k of copy c of
// block b in set s at words[s * setStride + k * valueStride + c * count + b].
struct DpGroup {
    DpSlot* words;
    int setStride, valueStride;
    int count, me;
    int* abortFlag;
    long long waitNs;
    unsigned long long withholdEpoch;  // test hook: the last block never publishes this epoch (0: none)
};

template <typename V>
struct DpArgs {
    DiaArgs<V> A;
    int R;                           // rows per block (a multiple of 32)
    int nwin, ownWin;                // windows, the one that holds offset 0
    int span;                        // window w: columns r + winLo[w] .. r + winLo[w] + span, at w * (R + span)
    int winLo[kMaxDiagonals + 3];
    int wofs[kMaxDiagonals];         // operand of row i on diagonal d: windows[wofs[d] + i]
    int minOff, maxOff;
    int homes;                       // DpHome bits
    const V* __restrict__ dinv;
    V* x;
    V* r;
    V* q;
    V* z;
    V* p0;  // p_k for even k
    V* p1;  // p_k for odd k
    DpSlot* slots;
    int* abortFlag;
    unsigned long long epoch0;
    long long waitNs;
    unsigned long long withholdEpoch;  // test hook: the last block never publishes this epoch (0: none)
};

// What warp 0's decisions hand to the block.
struct DpCommand {
    double alpha, beta;
    int go;      // 0: leave the loop
    int step;    // 0: x and r stay (an FP32 breakdown)
    int first;   // p = z
    int parity;  // p_k goes to p1 when set
};

__device__ __forceinline__ void dp_store(DpSlot* s, double v, unsigned long long epoch) {
    asm volatile(
        "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(s),
        "l"(__double_as_longlong(v)), "l"(epoch)
        : "memory");
}

__device__ __forceinline__ void dp_load(const DpSlot* s, double& v, unsigned long long& epoch) {
    long long bits;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(bits), "=l"(epoch)
                 : "l"(s)
                 : "memory");
    v = __longlong_as_double(bits);
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Sums `mine` over the group and runs decide(sums) in lane 0 of warp 0 of every
// block; the command it leaves in shared memory is valid for the whole block on
// return.  ORDER: the other blocks' stores before their publication are visible
// afterwards.  (The exchange after S needs no such order: the stores of p_k become
// visible with the exchange after U, and the published sum depends on every entry
// the block has read, so no block can overwrite an entry before it was read.)  False when a wait gave up or another block aborted.
template <int K, bool ORDER, typename Decide>
__device__ __forceinline__ bool dp_exchange(const double (&mine)[K], int set, unsigned long long epoch,
                                            const DpGroup& P, double* s_red, int* s_ok, Decide&& decide) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double v = warp_sum(mine[k]);
        if (lane == 0) s_red[k * 32 + warp] = v;
    }
    __syncthreads();
    if (warp == 0) {
        double sum[K];
#pragma unroll
        for (int k = 0; k < K; ++k) sum[k] = warp_sum(lane < warps ? s_red[k * 32 + lane] : 0.0);
        const int G = P.count;
        DpSlot* words = P.words + static_cast<size_t>(set) * P.setStride;
        if (ORDER) fence_gpu();  // the block's stores, ordered before the barrier above, precede its words
        if (lane < kDpCopies && !(epoch == P.withholdEpoch && P.me == G - 1)) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                dp_store(words + k * P.valueStride + lane * G + P.me, sum[k], epoch);
        }
        const DpSlot* mineCopy = words + (P.me % kDpCopies) * G;
        constexpr int N = kDpMaxBlocks / 32;
        double got[K][N];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int j = 0; j < N; ++j) got[k][j] = 0.0;
        unsigned need = 0;  // bit k * N + j: word not seen yet
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (lane + 32 * j < G) need |= 1u << (k * N + j);
        bool ok = true;
        unsigned long long t0 = 0;
        unsigned spin = 0;
        while (true) {
            // every word's load in flight before the first is looked at
            double v[K][N];
            unsigned long long e[K][N];
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (32 * j < G) dp_load(mineCopy + k * P.valueStride + min(lane + 32 * j, G - 1), v[k][j], e[k][j]);
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (32 * j < G && e[k][j] == epoch && (need & (1u << (k * N + j)))) {
                        got[k][j] = v[k][j];
                        need &= ~(1u << (k * N + j));
                    }
            if (__all_sync(0xffffffffu, need == 0)) break;
            if ((++spin & 63u) == 0u) {
                if (t0 == 0) t0 = global_ns();
                const bool stop = *reinterpret_cast<volatile int*>(P.abortFlag) ||
                                  global_ns() - t0 > static_cast<unsigned long long>(P.waitNs);
                if (__any_sync(0xffffffffu, stop)) {
                    if (lane == 0) atomicExch(P.abortFlag, 1);
                    ok = false;
                    break;
                }
            }
        }
        if (ok && ORDER) fence_gpu();  // (acquiring loads instead would go one after another)
        double tot[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double t = 0.0;
#pragma unroll
            for (int j = 0; j < N; ++j) t += got[k][j];
            tot[k] = warp_sum(t);
        }
        if (lane == 0) {
            *s_ok = ok ? 1 : 0;
            if (ok) decide(tot);
        }
    }
    __syncthreads();
    return *s_ok != 0;
}

// z + beta p with the rounding of the solver's direction kernel: FP64 rounds the
// product and the sum (space.scale then space.add), FP32 is one FMA.
__device__ __forceinline__ double dp_direction(double z, double beta, double p) {
    return __dadd_rn(__dmul_rn(p, beta), z);
}
__device__ __forceinline__ float dp_direction(float z, float beta, float p) { return fmaf(beta, p, z); }

__device__ __forceinline__ double dp_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float dp_mul(float a, float b) { return a * b; }

// Ctl: Scalars, and three static functions run by one thread on the block's copy of
// the scalars: bool start(Scalars&, DpCommand&) (false: nothing to do),
// void afterProduct(Scalars&, DpCommand&, pq), void afterUpdate(Scalars&, DpCommand&, rr, rz).
template <typename V, int ND, bool SYM, bool RESIDENT, bool PRECOND, typename Ctl>
__device__ __forceinline__ void dp_solve(const DpArgs<V>& P, typename Ctl::Scalars* scalars) {
    extern __shared__ __align__(128) unsigned char dp_smem[];
    __shared__ typename Ctl::Scalars s_scalars;
    __shared__ DpCommand s_cmd;
    __shared__ double s_red[64];
    __shared__ int s_ok, s_run;
    const int T = blockDim.x, tid = threadIdx.x;
    const int n = P.A.nrows, R = P.R, nd = ND ? ND : P.A.ndiag;
    const int rb = min(blockIdx.x * R, n), nr = min(R, n - rb);
    if (tid == 0) {
        s_scalars = *scalars;
        s_run = *reinterpret_cast<volatile int*>(P.abortFlag) == 0 && Ctl::start(s_scalars, s_cmd) ? 1 : 0;
    }
    __syncthreads();
    if (!s_run) return;  // the same in every block: *scalars is written back after the last exchange only
    V* s_next = reinterpret_cast<V*>(dp_smem);
    auto take = [&](int count) {
        V* at = s_next;
        s_next += count;
        return at;
    };
    const int winStride = R + P.span;
    V* s_mat = RESIDENT ? take(nd * R) : nullptr;
    V* s_win = take(P.nwin * winStride);
    V* hq = P.homes & kDpQ ? take(R) : P.q + rb;
    V* hr = P.homes & kDpR ? take(R) : P.r + rb;
    V* hx = P.homes & kDpX ? take(R) : P.x + rb;
    V* sp = P.homes & kDpP ? take(R) : nullptr;
    V* sd = P.homes & kDpD ? take(R) : nullptr;
    for (int i = tid; i < nr; i += T) {
        if (P.homes & kDpR) hr[i] = P.r[rb + i];
        if (P.homes & kDpX) hx[i] = P.x[rb + i];
        if (PRECOND && sd) sd[i] = P.dinv[rb + i];
    }
    const V* hd = sd ? sd : P.dinv + rb;
    // diagonal d's entry for row r in the copy (column c = r + off[d])
    auto entry = [&](int d, int r) {
        const long at = SYM && d < nd / 2 ? static_cast<long>(nd - 1 - d) * P.A.ld + r + P.A.off[d]
                                          : static_cast<long>(d) * P.A.ld + r;
        return __ldg(P.A.val + at);
    };
    auto inside = [&](int c) { return static_cast<unsigned>(c) < static_cast<unsigned>(n); };
    if (RESIDENT)
        for (int d = 0; d < nd; ++d)
            for (int i = tid; i < nr; i += T)
                s_mat[d * R + i] = inside(rb + i + P.A.off[d]) ? entry(d, rb + i) : V(0);
    const bool edge = rb + P.minOff < 0 || rb + R - 1 + P.maxOff >= n;  // some operand lies outside the matrix
    __syncthreads();
    const DpGroup group{P.slots, 2 * kDpCopies * kDpMaxBlocks, kDpCopies * kDpMaxBlocks, static_cast<int>(gridDim.x),
                        static_cast<int>(blockIdx.x), P.abortFlag, P.waitNs, P.withholdEpoch};
    unsigned long long epoch = P.epoch0;
    bool aborted = false;
    while (true) {
        // ---- S ------------------------------------------------------------------
        const V* pprev = s_cmd.parity ? P.p0 : P.p1;
        V* pcur = s_cmd.parity ? P.p1 : P.p0;
        const V beta = static_cast<V>(s_cmd.beta);
        const bool first = s_cmd.first;
        // the windows: three windows' loads of two entries each in flight
        const int winLen = nr + P.span;
        for (int w0 = 0; w0 < P.nwin; w0 += 3)
            for (int x0 = tid; x0 < winLen; x0 += 2 * T) {
                V zv[2][3], pv[2][3];
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int w = 0; w < 3; ++w) {
                        const int x = x0 + u * T, c = rb + P.winLo[w0 + w] + x;
                        const bool in = x < winLen && w0 + w < P.nwin && inside(c);
                        zv[u][w] = in ? __ldcg(P.z + c) : V(0);
                        pv[u][w] = in && !first ? __ldcg(pprev + c) : V(0);
                    }
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int w = 0; w < 3; ++w) {
                        const int x = x0 + u * T;
                        if (x >= winLen || w0 + w >= P.nwin) continue;
                        const V p = first ? zv[u][w] : dp_direction(zv[u][w], beta, pv[u][w]);
                        s_win[(w0 + w) * winStride + x] = p;
                        const int i = x + P.winLo[w0 + w];
                        if (w0 + w == P.ownWin && i >= 0 && i < nr) {
                            pcur[rb + i] = p;
                            if (sp) sp[i] = p;
                        }
                    }
            }
        __syncthreads();
        const int ownAt = P.ownWin * winStride - P.winLo[P.ownWin];
        double pq = 0.0;
        auto rows = [&](auto atEdge) {
            constexpr bool EDGE = decltype(atEdge)::value;
            constexpr int B = RESIDENT ? 1 : (ND == 27 ? (sizeof(V) == 8 ? 14 : 27) : 9);  // entries in flight
            for (int i = tid; i < nr; i += T) {
                const V* operand = s_win + i;
                V sum = V(0);
                auto group = [&](int d0) {
                    V v[B];
#pragma unroll
                    for (int u = 0; u < B; ++u) {
                        const int d = d0 + u;
                        if (ND ? d >= ND : d >= nd) continue;
                        v[u] = RESIDENT ? s_mat[d * R + i]
                                        : (!EDGE || inside(rb + i + P.A.off[d]) ? entry(d, rb + i) : V(0));
                    }
#pragma unroll
                    for (int u = 0; u < B; ++u) {
                        const int d = d0 + u;
                        if (ND ? d < ND : d < nd) sum = fma(v[u], operand[P.wofs[d]], sum);
                    }
                };
                if constexpr (ND > 0) {
#pragma unroll
                    for (int d0 = 0; d0 < ND; d0 += B) group(d0);
                } else {
                    for (int d0 = 0; d0 < nd; d0 += B) group(d0);
                }
                hq[i] = sum;
                pq = fma(static_cast<double>(operand[ownAt]), static_cast<double>(sum), pq);
            }
        };
        if (!RESIDENT && edge) rows(std::true_type{});
        else rows(std::false_type{});
        {
            const double mine[1] = {pq};
            if (!dp_exchange<1, false>(mine, 0, ++epoch, group, s_red, &s_ok,
                                       [&](const double (&tot)[1]) { Ctl::afterProduct(s_scalars, s_cmd, tot[0]); })) {
                aborted = true;
                break;
            }
        }
        if (!s_cmd.go) break;
        // ---- U ------------------------------------------------------------------
        const V alpha = static_cast<V>(s_cmd.alpha);
        const bool step = s_cmd.step;
        const V* hp = sp ? sp : pcur + rb;
        double rr = 0.0, rz = 0.0;
        for (int i0 = tid; i0 < nr; i0 += kDpBatch * T) {
            V rv[kDpBatch], xv[kDpBatch], pv[kDpBatch], qv[kDpBatch], dv[kDpBatch];
#pragma unroll
            for (int u = 0; u < kDpBatch; ++u) {
                const int i = i0 + u * T;
                const bool in = i < nr;
                rv[u] = in ? hr[i] : V(0);
                dv[u] = PRECOND && in ? hd[i] : V(1);
                xv[u] = in && step ? hx[i] : V(0);
                pv[u] = in && step ? hp[i] : V(0);
                qv[u] = in && step ? hq[i] : V(0);
            }
#pragma unroll
            for (int u = 0; u < kDpBatch; ++u) {
                const int i = i0 + u * T;
                if (i >= nr) break;
                V ri = rv[u];
                if (step) {
                    hx[i] = fma(alpha, pv[u], xv[u]);
                    ri = fma(-alpha, qv[u], ri);
                    hr[i] = ri;
                }
                const V zi = PRECOND ? dp_mul(ri, dv[u]) : ri;
                P.z[rb + i] = zi;
                rr = fma(static_cast<double>(ri), static_cast<double>(ri), rr);
                if (PRECOND) rz = fma(static_cast<double>(ri), static_cast<double>(zi), rz);
            }
        }
        {
            const double mine[2] = {rr, rz};
            if (!dp_exchange<2, true>(mine, 1, ++epoch, group, s_red, &s_ok, [&](const double (&tot)[2]) {
                    Ctl::afterUpdate(s_scalars, s_cmd, tot[0], PRECOND ? tot[1] : tot[0]);
                })) {
                aborted = true;
                break;
            }
        }
        if (!s_cmd.go) break;
    }
    if (aborted) return;
    for (int i = tid; i < nr; i += T) {
        if (P.homes & kDpR) P.r[rb + i] = hr[i];
        if (P.homes & kDpX) P.x[rb + i] = hx[i];
    }
    if (blockIdx.x == 0 && tid == 0) *scalars = s_scalars;
}

// Shape of a launch.
struct DpPlan {
    int grid = 0, threads = 0;  // grid 0: no launch of this form fits
    size_t smem = 0;
    bool resident = false;
};

// Fills the shape fields of `a` (a.A set).  Blocks take at least 128 rows (fewer
// blocks make an exchange cheaper than the rows they would share out) and at most
// one block runs per SM.
template <typename V>
DpPlan dp_plan(DpArgs<V>& a, int sms, size_t optin) {
    DpPlan plan;
    const int n = a.A.nrows, nd = a.A.ndiag;
    const int blocks = std::max(1, std::min(std::min(sms, kDpMaxBlocks), (n + 127) / 128));
    a.R = ((n + blocks - 1) / blocks + 31) / 32 * 32;
    const size_t budget = (optin > 4096 ? optin - 4096 : 0) / sizeof(V);  // static shared memory beside it
    // Windows of the offsets (and of 0, the own rows): offsets closer than R share
    // one.  All windows are as long as the longest.
    std::vector<int> off(a.A.off, a.A.off + nd);
    if (std::find(off.begin(), off.end(), 0) == off.end()) off.push_back(0);
    std::sort(off.begin(), off.end());
    std::vector<int> lo{off[0]}, hi{off[0]};
    for (int o : off) {
        if (static_cast<long>(o) - hi.back() > a.R) {
            lo.push_back(o);
            hi.push_back(o);
        }
        hi.back() = o;
    }
    a.minOff = off.front();
    a.maxOff = off.back();
    a.nwin = static_cast<int>(lo.size());
    a.span = 0;
    for (int w = 0; w < a.nwin; ++w) a.span = std::max(a.span, hi[w] - lo[w]);
    const long winStride = static_cast<long>(a.R) + a.span;
    if (a.nwin * winStride > static_cast<long>(budget)) return plan;
    for (int w = 0; w < a.nwin; ++w) {
        a.winLo[w] = lo[w];
        if (lo[w] <= 0 && hi[w] >= 0) a.ownWin = w;
        for (int d = 0; d < nd; ++d)
            if (a.A.off[d] >= lo[w] && a.A.off[d] <= hi[w])
                a.wofs[d] = static_cast<int>(w * winStride) + a.A.off[d] - lo[w];
    }
    size_t used = static_cast<size_t>(a.nwin * winStride) + 3 * static_cast<size_t>(a.R);
    if (used > budget) return plan;
    a.homes = kDpQ | kDpR | kDpX;
    plan.resident = used + static_cast<size_t>(nd) * a.R <= budget;
    if (plan.resident) used += static_cast<size_t>(nd) * a.R;
    for (int home : {kDpP, kDpD})
        if (used + a.R <= budget) {
            used += a.R;
            a.homes |= home;
        }
    plan.threads = !plan.resident && a.R >= 768 ? 1024 : (a.R >= 384 ? 512 : 256);
    plan.grid = (n + a.R - 1) / a.R;
    plan.smem = std::max<size_t>(16, used * sizeof(V));
    return plan;
}

}  // namespace ciecu
