// Copy and plan of the single-launch solves over sliced rows (sell_persistent.cuh).
#include "sell_persistent.cuh"
#include "sortscan.cuh"
#include "space.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <iterator>
#include <set>
#include <utility>

namespace ciecu {
namespace {

constexpr int kT = 256;

// Deals the rows of each run of kSpSort rows (one block of kSpSort threads; `runRow`
// the run's first row, `runEnd` its system's end) to its slices by descending length,
// equal lengths in row order; the steps of the slices and the smallest and largest
// column offset of the run's system.  Rows of more than `longest` entries are in no slice.
__global__ void __launch_bounds__(kSpSort) sp_shape_kernel(const int* __restrict__ runRow,
                                                           const int* __restrict__ runEnd,
                                                           const int* __restrict__ runSystem,
                                                           const int* __restrict__ rowptr, const int* __restrict__ col,
                                                           int longest, int* __restrict__ row, int* __restrict__ steps,
                                                           int* __restrict__ lo, int* __restrict__ hi) {
    __shared__ int s_len[kSpSort];
    constexpr int kSlices = kSpSort / 32;
    const int i = threadIdx.x, r = runRow[blockIdx.x] + i;
    const bool live = r < runEnd[blockIdx.x];
    int len = -1, mn = INT_MAX, mx = INT_MIN;
    if (live) {
        const int k0 = rowptr[r], k1 = rowptr[r + 1];
        len = k1 - k0;
        for (int k = k0; k < k1; ++k) {
            mn = min(mn, col[k] - r);
            mx = max(mx, col[k] - r);
        }
    }
    const bool sliced = live && len <= longest;
    if (!sliced) len = -1;
    s_len[i] = len;
    __syncthreads();
    int place = 0;
    for (int j = 0; j < kSpSort; ++j) place += s_len[j] > len || (s_len[j] == len && j < i) ? 1 : 0;
    const long slice = static_cast<long>(blockIdx.x) * kSlices + place / 32;
    row[slice * 32 + place % 32] = sliced ? r : -1;
    if (place % 32 == 0) steps[slice] = (max(len, 0) + 1) / 2;  // the slice's longest row
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((i & 31) == 0 && mn <= mx) {
        atomicMin(lo + runSystem[blockIdx.x], mn);
        atomicMax(hi + runSystem[blockIdx.x], mx);
    }
}

// Values (or, when `off` is given, the operands' places against the rows' own) of every
// slice; padding zero.  origin: first column of the window of the slice's system for its
// first row (parts start at even rows of the system, so places differ by the same for
// every part).
__global__ void sp_fill_kernel(long slices, const int* __restrict__ row, const int* __restrict__ sliceStep,
                               const int* __restrict__ rowptr, const int* __restrict__ col,
                               const double* __restrict__ val, double2* __restrict__ out, short2* __restrict__ off,
                               const int* __restrict__ origin, int half) {
    const int lane = threadIdx.x & 31;
    const long warps = static_cast<long>(gridDim.x) * (kT / 32);
    for (long s = static_cast<long>(blockIdx.x) * (kT / 32) + (threadIdx.x >> 5); s < slices; s += warps) {
        const int r = row[s * 32 + lane];
        const int k0 = r >= 0 ? rowptr[r] : 0, len = r >= 0 ? rowptr[r + 1] - k0 : 0;
        const int t0 = sliceStep[s], t1 = sliceStep[s + 1];
#pragma unroll 4
        for (int t = t0; t < t1; ++t) {
            const int j = 2 * (t - t0);
            if (off) {
                const int o0 = origin[s], own = sp_place(r - o0, half);
                short2 o;
                o.x = j < len ? static_cast<short>(sp_place(col[k0 + j] - o0, half) - own) : short(0);
                o.y = j + 1 < len ? static_cast<short>(sp_place(col[k0 + j + 1] - o0, half) - own) : short(0);
                off[static_cast<long>(t) * 32 + lane] = o;
            } else {
                double2 v;
                v.x = j < len ? __ldg(val + k0 + j) : 0.0;
                v.y = j + 1 < len ? __ldg(val + k0 + j + 1) : 0.0;
                out[static_cast<long>(t) * 32 + lane] = v;
            }
        }
    }
}

}  // namespace

void sp_destroy(SpPlan& p) {
    pool_release({p.val, p.off, p.sliceStep, p.row, p.longRow, p.items, p.itemBegin, p.slots});
    p = SpPlan{};
}

int sp_fill(const SpPlan& p, const ciecu_csr_s* csr, cudaStream_t st) {
    sp_fill_kernel<<<grid_for(p.slices * 32, kT, 8), kT, 0, st>>>(p.slices, p.row, p.sliceStep, csr->rowptr, csr->col,
                                                                  static_cast<const double*>(csr->val),
                                                                  reinterpret_cast<double2*>(p.val), nullptr, nullptr, 0);
    count_launch();
    CIECU_CHECK_LAUNCH("sp_fill_kernel");
    return CIECU_OK;
}

int sp_build(SpPlan& p, const ciecu_csr_s* csr, const std::vector<long long>& rowOffsets, const SpLimits& limits,
             cudaStream_t st) {
    if (p.state != 0) return CIECU_OK;
    p.state = 2;
    const int systems = static_cast<int>(rowOffsets.size()) - 1;
    const long n = systems > 0 ? static_cast<long>(rowOffsets.back()) : 0;
    if (systems < 1 || n < 1 || csr->nnz < 1) return CIECU_OK;
    int device = 0, optin = 0;
    CIECU_CUDA(cudaGetDevice(&device));
    CIECU_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    const int sms = std::min(sm_count(), kDpMaxBlocks);
    auto tooMany = [&](long parts) {
        return limits.rounds && !limits.rounds(static_cast<double>(parts) / sms, static_cast<double>(csr->nnz) / parts);
    };
    if (tooMany(systems)) return CIECU_OK;  // each has a part at least
    const long budget = (optin > 4096 ? optin - 4096 : 0) / static_cast<long>(sizeof(double));
    // runs of kSpSort rows, none across two systems
    std::vector<int> runRow, runEnd, runSystem, sliceBase(static_cast<size_t>(systems));
    for (int s = 0; s < systems; ++s) {
        sliceBase[s] = static_cast<int>(runRow.size()) * (kSpSort / 32);
        for (long long r = rowOffsets[s]; r < rowOffsets[s + 1]; r += kSpSort) {
            runRow.push_back(static_cast<int>(r));
            runEnd.push_back(static_cast<int>(rowOffsets[s + 1]));
            runSystem.push_back(s);
        }
    }
    const long runs = static_cast<long>(runRow.size()), slices = runs * (kSpSort / 32);
    if (slices == 0) return CIECU_OK;
    const bool few = csr->longRows <= kFewLongRows;  // those rows are in no slice
    int *d_scratch = nullptr, *d_steps = nullptr;
    auto bytes = [](long k) { return sizeof(int) * static_cast<size_t>(std::max<long>(k, 1)); };
    cudaError_t e = pool_alloc(&p.row, bytes(slices * 32), st);
    if (e == cudaSuccess) e = pool_alloc(&p.sliceStep, bytes(slices + 1), st);
    if (e == cudaSuccess) e = pool_alloc(&d_scratch, bytes(3 * runs + 2L * systems + scan_work(slices)), st);
    if (e == cudaSuccess) e = pool_alloc(&d_steps, bytes(slices), st);
    int* d_row = d_scratch;
    int* d_end = d_row + runs;
    int* d_system = d_end + runs;
    int* d_lo = d_system + runs;
    int* d_hi = d_lo + systems;
    int* d_scan = d_hi + systems;
    std::vector<int> lo(static_cast<size_t>(systems), INT_MAX), hi(static_cast<size_t>(systems), INT_MIN);
    auto up = [&](int* d, const std::vector<int>& h) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(d, h.data(), sizeof(int) * h.size(), cudaMemcpyHostToDevice, st);
    };
    up(d_row, runRow);
    up(d_end, runEnd);
    up(d_system, runSystem);
    up(d_lo, lo);
    up(d_hi, hi);
    int status = CIECU_OK, steps = 0;
    if (e == cudaSuccess) {
        sp_shape_kernel<<<static_cast<unsigned>(runs), kSpSort, 0, st>>>(d_row, d_end, d_system, csr->rowptr, csr->col,
                                                                        few ? kLongRow : INT_MAX, p.row, d_steps, d_lo,
                                                                        d_hi);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) status = exclusive_scan(d_steps, p.sliceStep, slices, d_scan, st);
    auto down = [&](void* h, const int* d, size_t count) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(int) * count, cudaMemcpyDeviceToHost, st);
    };
    if (e == cudaSuccess && status == CIECU_OK) {
        down(&steps, p.sliceStep + slices, 1);
        down(lo.data(), d_lo, lo.size());
        down(hi.data(), d_hi, hi.size());
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (d_scratch) cudaFreeAsync(d_scratch, st);
    if (d_steps) cudaFreeAsync(d_steps, st);
    auto unsuitable = [&]() {
        sp_destroy(p);
        p.state = 2;
        return CIECU_OK;
    };
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();  // no room: the caller keeps its other loop
        return unsuitable();
    }
    if (e != cudaSuccess || status != CIECU_OK) {
        sp_destroy(p);
        p.state = 0;
        return status != CIECU_OK ? status : cuda_fail(e, "sliced copy: shape");
    }
    if (64.0 * steps > 1.6 * static_cast<double>(csr->nnz) + 65536.0) return unsuitable();
    if (!few && 64.0 * steps > limits.padding * static_cast<double>(csr->nnz)) return unsuitable();
    int span = 0;
    for (int s = 0; s < systems; ++s) {
        lo[s] = std::min(lo[s], 0);
        hi[s] = std::max(hi[s], 0);
        if (rowOffsets[s + 1] == rowOffsets[s]) lo[s] = hi[s] = 0;
        if (static_cast<long>(hi[s]) - lo[s] > budget) return unsuitable();
        span = std::max(span, hi[s] - lo[s]);
    }
    // Rows of a block: all blocks busy with one part each where that is possible,
    // and at most mostRows or what shared memory holds beside the widest window.
    const long most = std::min<long>(limits.rows, (budget - span - 8) * 2 / 7) / kSpSort * kSpSort;
    if (most < kSpSort) return unsuitable();
    long R = std::min(most, ((n + sms - 1) / sms + kSpSort - 1) / kSpSort * kSpSort);
    auto parts = [&](long rowsEach) {
        long c = 0;
        for (int s = 0; s < systems; ++s) c += (rowOffsets[s + 1] - rowOffsets[s] + rowsEach - 1) / rowsEach;
        return c;
    };
    while (R + kSpSort <= most && (systems > sms || parts(R) > sms)) R += kSpSort;
    long largest = 0;
    for (int s = 0; s < systems; ++s) largest = std::max<long>(largest, rowOffsets[s + 1] - rowOffsets[s]);
    if ((largest + R - 1) / R > sms) return unsuitable();  // a system needs more blocks than are resident
    const long allParts = parts(R);
    if (tooMany(allParts)) return unsuitable();
    if (R + span > limits.window && csr->nnz < limits.entriesPerColumn * (R + span)) return unsuitable();
    // Systems in descending size to the blocks that are free first; a block's time is
    // measured in iterations, which grow with the square root of a 2D system's rows.
    std::vector<int> order(static_cast<size_t>(systems));
    for (int s = 0; s < systems; ++s) order[s] = s;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return rowOffsets[a + 1] - rowOffsets[a] > rowOffsets[b + 1] - rowOffsets[b];
    });
    const int G = static_cast<int>(std::min<long>(sms, std::max<long>(1, allParts)));
    std::vector<std::vector<SpItem>> lists(static_cast<size_t>(G));
    // the blocks by the time they are free, equal ones in order
    std::set<std::pair<double, int>> blocks;
    for (int b = 0; b < G; ++b) blocks.emplace(0.0, b);
    std::vector<std::pair<double, int>> taken;
    const std::vector<int> longRows(csr->longRow, csr->longRow + (few ? csr->longRows : 0));
    int slots = 0, rowsMost = kSpSort;
    for (int s : order) {
        const long ns = rowOffsets[s + 1] - rowOffsets[s];
        if (ns == 0) continue;
        const int c = static_cast<int>((ns + R - 1) / R);
        const int each = static_cast<int>(((ns + c - 1) / c + kSpSort - 1) / kSpSort * kSpSort);
        const int used = static_cast<int>((ns + each - 1) / each);
        taken.assign(blocks.begin(), std::next(blocks.begin(), used));
        blocks.erase(blocks.begin(), std::next(blocks.begin(), used));
        const double start = taken.back().first;
        for (int k = 0; k < used; ++k) {
            const int b = taken[k].second;
            const long begin = rowOffsets[s] + static_cast<long>(k) * each;
            SpItem I{};
            I.system = s;
            I.part = k;
            I.parts = used;
            I.rowBegin = static_cast<int>(begin);
            I.rows = static_cast<int>(std::min<long>(each, rowOffsets[s + 1] - begin));
            I.sliceBegin = sliceBase[s] + k * (each / 32);
            I.sysBegin = static_cast<int>(rowOffsets[s]);
            I.sysEnd = static_cast<int>(rowOffsets[s + 1]);
            I.lo = lo[s];
            I.span = hi[s] - lo[s];
            I.slotBase = slots;
            const auto first = std::lower_bound(longRows.begin(), longRows.end(), I.rowBegin);
            I.longBegin = static_cast<int>(first - longRows.begin());
            I.longRows = static_cast<int>(std::lower_bound(first, longRows.end(), I.rowBegin + I.rows) - first);
            lists[b].push_back(I);
            rowsMost = std::max(rowsMost, each);
            blocks.emplace(start + std::sqrt(static_cast<double>(ns)) * (1000.0 + each), b);
        }
        slots += used;
    }
    std::vector<SpItem> items;
    std::vector<int> begin(1, 0);
    for (const auto& l : lists) {
        p.longestList = std::max(p.longestList, static_cast<long>(l.size()));
        items.insert(items.end(), l.begin(), l.end());
        begin.push_back(static_cast<int>(items.size()));
    }
    p.slices = slices;
    p.steps = steps;
    p.grid = G;
    // as many warps as share a block's slices evenly
    const int blockSlices = rowsMost / 32, rounds = (blockSlices + kSpThreads / 32 - 1) / (kSpThreads / 32);
    p.threads = std::max(256, 32 * ((blockSlices + rounds - 1) / rounds));
    p.args.R = rowsMost;
    p.args.winLen = (rowsMost + span + 1) / 2 * 2;
    // the windows, q, r and x, and the schedule of the slices (s_step, s_row)
    long used = p.args.winLen + 3L * rowsMost + (4L * (rowsMost / 32 + 1) + 2L * rowsMost + 15) / 8;
    if (used > budget || p.args.winLen > 32767) return unsuitable();  // places are 16-bit
    p.args.homes = 0;
    for (int home : {kDpP, kDpD})
        if (used + rowsMost <= budget) {
            used += rowsMost;
            p.args.homes |= home;
        }
    p.smem = sizeof(double) * static_cast<size_t>(used);
    const size_t pairs = static_cast<size_t>(steps) * 32;
    const size_t slotBytes = sizeof(DpSlot) * kSpWords * static_cast<size_t>(std::max(slots, 1));
    e = pool_alloc(&p.val, sizeof(double2) * std::max<size_t>(pairs, 1), st);
    if (e == cudaSuccess) e = pool_alloc(&p.off, sizeof(short2) * std::max<size_t>(pairs, 1), st);
    if (e == cudaSuccess) e = pool_alloc(&p.longRow, bytes(static_cast<long>(longRows.size())), st);
    if (e == cudaSuccess) e = pool_alloc(&p.items, sizeof(SpItem) * std::max<size_t>(items.size(), 1), st);
    if (e == cudaSuccess) e = pool_alloc(&p.itemBegin, sizeof(int) * begin.size(), st);
    if (e == cudaSuccess) e = pool_alloc(&p.slots, slotBytes, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(p.slots, 0, slotBytes, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(p.items, items.data(), sizeof(SpItem) * items.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(p.itemBegin, begin.data(), sizeof(int) * begin.size(), cudaMemcpyHostToDevice, st);
    up(p.longRow, longRows);
    if (e != cudaSuccess) {
        cudaGetLastError();  // no room for the copy: the caller keeps its other loop
        return unsuitable();
    }
    std::vector<int> origin(static_cast<size_t>(slices));
    for (long k = 0; k < slices; ++k) {
        const int s = runSystem[k / (kSpSort / 32)];
        origin[k] = static_cast<int>(rowOffsets[s]) + lo[s];
    }
    int* d_origin = nullptr;
    e = pool_alloc(&d_origin, bytes(slices), st);
    up(d_origin, origin);
    if (e == cudaSuccess) {
        sp_fill_kernel<<<grid_for(slices * 32, kT, 8), kT, 0, st>>>(slices, p.row, p.sliceStep, csr->rowptr, csr->col,
                                                                    nullptr, nullptr, p.off, d_origin,
                                                                    p.args.winLen / 2);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // the host lists are in use until here
    if (d_origin) cudaFreeAsync(d_origin, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return unsuitable();
    }
    if (e != cudaSuccess) {
        sp_destroy(p);
        p.state = 0;
        return cuda_fail(e, "sliced copy: offsets");
    }
    p.longRows = !longRows.empty();
    p.args.A = SpMatrix{p.val, p.off, p.sliceStep, p.row, p.longRow, csr->rowptr, csr->col,
                        static_cast<const double*>(csr->val)};
    p.args.items = p.items;
    p.args.itemBegin = p.itemBegin;
    p.args.slots = p.slots;
    p.state = 1;
    return CIECU_OK;
}

}  // namespace ciecu
