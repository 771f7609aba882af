// The FP32 smoother's row pass over a sliced copy of its matrix with 16-bit column
// offsets: a Chebyshev step or the cycle's residual, one launch each.
//
// A block owns a contiguous range of rows (about equal work per block) and sums them from
// a window of the operand in shared memory, copied in bulk: its rows and the bandwidth to
// either side.  Its rows are ordered by length and dealt to slices of 8; four lanes share a
// row, each with four entries (16 bytes of values, 8 of offsets) of the 16 of a step, so
// a warp reads 512 + 256 contiguous bytes a step.  The slices are dealt to the warps by
// length, longest first, to the warp with the least work, and lie in the order in which
// their warp reads them: a warp reads ONE contiguous stream, kSlSteps steps ahead, across
// the ends of its rows.  Padding has value 0 and offset 0.  A row's sum is kept in 16
// partial sums, so no chain is longer than a sixteenth of the row, and they are added in the
// order of the CSR kernel of 16 lanes a row: the same bits.
//
// What bounds it: a launch costs 7.5 us whatever the size (start, block, window, epilogue);
// the copy then comes from L2 at the 11 TB/s that all SMs draw together.  117,649 rows of
// Q3 elements (87 MB): 14.3 us a step back to back, 15 in the cycle, against 31.4 by the
// CSR kernel of 8 lanes a row (cycle's residual: 13 against 25).  Warps count, steps in
// flight hardly do: threads x steps 512 x 4, 512 x 8, 640 x 6, 768 x 4, 1024 x 3 measured
// 20.5, 20.5, 16.4, 14.3, 14.3 us.  The lanes of a row take neighbouring entries
// (entry 16 t + 4 c + lane for component c): mostly neighbouring columns, no bank twice.
#pragma once

#include "common.cuh"

#include <algorithm>
#include <vector>

namespace ciecu {

constexpr int kSlThreads = 768;
constexpr int kSlWarps = kSlThreads / 32;
constexpr int kSlSteps = 4;        // steps of a warp in flight
constexpr int kSlRows = 8;         // rows of a slice
constexpr int kSlEntries = 16;     // entries of a row in a step
constexpr int kSlBlockRows = 2048; // rows of a block at most
constexpr int kSlAhead = 2;        // rows of a thread whose vectors are read ahead

struct SlBlock {
    int rowBegin, rows, sliceBegin, slices;
    int warpSlice[kSlWarps + 1];  // slices of each warp, from sliceBegin
    int warpStep[kSlWarps + 1];   // first step of each warp
};

struct SlArgs {
    const float4* __restrict__ val;
    const short4* __restrict__ off;
    const SlBlock* __restrict__ blocks;
    const int* __restrict__ sliceEnd;  // one past the last step of a slice
    const short* __restrict__ row;     // kSlRows per slice: the row in the block, -1: none
    int n, lo, hi;                     // smallest and largest column offset
    int winLen;                        // window entries of any block
    int surplus;                       // test hook: bytes that block 0 waits for but nobody copies
};

struct SlPlan {
    SlArgs args{};
    int blocks = 0;
    size_t smem = 0;
    long steps = 0;
    void* memory = nullptr;
};

__device__ __forceinline__ void sl_use(float (&acc)[4], const float4& v, const short4& o, const float* win) {
    acc[0] = fmaf(v.x, win[o.x], acc[0]);
    acc[1] = fmaf(v.y, win[o.y], acc[1]);
    acc[2] = fmaf(v.z, win[o.z], acc[2]);
    acc[3] = fmaf(v.w, win[o.w], acc[3]);
}

// Whether the one phase of `bar` ended within about a second (it never takes that long).
__device__ __forceinline__ bool sl_arrived(unsigned bar) {
    unsigned arrived = 0;
    for (long long begun = clock64(); !arrived;) {
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(arrived)
            : "r"(bar)
            : "memory");
        if (!arrived && clock64() - begun > (1LL << 31)) break;
    }
    return arrived != 0;
}

// Op: Pre pre(row), post(row, pre, sum, operand of the row), expired() when the window's
// copy did not arrive.
template <typename Op>
__device__ __forceinline__ void sl_rows(const SlArgs& A, const float* __restrict__ x, const Op& op) {
    extern __shared__ __align__(16) unsigned char sl_smem[];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ SlBlock s_block;
    float* win = reinterpret_cast<float*>(sl_smem);
    float* sum = win + A.winLen;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < static_cast<int>(sizeof(SlBlock) / 4); i += kSlThreads)
        reinterpret_cast<int*>(&s_block)[i] = reinterpret_cast<const int*>(A.blocks + blockIdx.x)[i];
    const unsigned bar = static_cast<unsigned>(__cvta_generic_to_shared(&s_bar));
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int rb = s_block.rowBegin, nr = s_block.rows;
    const int first = max(rb + A.lo, 0) & ~3;                       // 16 bytes
    const int last = min(rb + nr + A.hi, A.n);                      // one past the window's last entry
    const int bytes = ((last - first) + 3) / 4 * 16;                // the vectors are padded to 16 bytes
    if (tid == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(bytes + (blockIdx.x == 0 ? A.surplus : 0))
                     : "memory");
        for (int done = 0; done < bytes; done += 16384)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             static_cast<unsigned>(__cvta_generic_to_shared(win)) + done),
                         "l"(reinterpret_cast<const char*>(x + first) + done), "r"(min(bytes - done, 16384)), "r"(bar)
                         : "memory");
    }
    typename Op::Pre pre[kSlAhead];
#pragma unroll
    for (int k = 0; k < kSlAhead; ++k)
        if (tid + k * kSlThreads < nr) pre[k] = op.pre(rb + tid + k * kSlThreads);
    int t = s_block.warpStep[warp];
    const int end = s_block.warpStep[warp + 1];
    float4 v[kSlSteps];
    short4 o[kSlSteps];
#pragma unroll
    for (int u = 0; u < kSlSteps; ++u)
        if (t + u < end) {
            v[u] = __ldg(A.val + (t + u) * 32L + lane);
            o[u] = __ldg(A.off + (t + u) * 32L + lane);
        }
    // the rows of the warp's slices and where they end, one slice ahead
    int slice = s_block.sliceBegin + s_block.warpSlice[warp];
    const int sliceLast = s_block.sliceBegin + s_block.warpSlice[warp + 1] - 1;
    int stop = 0, nextStop = 0, r = -1, nextRow = -1;
    if (t < end) {
        stop = A.sliceEnd[slice];
        r = A.row[slice * kSlRows + lane / 4];
        const int ahead = min(slice + 1, sliceLast);
        nextStop = A.sliceEnd[ahead];
        nextRow = A.row[ahead * kSlRows + lane / 4];
    }
    if (!__syncthreads_and(sl_arrived(bar))) {
        sl_arrived(bar);  // the copies may still be under way: the shared memory is kept for them
        if (tid == 0) op.expired();
        return;
    }
    const float* own = win + (rb - first);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const float* at = own + max(r, 0);
    for (; t < end; t += kSlSteps) {
#pragma unroll
        for (int u = 0; u < kSlSteps; ++u) {
            if (t + u < end) {
                sl_use(acc, v[u], o[u], at);
                if (t + u + kSlSteps < end) {
                    v[u] = __ldg(A.val + (t + u + kSlSteps) * 32L + lane);
                    o[u] = __ldg(A.off + (t + u + kSlSteps) * 32L + lane);
                }
                if (t + u + 1 == stop) {
                    float s = (acc[0] + acc[2]) + (acc[1] + acc[3]);
                    s += __shfl_xor_sync(0xffffffffu, s, 2);
                    s += __shfl_xor_sync(0xffffffffu, s, 1);
                    if ((lane & 3) == 0 && r >= 0) sum[r] = s;
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                    r = nextRow;
                    stop = nextStop;
                    at = own + max(r, 0);
                    ++slice;
                    const int ahead = min(slice + 1, sliceLast);
                    nextStop = A.sliceEnd[ahead];
                    nextRow = A.row[ahead * kSlRows + lane / 4];
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSlAhead; ++k) {
        const int i = tid + k * kSlThreads;
        if (i < nr) op.post(rb + i, pre[k], sum[i], own[i]);
    }
    for (int i = tid + kSlAhead * kSlThreads; i < nr; i += kSlThreads)
        op.post(rb + i, op.pre(rb + i), sum[i], own[i]);
}

// The copy's entries from the CSR matrix: a warp per slice.
__global__ void __launch_bounds__(256)
    sl_fill_kernel(SlArgs A, int nblocks, const int* __restrict__ rowptr, const short* __restrict__ off16,
                   const float* __restrict__ csr, float4* __restrict__ val, short4* __restrict__ off) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const SlBlock& B = A.blocks[b];
        for (int w = 0; w < kSlWarps; ++w)
            for (int s = B.warpSlice[w] + warp; s < B.warpSlice[w + 1]; s += warps) {
                const int slice = B.sliceBegin + s;
                const int begin = s == B.warpSlice[w] ? B.warpStep[w] : A.sliceEnd[slice - 1];
                const int r = A.row[slice * kSlRows + lane / 4];
                const int rowBegin = r < 0 ? 0 : rowptr[B.rowBegin + r], rowEnd = r < 0 ? 0 : rowptr[B.rowBegin + r + 1];
                for (int t = begin; t < A.sliceEnd[slice]; ++t) {
                    const int k = rowBegin + (t - begin) * kSlEntries + (lane & 3);
                    float v[4];
                    short o[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool in = k + 4 * j < rowEnd;
                        v[j] = in ? csr[k + 4 * j] : 0.f;
                        o[j] = in ? off16[k + 4 * j] : static_cast<short>(0);
                    }
                    val[t * 32L + lane] = make_float4(v[0], v[1], v[2], v[3]);
                    off[t * 32L + lane] = make_short4(o[0], o[1], o[2], o[3]);
                }
            }
    }
}

inline int sl_steps(int entries) { return std::max(1, (entries + kSlEntries - 1) / kSlEntries); }

// Blocks, slices and the warps' shares for rows of the given extents.  False where the
// copy does not pay: more than a quarter of it padding (rows of 9 entries: the CSR kernels
// read less), or a window that no block's shared memory holds.
inline bool sl_layout(int n, const int* rowptr, int lo, int hi, int sms, size_t maxSmem, std::vector<SlBlock>& blocks,
                      std::vector<int>& sliceEnd, std::vector<short>& row, int& winLen, size_t& smem, long& steps) {
    long work = 0;
    for (int i = 0; i < n; ++i) work += sl_steps(rowptr[i + 1] - rowptr[i]);
    // blocks in whole waves of the device, of 3/4 of the most rows on average
    const long wave = static_cast<long>(sms) * (kSlBlockRows * 3 / 4), waves = (n + wave - 1) / wave;
    const long parts = std::min<long>(sms * waves, (n + 4 * kSlRows - 1) / (4 * kSlRows));  // 4 slices at least
    const long span = static_cast<long>(hi) - lo;
    blocks.clear();
    sliceEnd.clear();
    row.clear();
    steps = 0;
    long longest = 0, done = 0;
    // a block's rows: their steps, the first place of each number of steps, the rows longest
    // first; the warp of each slice, the slices by warp
    std::vector<int> length, lengthBegin;
    std::vector<short> order, warpOf, mine;
    row.reserve(static_cast<size_t>(n) + static_cast<size_t>(n) / 8 + 8);
    sliceEnd.reserve(static_cast<size_t>(n) / kSlRows + static_cast<size_t>(n) / 64 + 8);
    for (int begin = 0, part = 0; begin < n; ++part) {
        const long until = std::max<long>(done + 1, work * (part + 1) / parts);
        int end = begin, most = 0;
        length.clear();
        while (end < n && end - begin < kSlBlockRows && (done < until || end - begin < kSlRows)) {
            const int k = sl_steps(rowptr[end + 1] - rowptr[end]);
            length.push_back(k);
            most = std::max(most, k);
            done += k;
            ++end;
        }
        const int rows = end - begin, count = (rows + kSlRows - 1) / kSlRows;
        lengthBegin.assign(static_cast<size_t>(most) + 2, 0);
        for (int k : length) ++lengthBegin[static_cast<size_t>(k)];
        for (int k = most, at = 0; k >= 0; --k) {
            const int here = lengthBegin[static_cast<size_t>(k)];
            lengthBegin[static_cast<size_t>(k)] = at;
            at += here;
        }
        order.resize(static_cast<size_t>(rows));
        for (int i = 0; i < rows; ++i)
            order[static_cast<size_t>(lengthBegin[static_cast<size_t>(length[static_cast<size_t>(i)])]++)] =
                static_cast<short>(i);
        // slices of 8 rows, longest first, each to the warp with the least work
        auto stepsOf = [&](int s) { return length[static_cast<size_t>(order[static_cast<size_t>(s) * kSlRows])]; };
        long load[kSlWarps] = {};
        int warpBegin[kSlWarps + 1] = {};
        warpOf.resize(static_cast<size_t>(count));
        mine.resize(static_cast<size_t>(count));
        for (int s = 0; s < count; ++s) {
            int w = 0;
            for (int k = 1; k < kSlWarps; ++k) w = load[k] < load[w] ? k : w;
            warpOf[static_cast<size_t>(s)] = static_cast<short>(w);
            load[w] += stepsOf(s);
            ++warpBegin[w + 1];
        }
        for (int w = 0; w < kSlWarps; ++w) warpBegin[w + 1] += warpBegin[w];
        for (int s = 0, next[kSlWarps] = {}; s < count; ++s) {
            const int w = warpOf[static_cast<size_t>(s)];
            mine[static_cast<size_t>(warpBegin[w] + next[w]++)] = static_cast<short>(s);
        }
        SlBlock B{};
        B.rowBegin = begin;
        B.rows = rows;
        B.sliceBegin = static_cast<int>(sliceEnd.size());
        B.slices = count;
        for (int w = 0; w < kSlWarps; ++w) {
            B.warpSlice[w] = static_cast<int>(sliceEnd.size()) - B.sliceBegin;
            B.warpStep[w] = static_cast<int>(steps);
            for (int k = warpBegin[w]; k < warpBegin[w + 1]; ++k) {
                const int s = mine[static_cast<size_t>(k)];
                steps += stepsOf(s);
                sliceEnd.push_back(static_cast<int>(steps));
                for (int i = s * kSlRows; i < (s + 1) * kSlRows; ++i)
                    row.push_back(i < rows ? order[static_cast<size_t>(i)] : static_cast<short>(-1));
            }
        }
        B.warpSlice[kSlWarps] = B.slices;
        B.warpStep[kSlWarps] = static_cast<int>(steps);
        blocks.push_back(B);
        longest = std::max<long>(longest, B.rows);
        begin = end;
    }
    const long window = (longest + span + 1 + 7) / 4 * 4;  // the start is rounded down, the end up
    smem = sizeof(float) * static_cast<size_t>(window + longest);
    winLen = static_cast<int>(window);
    return smem <= maxSmem && steps * 32 * 4 <= rowptr[n] + rowptr[n] / 4 && steps < (1L << 31) / 32;
}

}  // namespace ciecu
