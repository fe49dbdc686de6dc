// The hot part of a sweep: gathers of the most-used sources from shared memory.
//
// The gathers of a sweep are bound by L1 misses: one L1-to-L2 request per clock
// and SM (0.98 random 8-byte gathers per clock and SM measured on arrays of 2
// to 59 MB), whatever else the kernel does. Random gathers from shared memory
// run at 4.6 per clock and SM (4-byte: 7), and from arrays that L1 holds at
// 2.6. On power-law graphs a few leading ids (rows are numbered by in-degree,
// descending) are the sources of most arcs: on directed R-MAT 24 the first
// 24,576 ids of 32%, the first eight times as many of 64%. So the arcs of the
// longer rows are grouped by blocks of kHotIds sources, and this kernel, run
// before the regular sweep, sums every row's arcs in every block ("segments"):
// each CTA takes a contiguous, equal share of the segments in block order,
// copies the one or two blocks it needs into shared memory (192 KB of FP64
// values) and gathers there. The segment sums go to chunk slots of their rows,
// which the regular sweep (rows of at most kChunk arcs) or the fix-up (longer
// rows) adds to the sum of the row's other arcs.
//
// Layout: SELL-32 slices of segments of one block, longest first, as 16-bit
// numbers local to the block, eight arcs of a lane in 16 bytes (512-byte
// steps); absent arcs name the entry after the block, which holds `pad`.
//
// Measured (segment sums and regular sweep together, against one sweep of all
// arcs): R-MAT 24 0.604 against 0.865 ms in FP64, 0.525 against 0.765 in FP32;
// R-MAT 22 0.184 against 0.224 and 0.162 against 0.198. The kernel itself is
// bound by shared-memory wavefronts (85% of peak while an SM is busy; 5.7 per
// 32 random FP64 gathers) and by the copy and the last slices of a block.
#pragma once

#include "common.cuh"

namespace nkg {

// Sources per block: 192 KB of FP64 values, 96 KB of FP32 ones (28,672, the next
// multiple of 4,096, would still fit in FP64).
constexpr uint32_t kHotIds = 24576;
constexpr uint32_t kMaxBlocks = 31;
// A block is worth while where at least this many arcs, and this share of all,
// gather from it (every CTA that works on it copies its values and waits for
// its slowest warp, about 20,000 clocks); a segment from this many arcs: it
// costs a store, an index and a load, and is padded to eight arcs. Runs with
// segments from 4 / 6 arcs, R-MAT 24: 64.7 / 65.7 ms; with blocks of 1/256,
// 1/128 and 1/64 of the arcs, R-MAT 23: 32.8 / 33.6 / 36.6 ms.
constexpr uint32_t kBlockMinArcs = 256u << 10;
constexpr uint32_t kBlockShare = 256;
constexpr uint32_t kMinSegment = 4;
// Most arcs per chunk of a segment: the serial loop of a lane (R-MAT 23 with
// 64 / 128 / 256: 33.9 / 33.6 / 34.3 ms).
constexpr uint32_t kHotChunk = 128;
// Rows of at most this many arcs have no segments.
constexpr uint32_t kHotRow = 32;
// Graphs below have no blocks: building them takes 1.2 ms at 60M arcs, which
// the first run should win back. R-MAT, runs without / with blocks: 3.8M nodes
// (58.5M arcs, 76 iterations) 16.2 / 15.6 ms, 4.2M nodes (65.2M arcs, 103
// iterations) 23.4 / 20.1 ms, 8.4M nodes (131M arcs) 44.7 / 32.8 ms.
constexpr uint64_t kHotGraphArcs = 60ull << 20;
// Rows longer than this are partitioned by a whole CTA.
constexpr uint32_t kBigRow = 2048;

struct BlockPlan {
    uint32_t blocks;               // source blocks in use (0: none)
    uint32_t min_len[kMaxBlocks];  // least row length for block b (ascending)
    // Blocks a row of `len` arcs takes part in.
    __host__ __device__ uint32_t blocks_of(uint32_t len) const {
        uint32_t lo = 0, hi = blocks;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (min_len[mid] <= len)
                lo = mid + 1;
            else
                hi = mid;
        }
        return lo;
    }
};

// Slices of every block: block b's are [first[b], first[b + 1]).
struct HotBlocks {
    uint32_t first[kMaxBlocks + 1];
};

constexpr int kHotKernelThreads = 1024;

template <typename T>
constexpr size_t hot_bytes() {
    return (kHotIds + 16 / sizeof(T)) * sizeof(T);
}

template <typename T>
struct HotArgs {
    const uint4 *__restrict__ arcs;
    const uint32_t *__restrict__ off;        // first step of every slice (+1)
    const uint32_t *__restrict__ slot;       // 32 per slice: where the sum goes (kNone: nowhere)
    const uint32_t *__restrict__ cta_start;  // grid + 1 slices
    const T *__restrict__ y;                 // gathered values (n entries)
    T *__restrict__ sums;                    // chunk sums
    const int *skip;                         // nothing to do when set (a run that is over)
    HotBlocks blocks;
    uint32_t n;
    T pad;                                   // value of absent arcs
    T alpha;                                 // MODE 1: terms alpha * (1 + y)
};

template <typename T, int MODE>
__device__ __forceinline__ T hot_term(const T *s, uint32_t i, T alpha) {
    const T v = s[i];
    return MODE == 0 ? v : alpha * (T(1) + v);
}

template <typename T, int MODE>
__device__ __forceinline__ T hot_step(const T *s, uint4 w, T alpha) {
    const T a0 = hot_term<T, MODE>(s, w.x & 0xffffu, alpha), a1 = hot_term<T, MODE>(s, w.x >> 16, alpha);
    const T a2 = hot_term<T, MODE>(s, w.y & 0xffffu, alpha), a3 = hot_term<T, MODE>(s, w.y >> 16, alpha);
    const T a4 = hot_term<T, MODE>(s, w.z & 0xffffu, alpha), a5 = hot_term<T, MODE>(s, w.z >> 16, alpha);
    const T a6 = hot_term<T, MODE>(s, w.w & 0xffffu, alpha), a7 = hot_term<T, MODE>(s, w.w >> 16, alpha);
    return ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
}

__device__ __forceinline__ uint4 ld_stream_v4(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p), "l"(l2_evict_first_policy()));
    return v;
}

// A slice's steps and where this lane's sum goes.
struct HotSlice {
    uint32_t first, end, slot;
};
// Steps of the next slice loaded ahead: the registers
// of 1,024 threads (64 each) hold three beside FP32 sums, one beside FP64's
// address arithmetic. R-MAT 24: FP64 one 0.616 ms a sweep, two 0.621; FP32
// three 0.540, two 0.544.
template <typename T>
constexpr uint32_t kHotAhead = sizeof(T) == 8 ? 1 : 3;

template <typename T>
__device__ __forceinline__ HotSlice hot_slice(const HotArgs<T> &a, uint32_t s, uint32_t hi,
                                              uint32_t lane) {
    HotSlice h{0, 0, kNone};
    if (s < hi) {
        h.first = __ldg(a.off + s);
        h.end = __ldg(a.off + s + 1);
        h.slot = ld_stream(a.slot + s * 32 + lane);
    }
    return h;
}

template <typename T>
__device__ __forceinline__ void hot_head(const HotArgs<T> &a, const HotSlice &h, uint32_t lane,
                                         uint4 (&w)[kHotAhead<T>]) {
#pragma unroll
    for (uint32_t q = 0; q < kHotAhead<T>; ++q)
        if (h.first + q < h.end)
            w[q] = ld_stream_v4(a.arcs + static_cast<size_t>(h.first + q) * 32 + lane);
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kHotKernelThreads, 1) hot_kernel(HotArgs<T> a) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    T *s_y = reinterpret_cast<T *>(s_dyn);
    if (a.skip && *(volatile const int *)a.skip)
        return;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr uint32_t kWarps = kHotKernelThreads / 32;
    constexpr uint32_t kVec = 16 / sizeof(T);
    const uint32_t begin = a.cta_start[blockIdx.x], end = a.cta_start[blockIdx.x + 1];
    for (uint32_t b = 0; b < kMaxBlocks; ++b) {
        const uint32_t lo = max(begin, a.blocks.first[b]), hi = min(end, a.blocks.first[b + 1]);
        if (lo >= hi)
            continue;
        __syncthreads();  // the block before is done with
        const uint32_t base = b * kHotIds, cnt = min(kHotIds, a.n - base);
        // Every CTA starts at a place of its own: many copy the same block at
        // once, and in step they would all ask the same few L2 slices.
        const uint4 *src = reinterpret_cast<const uint4 *>(a.y + base);
        uint4 *dst = reinterpret_cast<uint4 *>(s_y);
        const uint32_t vecs = cnt / kVec;
        const uint32_t turn = static_cast<uint32_t>(static_cast<uint64_t>(vecs) * blockIdx.x / gridDim.x);
#pragma unroll 6
        for (uint32_t i = threadIdx.x; i < vecs; i += kHotKernelThreads) {
            const uint32_t k = i + turn < vecs ? i + turn : i + turn - vecs;
            dst[k] = __ldg(src + k);
        }
        if (threadIdx.x < cnt % kVec)
            s_y[cnt / kVec * kVec + threadIdx.x] = __ldg(a.y + base + cnt / kVec * kVec + threadIdx.x);
        if (threadIdx.x == 0)
            s_y[kHotIds] = a.pad;
        __syncthreads();
        // Most slices are one to four steps: the next slice's first steps and
        // the bounds of the one after it are loaded before this one is summed.
        uint32_t s = lo + wid;
        HotSlice cur = hot_slice(a, s, hi, lane), nxt = hot_slice(a, s + kWarps, hi, lane);
        constexpr uint32_t kAhead = kHotAhead<T>, kBatch = kAhead > 2 ? kAhead : 2;
        uint4 w[kAhead];
        hot_head(a, cur, lane, w);
        for (; s < hi; s += kWarps) {
            uint4 wn[kAhead];
            hot_head(a, nxt, lane, wn);
            const HotSlice nn = hot_slice(a, s + 2 * kWarps, hi, lane);
            const uint4 *p = a.arcs + static_cast<size_t>(cur.first) * 32 + lane;
            const uint32_t steps = cur.end - cur.first;
            T acc = T(0);
#pragma unroll
            for (uint32_t q = 0; q < kAhead; ++q)
                if (q < steps)
                    acc += hot_step<T, MODE>(s_y, w[q], a.alpha);
            for (uint32_t i = kAhead; i < steps; i += kBatch) {
                uint4 x[kBatch];
#pragma unroll
                for (uint32_t q = 0; q < kBatch; ++q)
                    if (i + q < steps)
                        x[q] = ld_stream_v4(p + static_cast<size_t>(i + q) * 32);
#pragma unroll
                for (uint32_t q = 0; q < kBatch; ++q)
                    if (i + q < steps)
                        acc += hot_step<T, MODE>(s_y, x[q], a.alpha);
            }
            if (cur.slot != kNone)
                a.sums[cur.slot] = acc;
            cur = nxt;
            nxt = nn;
#pragma unroll
            for (uint32_t q = 0; q < kAhead; ++q)
                w[q] = wn[q];
        }
    }
}

} // namespace nkg
