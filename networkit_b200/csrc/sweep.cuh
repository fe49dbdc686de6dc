// One Jacobi sweep of PageRank (PageRank.cpp:56-70) as a sliced-ELLPACK pull
// SpMV over the in-adjacency, plus a fix-up kernel that finishes the rows that
// were split into chunks and closes the iteration (residual, sink mass,
// convergence test).
//
// Storage of the iterate: "gather form" y[r] = x[r] / deg[r] for nodes with
// out-arcs and y[r] = x[r] for sinks, so a sweep gathers exactly the per-arc
// term x[v]*w/deg[v] of PageRank.cpp:62 (bit-identical for unweighted graphs,
// where w = 1). The previous x[r] for the stopping test (PageRank.cpp:41-51)
// is recovered as y[r]*deg[r]. y has one extra zero entry at index n, the
// target of padding slots.
//
// Layout (SELL-C-sigma, Kreutzer et al., SIAM J. Sci. Comput. 36(5), 2014, with
// C = 32 and sigma = n): nodes are relabelled by in-degree, descending, so 32
// consecutive rows have nearly equal length. Rows longer than kChunk arcs are
// cut into chunks of kChunk arcs ("virtual rows", placed first; kSmallChunk in
// graphs of fewer arcs); of rows with source blocks (hot.cuh) only the arcs outside the blocks are here. Slice s holds
// 32 virtual rows column-major: slot (j, lane) at col_sell[(off[s] + j) * 32 +
// lane], so a warp loads 128 contiguous bytes per step and every lane sums its
// own row sequentially, in the caller's arc order. No shared memory and no
// barriers are needed: the whole L1 is left to cache the hot part of y.
// The slices are cut into contiguous, cost-balanced ranges ("units", fixed at
// set-up). Every warp runs one unit of its own first and then takes the next
// unit from a device counter (next_unit), so no warp is left with a share that
// ends late. Each unit's residual and sink partials go to a slot of its own, so
// every sum has a fixed order and a run is bit-reproducible.
#pragma once

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace nkg {

// Arcs per chunk of a split row, which is also the longest sequential loop of a
// lane (256 steps are 32 dependent batches). Graphs of less than 160 arcs for
// every resident lane (7,104 warps) get shorter chunks, so that no warp ends
// long after the others. Run times with chunks of 256 / 64 arcs, FP64: R-MAT
// 23 34.1 / 36.7 ms, 22 21.0 / 21.7, 21 13.1 / 12.4; Barabasi-Albert of 64M
// arcs 6.4 / 6.6.
constexpr uint32_t kChunk = 256;
constexpr uint32_t kSmallChunk = 64;
inline uint32_t resident_lanes(unsigned sms) { return sms * 48 * 32; }
inline uint32_t chunk_for(uint64_t arcs, unsigned sms) {
    return arcs >= 160ull * resident_lanes(sms) ? kChunk : kSmallChunk;
}
// A split row with more chunk sums than this is summed by a whole warp in the
// fix-up, the others by one thread. With source blocks (hot.cuh) a row has a
// dozen sums and four lanes (R-MAT 24, FP64 iteration with four / eight
// lanes: 0.636 / 0.641 ms); without, two or three: eight lanes a row took
// 19 us of an iteration on 58M arcs, a thread a row 12.5 (iteration 0.223 /
// 0.209 ms).
constexpr uint32_t kShortChunks = 16;
constexpr uint32_t kShortSums = 128;
__host__ __device__ inline uint32_t row_lanes(uint32_t n_hot) { return n_hot ? 4u : 1u; }

// Work units of the queued sweeps: warp gw of nw runs unit gw first, with no
// ticket, then units nw + t for the tickets t it takes from `queue`, while
// any are left. A grid that covers all units takes no tickets at all, so small
// graphs pay no atomics. Returns the warp's next unit (>= units: done).
__device__ __forceinline__ uint32_t next_unit(unsigned int *queue, uint32_t units, uint32_t nw,
                                              int lane) {
    if (nw >= units)
        return units;
    uint32_t t = 0;
    if (lane == 0)
        t = atomicAdd(queue, 1u);
    return nw + __shfl_sync(0xffffffffu, t, 0);
}

// Fix-up CTAs of a queued sweep: those its split rows need, and enough that
// no thread adds more than kUnitsPerFixThread of the sweep's unit partials.
constexpr uint32_t kUnitsPerFixThread = 4;
inline unsigned fix_ctas_with_units(unsigned split_ctas, uint64_t units, unsigned threads) {
    const uint64_t per_cta = static_cast<uint64_t>(threads) * kUnitsPerFixThread;
    return static_cast<unsigned>(std::max<uint64_t>(split_ctas, (units + per_cta - 1) / per_cta));
}

// Constant per run, read from device memory so that captured CUDA graphs
// stay valid across runs with different parameters.
struct RunParams {
    double damp;
    double tele_uniform;  // (1 - damp) / n  (PageRank.cpp:25)
    double one_minus_damp;
    double inv_n;
    int distribute;       // distributeSinks
    int personal;         // teleport vector present
    int l2;               // norm == L2
    int pad;
    double tol;
    unsigned long long max_iterations;
};

// Mutable per-run state, advanced by the last CTA of every fix-up launch.
struct IterState {
    unsigned long long iteration;  // completed sweeps
    double residual;               // norm of the last sweep
    double residual_sum;           // its sum before the square root (L2)
    double sink_mass;              // sum of x over sinks of the last iterate
    double sink_coef;              // sink term applied by the next sweep
    int done;                      // converged / max reached
    unsigned int ticket;           // last-block detection in the fix-up
    int error;
    unsigned int queue;            // next work unit of a queued sweep (reset by the fix-up)
};

template <typename T>
struct SweepArgs {
    const uint32_t *__restrict__ col_sell;   // slices, column-major, padded with n
    const T *__restrict__ w_sell;            // matching weights (weighted graphs)
    const uint32_t *__restrict__ slice_off;  // S+1, in units of 32 slots
    const uint32_t *__restrict__ unit_start; // U+1 slice indices
    const uint32_t *__restrict__ chunk_begin;// n_long+1: chunks of split row r
    const uint32_t *__restrict__ degc;       // out-degree count (sink test)
    const T *__restrict__ degw;              // weighted out-degree (weighted graphs)
    const T *__restrict__ tele;              // personalised teleport (n) or null
    const T *__restrict__ y_in;              // n+1 (y_in[n] = 0)
    T *__restrict__ y_out;
    T *__restrict__ chunk_val;               // per chunk slot: partial row sum
    // Rows [0, n_hot) have segment sums of hot.cuh among their chunk sums
    // (chunk_begin then has n_hot + 1 entries).
    const uint32_t *__restrict__ chunk_slot; // where stored chunk i's sum goes (null: i)
    uint32_t n_hot;
    double *__restrict__ cta_res;            // per sweep CTA
    double *__restrict__ cta_sink;
    double *__restrict__ fix_res;            // per fix-up CTA
    double *__restrict__ fix_sink;
    const RunParams *__restrict__ rp;
    IterState *st;
    uint32_t n;
    uint32_t n_long;        // rows [0, n_long) are split into chunks
    uint32_t n_vlong;       // rows [0, n_vlong) are summed by a warp each
    uint32_t s_chunk;       // slices [0, s_chunk) hold chunks, the rest rows
    uint32_t units;
    uint32_t sweep_ctas;
    uint32_t hot;           // ids [0, hot) are read from the shared-memory tier
    uint32_t trace_cap;     // entries of trace
    double *trace;          // residual of completed sweep i at [i] (i < trace_cap)
    // Row slice of a partitioned run (PART kernels): local row r (in the
    // slice's own relabelled order) is slice row row_map[r]; the slice's
    // iterate entries, degrees, teleport and output are in slice row order,
    // and its previous iterate value sits at y_in[row_base + row_map[r]] of
    // the shared iterate, whose entry `pad` is the zero of padding slots.
    const uint32_t *__restrict__ row_map;
    uint32_t row_base;
    uint32_t pad;
    // Queued sweep: warps take units from IterState::queue and store each
    // unit's residual and sink partial sums here (indexed by unit), so the
    // sums keep a fixed order whichever warp ran the unit. Null: the static
    // round-robin assignment with per-CTA partials in cta_res / cta_sink.
    double *unit_res;
    double *unit_sink;
    // The queued sweep's last CTA closes the iteration itself (graphs with no
    // split rows and few units; no fix-up launch): see close_iteration.
    int close_in_sweep;
    int pad5;
};

// Graphs with no split rows and at most this many units close every
// iteration in the sweep's last CTA instead of a fix-up launch.
constexpr uint32_t kCloseInSweepUnits = 8192;

// Where the sum of chunk slice s / lane goes (chunk_slot null: storage order).
__device__ __forceinline__ uint32_t chunk_slot_of(const uint32_t *chunk_slot, uint32_t s, int lane) {
    const uint32_t i = s * 32 + lane;
    return chunk_slot ? ld_stream(chunk_slot + i) : i;
}

// Adds the segment sums of row r (hot.cuh; written by the kernel before) to
// the sum of its other arcs.
template <typename V>
__device__ __forceinline__ V with_segments(const uint32_t *__restrict__ chunk_begin,
                                           const V *chunk_val, uint32_t n_hot, uint32_t r, V acc) {
    if (r < n_hot) {
        const uint32_t e = chunk_begin[r + 1];
        for (uint32_t k = chunk_begin[r]; k < e; ++k)
            acc += chunk_val[k];
    }
    return acc;
}

template <typename T>
__device__ __forceinline__ T t_mul(T a, T b);
template <>
__device__ __forceinline__ double t_mul<double>(double a, double b) { return __dmul_rn(a, b); }
template <>
__device__ __forceinline__ float t_mul<float>(float a, float b) { return __fmul_rn(a, b); }
template <typename T>
__device__ __forceinline__ T t_add(T a, T b);
template <>
__device__ __forceinline__ double t_add<double>(double a, double b) { return __dadd_rn(a, b); }
template <>
__device__ __forceinline__ float t_add<float>(float a, float b) { return __fadd_rn(a, b); }

// Finish row r from its in-arc sum `acc`: PageRank.cpp:64-65 (plus the sink
// term of distributeSinks), the residual term of PageRank.cpp:34-39 and the
// new gather-form value. No FMA contraction: the reference rounds the
// multiply and the add separately.
template <typename T, bool WEIGHTED, bool PART = false>
__device__ __forceinline__ void finish_row(const SweepArgs<T> &a, const RunParams &rp, T sink_coef,
                                           uint32_t r0, T acc, double &res, double &sink) {
    const uint32_t r = PART ? a.row_map[r0] : r0;
    const uint32_t dc = ld_stream(a.degc + r);
    const T deg = WEIGHTED ? ld_stream(a.degw + r) : static_cast<T>(dc);
    const T yo = a.y_in[(PART ? a.row_base : 0u) + r];
    if (rp.distribute)
        acc = t_add(acc, rp.personal ? t_mul(sink_coef, a.tele[r]) : sink_coef);
    T x = t_mul(acc, static_cast<T>(rp.damp));
    x = t_add(x, rp.personal ? t_mul(static_cast<T>(rp.one_minus_damp), a.tele[r])
                             : static_cast<T>(rp.tele_uniform));
    const bool is_sink = dc == 0;
    const T xo = is_sink ? yo : t_mul(yo, deg);
    const double d = static_cast<double>(xo) - static_cast<double>(x);
    res += rp.l2 ? __dmul_rn(d, d) : fabs(d);
    if (is_sink) {
        sink += static_cast<double>(x);
        a.y_out[r] = x;
    } else {
        a.y_out[r] = x / deg;
    }
}

// Per-run constants read where a row is finished. The volatile asm keeps each
// load at its use, so the values are not hoisted into registers held across
// the gather loop.
__device__ __forceinline__ double ld_keep(const double *p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ld_keep(const int *p) {
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

template <typename T, bool WEIGHTED, bool PART = false>
__device__ __forceinline__ void finish_row_sweep(const SweepArgs<T> &a, uint32_t r, T acc,
                                                 double &res, double &sink) {
    RunParams rp;
    rp.damp = ld_keep(&a.rp->damp);
    rp.tele_uniform = ld_keep(&a.rp->tele_uniform);
    rp.one_minus_damp = ld_keep(&a.rp->one_minus_damp);
    rp.distribute = ld_keep(&a.rp->distribute);
    rp.personal = ld_keep(&a.rp->personal);
    rp.l2 = ld_keep(&a.rp->l2);
    const T sink_coef = static_cast<T>(ld_keep(&a.st->sink_coef));
    finish_row<T, WEIGHTED, PART>(a, rp, sink_coef, r, acc, res, sink);
}

// Padding slots (column n, whose gathered value is the zero entry y[n]) skip
// the load and add zero, the same sum bit for bit without the L1 lookup.
// Gathers go through L1 with the default policy (__ldg); the kernel uses no
// shared memory, so the whole L1 caches the hot scores. The sweep is bound by
// L1 miss requests to L2 (one sector per scattered lane). Measured
// alternatives that were slower on B200: L2-only loads; holding the hottest
// scores in the shared memory of this kernel, beside its other gathers (a kernel
// that gathers from shared memory only is hot.cuh); per-lane L1 evict-last / no-allocate hints (the
// predicated loads raise register use and cut occupancy).

// Launch shapes of the sweep kernel: threads per CTA and slot steps per batch
// of independent gathers.
template <int TH, int UNROLL_>
struct SweepShape {
    static constexpr int threads = TH, unroll = UNROLL_;
};
constexpr int kNumSweepShapes = 4;

template <typename F>
inline void with_sweep_shape(int v, F &&f) {
    switch (v) {
    case 1: f(SweepShape<256, 8>{}); break;
    case 2: f(SweepShape<256, 4>{}); break;
    case 3: f(SweepShape<256, 16>{}); break;
    default: f(SweepShape<512, 8>{}); break;
    }
}

// Hot-source tier. The rows are relabelled by in-degree, and on power-law
// graphs in- and out-degree go together, so the first ids are also the
// sources that most arcs gather from (on directed R-MAT scale 24 the first
// 28,672 ids are the sources of 34% of the arcs, the first 57,344 of 46%).
// The tier copies y_in[0, hot) into shared memory at the start of every
// sweep, and a gather of such an id is a shared-memory load instead of a
// request through L1. Every other gather goes through L1 as before. Each CTA
// holds its own copy of the tier: two CTAs of 768 threads per SM (48 warps,
// as the regular sweep) where two copies fit, else one CTA of 1024 threads.
// Measured on B200 it is not faster than the whole L1 for the gathers (the
// shared memory it takes is L1 the gathers lose), so it is off by default.
constexpr int kHotThreads = 1024;
constexpr int kHotThreadsPair = 768;
constexpr int kHotUnroll = 8;
// Largest tier: 224 KB of the 227 KB a CTA may opt into (the rest holds the
// block reduction's scratch).
constexpr uint32_t kHotMaxBytes = 224u * 1024u;

template <typename T, bool HOT, bool PART = false>
__device__ __forceinline__ T gather_y(const SweepArgs<T> &a, const T *s_y, uint32_t c) {
    if (HOT && c < a.hot)
        return s_y[c];
    return c != (PART ? a.pad : a.n) ? __ldg(a.y_in + c) : T(0);
}

// 16-byte read-only load that does not allocate in L1 (the tier copy).
__device__ __forceinline__ uint4 ld_na_v4(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// Closes an iteration from the reduced residual sum r and sink mass s
// (PageRank.cpp:68-70): iteration count, stopping norm, trace, the sink term
// of the next sweep, the convergence flag. One thread, after every partial
// sum of the sweep is in r and s.
template <typename T>
__device__ __forceinline__ void close_iteration(const SweepArgs<T> &a, const RunParams &rp, double r,
                                                double s) {
    IterState *st = a.st;
    const unsigned long long it = st->iteration + 1;
    const double norm = rp.l2 ? sqrt(r) : r;
    st->iteration = it;
    st->residual = norm;
    st->residual_sum = r;
    if (it - 1 < a.trace_cap)
        a.trace[it - 1] = norm;
    st->sink_mass = s;
    st->sink_coef = rp.distribute ? (rp.personal ? s : s / static_cast<double>(a.n)) : 0.0;
    st->ticket = 0;
    st->queue = 0;
    __threadfence();
    st->done = (it >= rp.max_iterations || norm <= rp.tol) ? 1 : 0;
}

// Slices [s_begin, s_end) of one work unit: each lane accumulates one
// virtual row of a slice in arc order. Chunk slices store partial sums; row
// slices finish rows, adding their residual and sink terms to res / sink.
template <typename T, bool WEIGHTED, int UNROLL, bool HOT, bool PART>
__device__ __forceinline__ void sweep_unit(const SweepArgs<T> &a, const T *s_y, uint32_t s_begin,
                                           uint32_t s_end, int lane, double &res, double &sink) {
    for (uint32_t s = s_begin; s < s_end; ++s) {
        const uint32_t off = a.slice_off[s];
        const uint32_t len = a.slice_off[s + 1] - off;
        const size_t base = static_cast<size_t>(off) * 32 + lane;
        const uint32_t *cp = a.col_sell + base;
        T acc = T(0);
        uint32_t j = 0;
        for (; j + UNROLL <= len; j += UNROLL) {
            uint32_t c[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                c[k] = ld_stream(cp + static_cast<size_t>(j + k) * 32);
            T v[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                v[k] = gather_y<T, HOT, PART>(a, s_y, c[k]);
            if (WEIGHTED) {
#pragma unroll
                for (int k = 0; k < UNROLL; ++k)
                    v[k] = t_mul(v[k], ld_stream(a.w_sell + base + static_cast<size_t>(j + k) * 32));
            }
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                acc += v[k];
        }
        if (j < len) {
            // The last len - j < UNROLL steps as one predicated batch, so
            // their gathers are in flight together; the sum keeps the same
            // order (absent steps add nothing).
            uint32_t c[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                c[k] = j + k < len ? ld_stream(cp + static_cast<size_t>(j + k) * 32) : 0u;
            T v[UNROLL];
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                v[k] = j + k < len ? gather_y<T, HOT, PART>(a, s_y, c[k]) : T(0);
            if (WEIGHTED) {
#pragma unroll
                for (int k = 0; k < UNROLL; ++k)
                    if (j + k < len)
                        v[k] = t_mul(v[k], ld_stream(a.w_sell + base + static_cast<size_t>(j + k) * 32));
            }
#pragma unroll
            for (int k = 0; k < UNROLL; ++k)
                if (j + k < len)
                    acc += v[k];
        }
        if (s < a.s_chunk) {
            a.chunk_val[chunk_slot_of(a.chunk_slot, s, lane)] = acc;
        } else {
            const uint32_t r = a.n_long + (s - a.s_chunk) * 32 + lane;
            if (!WEIGHTED && !PART)
                acc = with_segments(a.chunk_begin, a.chunk_val, a.n_hot, r, acc);
            if (r < a.n)
                finish_row_sweep<T, WEIGHTED, PART>(a, r, acc, res, sink);
        }
    }
}

// The sweep: each warp walks its units (sweep_unit).
// Registers are fitted to 48 warps per SM (more warps do not make the sweep
// faster: it is bound by the rate of L1 miss requests), and to 32 for the
// other batch depths and the weighted FP64 sweep, which would spill at 48.
// HOT: the variant with the shared-memory tier (a.hot * sizeof(T) bytes of
// dynamic shared memory, a multiple of 16). PART: the row slice of a
// partitioned run (see SweepArgs.row_map).
// QUEUED: after a first unit of their own, warps take the next unit from a
// device counter (next_unit) instead of a fixed round-robin share, so warps
// that run faster take more of the graph and the sweep ends when the work
// does, not when the slowest share does (R-MAT 24, FP64: 0.874 ms against
// 0.956 ms with 8 round-robin units per warp, same scores bit for bit). Every unit's residual and sink partials go to their
// own slots (unit_res, unit_sink) after a fixed-order warp sum, and the
// fix-up adds them in a fixed order: the result does not depend on which
// warp ran which unit. The regular PageRank sweep and the row slices of a
// partitioned run are always QUEUED; the shared-memory tier keeps the
// round-robin units.
template <typename T, bool WEIGHTED, int THREADS, int UNROLL, bool HOT = false, bool PART = false,
          bool QUEUED = false>
__global__ void __launch_bounds__(THREADS, UNROLL != 8 || (WEIGHTED && sizeof(T) > 4) ? 1024 / THREADS : 1536 / THREADS)
    sweep_kernel(SweepArgs<T> a) {
    static_assert(!(QUEUED && HOT), "the queued sweep has no shared-memory tier");
    __shared__ double s_red[32];
    extern __shared__ __align__(16) unsigned char s_dyn[];
    T *s_y = reinterpret_cast<T *>(s_dyn);
    if (*(volatile int *)&a.st->done)
        return;
    const int lane = threadIdx.x & 31;
    if (QUEUED) {
        const uint32_t nw = gridDim.x * (THREADS / 32);
        for (uint32_t u = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5); u < a.units;
             u = next_unit(&a.st->queue, a.units, nw, lane)) {
            double res = 0.0, sink = 0.0;
            sweep_unit<T, WEIGHTED, UNROLL, false, PART>(a, s_y, a.unit_start[u],
                                                          a.unit_start[u + 1], lane, res, sink);
            res = warp_sum(res);
            sink = warp_sum(sink);
            if (lane == 0) {
                a.unit_res[u] = res;
                a.unit_sink[u] = sink;
                if (a.close_in_sweep)
                    __threadfence();  // visible to the CTA that closes the iteration
            }
        }
        if (!a.close_in_sweep)
            return;
        // The last CTA to finish adds the units' partials in unit order (a
        // fixed tree) and closes the iteration; no CTA waits for another.
        __shared__ bool s_last;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            s_last = atomicAdd(&a.st->ticket, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!s_last)
            return;
        __threadfence();
        double r = 0.0, sk = 0.0;
        for (uint32_t i = threadIdx.x; i < a.units; i += THREADS) {
            r += ((volatile double *)a.unit_res)[i];
            sk += ((volatile double *)a.unit_sink)[i];
        }
        r = block_sum<THREADS>(r, s_red);
        sk = block_sum<THREADS>(sk, s_red);
        if (threadIdx.x == 0)
            close_iteration(a, *a.rp, r, sk);
        return;
    }
    if (HOT) {
        const uint32_t vecs = a.hot * static_cast<uint32_t>(sizeof(T)) / 16u;
        const uint4 *src = reinterpret_cast<const uint4 *>(a.y_in);
        uint4 *dst = reinterpret_cast<uint4 *>(s_dyn);
        for (uint32_t i = threadIdx.x; i < vecs; i += THREADS)
            dst[i] = ld_na_v4(src + i);
        __syncthreads();
    }
    const uint32_t wpc = THREADS / 32;
    const uint32_t gw = blockIdx.x * wpc + (threadIdx.x >> 5);
    const uint32_t nw = gridDim.x * wpc;
    double res = 0.0, sink = 0.0;
    for (uint32_t u = gw; u < a.units; u += nw)
        sweep_unit<T, WEIGHTED, UNROLL, HOT, PART>(a, s_y, a.unit_start[u], a.unit_start[u + 1],
                                                   lane, res, sink);
    const double bres = block_sum<THREADS>(res, s_red);
    const double bsink = block_sum<THREADS>(sink, s_red);
    if (threadIdx.x == 0) {
        a.cta_res[blockIdx.x] = bres;
        a.cta_sink[blockIdx.x] = bsink;
    }
}

// Fix-up: finish the split rows from their chunk sums, then (last CTA) reduce
// all partial sums in index order and close the iteration
// (PageRank.cpp:68-70).
constexpr int kFixThreads = 256;

// CTAs of THREADS threads that finish the split rows (for_split_rows): a warp
// for each of the first n_vlong rows, then row_lanes() lanes for each other
// row. With source blocks no more CTAs than are resident at once (4 per SM; R-MAT
// 24, eight lanes: 0.641 ms an iteration, 0.645 with 8 per SM, 0.654 with 2).
template <int THREADS>
inline unsigned split_fix_ctas(uint32_t n_long, uint32_t n_vlong, uint32_t n_hot) {
    constexpr uint32_t w = THREADS / 32;
    const uint32_t rows = THREADS / row_lanes(n_hot);
    const uint64_t short_rows = n_long > n_vlong ? n_long - n_vlong : 0;
    return static_cast<unsigned>(std::max<uint64_t>(
        1, (n_vlong + w - 1) / w + std::min<uint64_t>(n_hot ? 592 : 1184, (short_rows + rows - 1) / rows)));
}

// Sum of one split row's chunk sums v[first], v[first + STEP], ... before ce,
// in double and in that order, with 16 loads in flight at a time.
template <uint32_t STEP, typename V>
__device__ __forceinline__ double strided_chunk_sum(const V *__restrict__ v, uint32_t first,
                                                    uint32_t ce) {
    constexpr int kBatch = 16;
    double part = 0.0;
    for (uint32_t k0 = first; k0 < ce; k0 += STEP * kBatch) {
        V x[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            const uint32_t k = k0 + STEP * q;
            x[q] = k < ce ? v[k] : V(0);
        }
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
            part += static_cast<double>(x[q]);
    }
    return part;
}

// Rows of more chunk sums than this are summed by a whole CTA where it has no
// more than kCtaRows of them: a warp adds about 800 sums a microsecond, so a row
// of 8M arcs (125,000 chunks of 64) held an iteration up for 0.15 ms, but eight
// rows of 5,000 sums one after the other take a CTA 20 us and its eight warps 7.
// 40 iterations of 4M arcs and one row of 2M more, FP64, a warp / a CTA: 3.7 /
// 2.4 ms; of 8M more 10.2 / 4.2.
constexpr uint32_t kCtaSums = 2048;
constexpr uint32_t kCtaRows = 2;

// Calls finish(r, sum) once for every split row r < n_long with the sum of its
// chunk sums, in double and in a fixed order: a warp, or a CTA (kCtaSums),
// for each of the first n_vlong rows, row_lanes() lanes for each other (four
// loads of a lane in flight; one thread per row took 42 us of every R-MAT 24
// iteration where source blocks give a row a dozen sums).
// Every thread of the CTA calls it.
template <int THREADS, typename V, typename F>
__device__ __forceinline__ void for_split_rows(const uint32_t *__restrict__ chunk_begin,
                                               const V *__restrict__ chunk_val, uint32_t n_long,
                                               uint32_t n_vlong, uint32_t n_hot, F &&finish) {
    constexpr uint32_t w = THREADS / 32;
    const uint32_t lanes = row_lanes(n_hot), shift = n_hot ? 2 : 0, rows = THREADS >> shift;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t vctas = (n_vlong + w - 1) / w;
    if (blockIdx.x < vctas) {
        __shared__ double s_part[32];
        // Rows blockIdx.x, + vctas, ...: the longest rows, which are first, go to
        // CTAs of their own.
        const uint32_t r = blockIdx.x + wid * vctas;
        const uint32_t b = r < n_vlong ? chunk_begin[r] : 0u;
        const uint32_t e = r < n_vlong ? chunk_begin[r + 1] : 0u;
        const int many = __syncthreads_count(lane == 0 && e - b > kCtaSums);
        const bool cta_rows = many > 0 && many <= static_cast<int>(kCtaRows);
        for (uint32_t q = blockIdx.x; cta_rows && q < n_vlong; q += vctas) {
            const uint32_t qb = chunk_begin[q], qe = chunk_begin[q + 1];
            if (qe - qb <= kCtaSums)
                continue;
            const double sum = block_sum<THREADS>(
                strided_chunk_sum<THREADS>(chunk_val, qb + threadIdx.x, qe), s_part);
            if (threadIdx.x == 0)
                finish(q, static_cast<V>(sum));
        }
        if (r >= n_vlong || (cta_rows && e - b > kCtaSums))
            return;
        const double sum = warp_sum(strided_chunk_sum<32>(chunk_val, b + lane, e));
        if (lane == 0)
            finish(r, static_cast<V>(sum));
        return;
    }
    const uint32_t sub = lane & (lanes - 1);
    const uint32_t stride = (gridDim.x - vctas) * rows;
    for (uint32_t base = n_vlong + (blockIdx.x - vctas) * rows + wid * (32u >> shift);
         base < n_long; base += stride) {
        const uint32_t r = base + (lane >> shift);
        const uint32_t e = r < n_long ? chunk_begin[r + 1] : 0u;
        double sum = 0.0;
        for (uint32_t k = r < n_long ? chunk_begin[r] + sub : 0u; k < e; k += 4 * lanes) {
            V x[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                x[q] = k + q * lanes < e ? chunk_val[k + q * lanes] : V(0);
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                sum += static_cast<double>(x[q]);
        }
        __syncwarp();
        for (uint32_t o = lanes / 2; o > 0; o >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (sub == 0 && r < n_long)
            finish(r, static_cast<V>(sum));
    }
}

template <typename T, bool WEIGHTED, bool PART = false>
__global__ void __launch_bounds__(kFixThreads) fixup_kernel(SweepArgs<T> a) {
    __shared__ double s_red[32];
    __shared__ bool s_last;
    if (*(volatile int *)&a.st->done)
        return;
    const RunParams rp = *a.rp;
    const T sink_coef = static_cast<T>(a.st->sink_coef);
    double res = 0.0, sink = 0.0;
    if (a.unit_res) {
        // Partials of a queued sweep: a fixed share of the units per thread.
        for (uint32_t i = blockIdx.x * kFixThreads + threadIdx.x; i < a.units;
             i += gridDim.x * kFixThreads) {
            res += a.unit_res[i];
            sink += a.unit_sink[i];
        }
    }
    for_split_rows<kFixThreads, T>(
        a.chunk_begin, a.chunk_val, a.n_long, a.n_vlong, a.n_hot, [&](uint32_t r, T sum) {
            finish_row<T, WEIGHTED, PART>(a, rp, sink_coef, r, sum, res, sink);
        });
    const double bres = block_sum<kFixThreads>(res, s_red);
    const double bsink = block_sum<kFixThreads>(sink, s_red);
    if (threadIdx.x == 0) {
        a.fix_res[blockIdx.x] = bres;
        a.fix_sink[blockIdx.x] = bsink;
        __threadfence();
        const unsigned prev = atomicAdd(&a.st->ticket, 1u);
        s_last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    // Fixed-order reduction of sweep-CTA and fix-up-CTA partials.
    double r = 0.0, s = 0.0;
    const uint32_t sweep_parts = a.unit_res ? 0u : a.sweep_ctas;
    for (uint32_t i = threadIdx.x; i < sweep_parts; i += kFixThreads) {
        r += ((volatile double *)a.cta_res)[i];
        s += ((volatile double *)a.cta_sink)[i];
    }
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += kFixThreads) {
        r += ((volatile double *)a.fix_res)[i];
        s += ((volatile double *)a.fix_sink)[i];
    }
    r = block_sum<kFixThreads>(r, s_red);
    s = block_sum<kFixThreads>(s, s_red);
    if (threadIdx.x == 0)
        close_iteration(a, rp, r, s);
}

} // namespace nkg
