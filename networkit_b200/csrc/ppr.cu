// Batched personalised PageRank: k teleport vectors t_j = e_{seed_j} solved
// together as one FP32 SpMM over the shared in-CSR (no reference counterpart;
// each column is PageRank.cpp:56-70 with the uniform teleport replaced by
// t_j). Per column: FP64 residual, FP64 sink mass, and the column stops
// (freezes) once its residual is at most tol.
//
// Layout: the iterate is node-major, Y[r * kp + j], in gather form (x/deg,
// sinks x), with kp the columns rounded up to whole 32-byte sectors (k = 37:
// 40 columns, where rows padded to 128 columns moved 3.2 times the bytes).
// A virtual row is a whole row, or a kChunk-arc chunk of a long row; warps
// walk contiguous, cost-balanced ranges of them, so every sum has a fixed
// order. Up to 64 columns (ppr_sweep) a lane holds 4 columns of a row and the
// warp's groups of `lanes` lanes take different arcs of the same row (37
// columns: 3 arcs at a time); the groups' sums are added at the row's end. With
// more columns (ppr_sweep_one) the whole warp takes one arc. The other kernels
// treat a row of more than 128 columns as two parts, each the work of its own warp.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "graph.hpp"
#include "host.hpp"

namespace nkg {
namespace {

constexpr int kPprThreads = 256;
constexpr int kPprWarps = kPprThreads / 32;
constexpr uint32_t kPprBatch = 4;  // arcs of a lane in flight (6 and 8 cost warps: slower)

struct PprState {
    unsigned long long iteration;
    int all_done;
    unsigned int ticket;
};

struct PprArgs {
    const uint32_t *__restrict__ row_ptr;    // n+1 (relabelled in-CSR)
    const uint32_t *__restrict__ col;
    const uint32_t *__restrict__ degc;
    const uint32_t *__restrict__ chunk_begin;  // n_long+1
    const uint2 *__restrict__ vrange;          // per virtual row: its arcs [x, y)
    const uint32_t *__restrict__ unit_start;   // units+1 virtual-row indices
    const uint32_t *__restrict__ seed;         // kp: relabelled seed id (kNone: padding column)
    const float *__restrict__ y_in;            // n * kp
    float *__restrict__ y_out;
    float *__restrict__ chunk_val;             // n_chunks * kp
    int *__restrict__ active;                  // kp
    float *__restrict__ sink_coef;             // kp: sink term of the next sweep
    double *__restrict__ cta_res;              // per CTA * kp
    double *__restrict__ cta_sink;
    double *__restrict__ col_res;              // kp: last residual
    unsigned long long *__restrict__ col_iter; // kp: sweeps until converged
    PprState *st;
    double damp, tol;
    unsigned long long max_iterations;
    uint32_t n, n_long, n_chunks, units, kp, sweep_ctas;
    uint32_t lanes, groups, parts;             // lane layout of a row (above)
    int l2, distribute;
};

// This lane's place in the layout: its group of lanes (>= groups: idle), its
// first column, whether it finishes rows (group 0).
struct PprLane {
    uint32_t group, col;
    bool on;     // loads columns
    bool first;  // holds the row's sums
};
__device__ __forceinline__ PprLane ppr_lane(const PprArgs &a) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    PprLane L;
    L.group = lane / a.lanes;
    L.on = L.group < a.groups;
    L.first = L.group == 0;
    L.col = ((wid & (a.parts - 1)) * a.lanes + lane % a.lanes) * 4;
    return L;
}

// Virtual rows: [0, n_chunks) chunks of the long rows, then rows n_long..n-1.

__device__ __forceinline__ void add4(float (&acc)[4], const float4 &v) {
    acc[0] += v.x;
    acc[1] += v.y;
    acc[2] += v.z;
    acc[3] += v.w;
}

// Sum of the source rows of arcs [b, e) in this lane's columns. Group g takes
// arcs g, g + groups, ...; the groups' sums are added into group 0 in a fixed
// order.
__device__ __forceinline__ void accumulate(const PprArgs &a, const PprLane &L, uint32_t b,
                                           uint32_t e, float (&acc)[4]) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t groups = a.groups;
    const float *y = a.y_in + L.col;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        acc[c] = 0.f;
    for (uint32_t base = b; base < e; base += 32) {
        const uint32_t cnt = min(32u, e - base);
        const uint32_t cl = lane < cnt ? ld_stream(a.col + base + lane) : 0u;
        for (uint32_t i = 0; i < cnt; i += kPprBatch * groups) {
            float4 v[kPprBatch];
#pragma unroll
            for (uint32_t u = 0; u < kPprBatch; ++u) {
                const uint32_t k = i + u * groups + L.group;
                const uint32_t src = __shfl_sync(0xffffffffu, cl, k & 31);
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (L.on && k < cnt)
                    v[u] = __ldg(reinterpret_cast<const float4 *>(y + static_cast<size_t>(src) * a.kp));
            }
#pragma unroll
            for (uint32_t u = 0; u < kPprBatch; ++u)
                add4(acc, v[u]);
        }
    }
    if (a.lanes * groups == 32 && !(groups & (groups - 1))) {
        // As a tree: one group after the other took 124 shuffles with 32 groups, more
        // than the gathers of a short row (1M rows of two arcs, 16 sweeps of one column:
        // 12.3 ms one by one, 9.4 with rows padded to 128 columns before that).
        for (uint32_t o = a.lanes; o < 32; o <<= 1)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        return;
    }
    const float t[4] = {acc[0], acc[1], acc[2], acc[3]};
    for (uint32_t g = 1; g < groups; ++g) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            acc[c] += __shfl_sync(0xffffffffu, t[c], (lane + g * a.lanes) & 31);
    }
}

// Row r's new value in one column (PageRank.cpp:64-65 in gather form) from its
// sum; frozen columns keep the old one.
__device__ __forceinline__ float finish_column(const PprArgs &a, uint32_t r, uint32_t dc, float deg,
                                               float dampf, float omd, float sum, float yo, int act,
                                               float sc, uint32_t seed, double &res, double &sink) {
    if (!act)
        return yo;
    const float tel = (r == seed) ? 1.f : 0.f;
    if (a.distribute)
        sum = __fadd_rn(sum, __fmul_rn(sc, tel));
    float x = __fmul_rn(sum, dampf);
    x = __fadd_rn(x, __fmul_rn(omd, tel));
    const float xo = dc ? __fmul_rn(yo, deg) : yo;
    const double d = static_cast<double>(xo) - static_cast<double>(x);
    res += a.l2 ? d * d : fabs(d);
    if (dc)
        return x / deg;
    sink += static_cast<double>(x);
    return x;
}

// Finish row r in columns col .. + 3. What is constant per column is loaded
// here: held across the gathers it made the sweep spill at 64 registers.
template <typename Sink>
__device__ __forceinline__ void finish(const PprArgs &a, uint32_t col, uint32_t r,
                                       const float (&acc)[4], double (&res)[4], Sink &&sink) {
    const int4 on = __ldg(reinterpret_cast<const int4 *>(a.active + col));
    const uint4 sd = __ldg(reinterpret_cast<const uint4 *>(a.seed + col));
    const float4 s4 = a.distribute ? __ldg(reinterpret_cast<const float4 *>(a.sink_coef + col))
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
    const int act[4] = {on.x, on.y, on.z, on.w};
    const uint32_t seed[4] = {sd.x, sd.y, sd.z, sd.w};
    const float sc[4] = {s4.x, s4.y, s4.z, s4.w};
    const uint32_t dc = ld_stream(a.degc + r);
    const float deg = static_cast<float>(dc);
    const size_t at = static_cast<size_t>(r) * a.kp + col;
    const float dampf = static_cast<float>(a.damp), omd = static_cast<float>(1.0 - a.damp);
    const float4 yo4 = __ldg(reinterpret_cast<const float4 *>(a.y_in + at));
    const float yo[4] = {yo4.x, yo4.y, yo4.z, yo4.w};
    float yn[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
        yn[c] = finish_column(a, r, dc, deg, dampf, omd, acc[c], yo[c], act[c], sc[c], seed[c],
                              res[c], sink[c]);
    *reinterpret_cast<float4 *>(a.y_out + at) = make_float4(yn[0], yn[1], yn[2], yn[3]);
}

// Per-column block sums of `res` and `sink` over the warps (and, with `groups`
// > 1, the groups of lanes) that hold the column, plus rows blockIdx.x,
// blockIdx.x + gridDim.x, ... of `more` rows of earlier partials, into
// out_res/out_sink[blockIdx.x * kp ..]. s_buf: kPprWarps * 128 doubles.
__device__ __forceinline__ void column_partials(const PprArgs &a, const PprLane &L, uint32_t groups,
                                                const double (&res)[4], const double (&sink)[4],
                                                double *s_buf, double *out_res, double *out_sink,
                                                const double *more_res, const double *more_sink,
                                                uint32_t more) {
    const uint32_t wid = threadIdx.x >> 5, kp = a.kp, w4 = 4 * a.lanes;
    const uint32_t part_col = L.col - (wid & (a.parts - 1)) * w4;
    for (int pass = 0; pass < 2; ++pass) {
        __syncthreads();
        if (L.group < groups)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                s_buf[(wid * groups + L.group) * w4 + part_col + c] = pass == 0 ? res[c] : sink[c];
        __syncthreads();
        const double *m = pass == 0 ? more_res : more_sink;
        for (uint32_t col = threadIdx.x; col < kp; col += kPprThreads) {
            const uint32_t part = col / w4;
            double s = 0.0;
            for (uint32_t w = part; w < kPprWarps; w += a.parts)
                for (uint32_t g = 0; g < groups; ++g)
                    s += s_buf[(w * groups + g) * w4 + col - part * w4];
#pragma unroll 4
            for (uint32_t i = blockIdx.x; i < more; i += gridDim.x)
                s += m[static_cast<size_t>(i) * kp + col];
            (pass == 0 ? out_res : out_sink)[static_cast<size_t>(blockIdx.x) * kp + col] = s;
        }
    }
    __threadfence();  // partials visible device-wide before any ticket
}

// The sweep of more than 64 columns: all lanes of a warp take the same arc, a
// lane holding 4 H columns of it (H 2: more than 128 columns). Its gathers are
// unconditional (lanes past the columns load the first ones, arcs past a row's
// last whole batch go one by one): with loads under a condition, as ppr_sweep
// has them, the compiler branches around each and the four of a batch no longer
// overlap. Bound by L2 and DRAM on random rows and by the row ends, where a warp
// has nothing in flight: 24 warps per SM for H 2 (80 registers; the sink sums,
// which few rows add to, are in shared memory), 32 for H 1. 16 sweeps, ms, with
// the rows as bulk copies into shared memory instead / now: 256 columns R-MAT 20
// 59.8 / 41.6, hyperbolic 1M 48.2 / 39.6, Barabasi-Albert 4M 204 / 205,
// Erdos-Renyi 1M 37.5 / 37.9; 129 columns 52.8 / 33.5, 44.6 / 33.5, 178 / 168,
// 32.7 / 32.5. The copies go past L1 and cost an issue slot each, so they lost
// where sources repeat and won nowhere by more than 1%. H 1 against ppr_sweep:
// R-MAT 22, 128 columns 75.1 / 89.2, 68 columns 66.6 / 83.7.
template <int H>
__global__ void __launch_bounds__(kPprThreads, H == 1 ? 4 : 3) ppr_sweep_one(PprArgs a) {
    extern __shared__ double s_buf[];
    if (*(volatile int *)&a.st->all_done)
        return;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool on = lane * 4 * H < a.kp;
    const uint32_t col = on ? lane * 4 * H : 0;
    double res[H][4];
    double *sink = s_buf + wid * a.kp + col;
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            res[h][c] = 0.0;
            if (on)
                sink[4 * h + c] = 0.0;
        }
    const float *ycol = a.y_in + col;
    const uint32_t gw = blockIdx.x * kPprWarps + wid, nw = gridDim.x * kPprWarps;
    for (uint32_t u = gw; u < a.units; u += nw) {
        const uint32_t v_end = a.unit_start[u + 1];
        for (uint32_t v = a.unit_start[u]; v < v_end; ++v) {
            const uint2 arcs = __ldg(a.vrange + v);
            float acc[H][4];
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    acc[h][c] = 0.f;
            for (uint32_t base = arcs.x; base < arcs.y; base += 32) {
                const uint32_t cnt = min(32u, arcs.y - base);
                const uint32_t cl = lane < cnt ? ld_stream(a.col + base + lane) : 0u;
                uint32_t i = 0;
                for (; i + kPprBatch <= cnt; i += kPprBatch) {
                    float4 x[kPprBatch][H];
#pragma unroll
                    for (uint32_t q = 0; q < kPprBatch; ++q) {
                        const uint32_t src = __shfl_sync(0xffffffffu, cl, i + q);
                        const float4 *y =
                            reinterpret_cast<const float4 *>(ycol + static_cast<size_t>(src) * a.kp);
#pragma unroll
                        for (int h = 0; h < H; ++h)
                            x[q][h] = __ldg(y + h);
                    }
#pragma unroll
                    for (uint32_t q = 0; q < kPprBatch; ++q)
#pragma unroll
                        for (int h = 0; h < H; ++h)
                            add4(acc[h], x[q][h]);
                }
                for (; i < cnt; ++i) {
                    const uint32_t src = __shfl_sync(0xffffffffu, cl, i);
                    const float4 *y =
                        reinterpret_cast<const float4 *>(ycol + static_cast<size_t>(src) * a.kp);
#pragma unroll
                    for (int h = 0; h < H; ++h)
                        add4(acc[h], __ldg(y + h));
                }
            }
            if (!on)
                continue;
#pragma unroll
            for (int h = 0; h < H; ++h) {
                if (v < a.n_chunks)
                    *reinterpret_cast<float4 *>(a.chunk_val + static_cast<size_t>(v) * a.kp + col +
                                                4 * h) =
                        make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
                else
                    finish(a, col + 4 * h, a.n_long + (v - a.n_chunks), acc[h], res[h], sink + 4 * h);
            }
        }
    }
    // Per-column sums over the warps (column_partials).
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            __syncthreads();
            if (on)
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        sink[4 * h + c] = res[h][c];
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < a.kp; k += kPprThreads) {
            double sum = 0.0;
            for (uint32_t w = 0; w < kPprWarps; ++w)
                sum += s_buf[w * a.kp + k];
            (pass == 0 ? a.cta_sink : a.cta_res)[static_cast<size_t>(blockIdx.x) * a.kp + k] = sum;
        }
    }
}

__global__ void __launch_bounds__(kPprThreads, 4) ppr_sweep(PprArgs a) {
    extern __shared__ double s_buf[];
    if (*(volatile int *)&a.st->all_done)
        return;
    const PprLane L = ppr_lane(a);
    double res[4], sink[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
        res[c] = sink[c] = 0.0;
    const uint32_t gw = blockIdx.x * kPprWarps + (threadIdx.x >> 5);
    const uint32_t nw = gridDim.x * kPprWarps;
    for (uint32_t u = gw; u < a.units; u += nw) {
        const uint32_t v_end = a.unit_start[u + 1];
        uint32_t v = a.unit_start[u];
        if (v >= v_end)
            continue;
        uint2 cur = __ldg(a.vrange + v);
        for (; v < v_end; ++v) {
            const uint2 nxt = v + 1 < v_end ? __ldg(a.vrange + v + 1) : make_uint2(0u, 0u);
            float acc[4];
            accumulate(a, L, cur.x, cur.y, acc);
            if (L.first) {
                if (v < a.n_chunks)
                    *reinterpret_cast<float4 *>(a.chunk_val + static_cast<size_t>(v) * a.kp + L.col) =
                        make_float4(acc[0], acc[1], acc[2], acc[3]);
                else
                    finish(a, L.col, a.n_long + (v - a.n_chunks), acc, res, sink);
            }
            cur = nxt;
        }
    }
    column_partials(a, L, 1, res, sink, s_buf, a.cta_res, a.cta_sink, nullptr, nullptr, 0);
}

// Long rows: sum their chunk partials in order (a warp per row and part),
// finish them, then the last CTA closes the iteration per column. Every CTA
// adds its share of the sweep's per-CTA partials to its own, so the last one
// is left with gridDim.x rows of partials, which it adds eight at a time (one
// CTA that added the sweep's 600 to 900 rows itself, one after the other, took
// 0.4 ms of every sweep).
__global__ void __launch_bounds__(kPprThreads) ppr_fixup(PprArgs a, double *fix_res,
                                                         double *fix_sink) {
    extern __shared__ double s_buf[];
    __shared__ bool s_last;
    if (*(volatile int *)&a.st->all_done)
        return;
    const PprLane L = ppr_lane(a);
    double res[4], sink[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
        res[c] = sink[c] = 0.0;
    const uint32_t wpc = kPprWarps / a.parts;
    const uint32_t gw = blockIdx.x * wpc + (threadIdx.x >> 5) / a.parts;
    const uint32_t nw = gridDim.x * wpc;
    for (uint32_t r = gw; r < a.n_long; r += nw) {
        if (!L.first)
            continue;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const uint32_t ke = a.chunk_begin[r + 1];
#pragma unroll 8
        for (uint32_t k = a.chunk_begin[r]; k < ke; ++k)
            add4(acc, *reinterpret_cast<const float4 *>(a.chunk_val + static_cast<size_t>(k) * a.kp + L.col));
        finish(a, L.col, r, acc, res, sink);
    }
    column_partials(a, L, 1, res, sink, s_buf, fix_res, fix_sink, a.cta_res, a.cta_sink,
                    a.sweep_ctas);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&a.st->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    const unsigned long long it = a.st->iteration + 1;
    int any_active = 0;
    for (uint32_t col = threadIdx.x; col < a.kp; col += kPprThreads) {
        double r = 0.0, s = 0.0;
#pragma unroll 8
        for (uint32_t i = 0; i < gridDim.x; ++i) {
            r += __ldcg(fix_res + static_cast<size_t>(i) * a.kp + col);
            s += __ldcg(fix_sink + static_cast<size_t>(i) * a.kp + col);
        }
        if (a.active[col]) {
            const double norm = a.l2 ? sqrt(r) : r;
            a.col_res[col] = norm;
            a.col_iter[col] = it;
            a.sink_coef[col] = static_cast<float>(s);
            if (norm <= a.tol || it >= a.max_iterations)
                a.active[col] = 0;
            else
                any_active = 1;
        }
    }
    any_active = __syncthreads_or(any_active);
    if (threadIdx.x == 0) {
        a.st->iteration = it;
        a.st->ticket = 0;
        __threadfence();
        a.st->all_done = any_active ? 0 : 1;
    }
}

// x = 1/n in gather form for every column.
__global__ void ppr_init(float *__restrict__ y, const uint32_t *__restrict__ degc, uint32_t n,
                         uint32_t kp, float x0) {
    const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (i >= static_cast<uint64_t>(n) * kp)
        return;
    const uint32_t dc = degc[i / kp];
    y[i] = dc ? x0 / static_cast<float>(dc) : x0;
}

// Column sums of x (and of x over sinks), FP64, fixed order: every group of
// lanes takes rows of its own.
__global__ void __launch_bounds__(kPprThreads) ppr_colsum(PprArgs a, const float *__restrict__ y,
                                                          double *part_sum, double *part_sink) {
    extern __shared__ double s_buf[];
    const PprLane L = ppr_lane(a);
    double sum[4], sink[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
        sum[c] = sink[c] = 0.0;
    const uint32_t wpc = kPprWarps / a.parts;
    const uint32_t gw = blockIdx.x * wpc + (threadIdx.x >> 5) / a.parts;
    const uint32_t nw = gridDim.x * wpc;
    if (L.on) {
#pragma unroll 4
        for (uint32_t r = gw * a.groups + L.group; r < a.n; r += nw * a.groups) {
            const uint32_t dc = __ldg(a.degc + r);
            const float4 v =
                __ldg(reinterpret_cast<const float4 *>(y + static_cast<size_t>(r) * a.kp + L.col));
            const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float x = dc ? __fmul_rn(vv[t], static_cast<float>(dc)) : vv[t];
                sum[t] += x;
                if (!dc)
                    sink[t] += x;
            }
        }
    }
    column_partials(a, L, a.groups, sum, sink, s_buf, part_sum, part_sink, nullptr, nullptr, 0);
}

// Column j of the output (caller's ids): out[j*z + o] = x_j(inv[o]) / factor_j.
// A block transposes 32 nodes x kp columns through shared memory.
__global__ void ppr_output(const float *__restrict__ y, const uint32_t *__restrict__ degc,
                           const uint32_t *__restrict__ inv, uint64_t z, uint32_t n, uint32_t k,
                           uint32_t kp, const double *__restrict__ factor, float *__restrict__ out) {
    extern __shared__ float s_tile[];  // 32 x (kp + 1)
    const uint64_t o0 = static_cast<uint64_t>(blockIdx.x) * 32;
    for (uint32_t i = threadIdx.x; i < 32 * kp; i += blockDim.x) {
        const uint32_t node = i / kp, col = i % kp;
        const uint64_t o = o0 + node;
        float v = 0.f;
        if (o < z) {
            const uint32_t r = inv[o];
            if (r == kNone) {
                v = 1.f / static_cast<float>(n);
            } else {
                const uint32_t dc = degc[r];
                const float yv = y[static_cast<size_t>(r) * kp + col];
                const double x = dc ? static_cast<double>(__fmul_rn(yv, static_cast<float>(dc)))
                                    : static_cast<double>(yv);
                v = static_cast<float>(x / factor[col]);
            }
        }
        s_tile[node * (kp + 1) + col] = v;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 32 * k; i += blockDim.x) {
        const uint32_t col = i / 32, node = i % 32;
        const uint64_t o = o0 + node;
        if (o < z)
            out[static_cast<size_t>(col) * z + o] = s_tile[node * (kp + 1) + col];
    }
}

// Arcs [x, y) and cost of every virtual row.
__global__ void ppr_vrow_ranges(const uint32_t *__restrict__ row_ptr,
                                const uint32_t *__restrict__ chunk_begin,
                                const uint32_t *__restrict__ chunk_row, uint32_t n_chunks,
                                uint32_t n_long, uint32_t n, uint2 *__restrict__ range,
                                uint64_t *__restrict__ cost) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nv = n_chunks + (n - n_long);
    if (v >= nv)
        return;
    uint32_t b, e;
    if (v < n_chunks) {
        const uint32_t r = chunk_row[v];
        const uint32_t c = v - chunk_begin[r];
        b = row_ptr[r] + c * kChunk;
        e = min(row_ptr[r + 1], b + kChunk);
    } else {
        const uint32_t r = n_long + (v - n_chunks);
        b = row_ptr[r];
        e = row_ptr[r + 1];
    }
    range[v] = make_uint2(b, e);
    // Arcs, and eight arcs' time for the row's end. With four, the rows without
    // arcs, which are last in the order, made the last units the longest: R-MAT
    // 20, 16 sweeps, 4 / 8 / 16 arcs: 37 columns 15.1 / 13.5 / 12.9 ms, 64 16.4 /
    // 14.6 / 14.7, 256 47.2 / 41.4 / 42.9.
    cost[v] = static_cast<uint64_t>(e - b) + 8;
}

__global__ void ppr_unit_bounds(const uint64_t *__restrict__ cost_incl, uint32_t nv, uint32_t units,
                                uint32_t *__restrict__ unit_start) {
    const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u > units)
        return;
    if (u == 0) {
        unit_start[0] = 0;
        return;
    }
    if (u == units) {
        unit_start[u] = nv;
        return;
    }
    const uint64_t target = cost_incl[nv - 1] * u / units;
    uint32_t lo = 0, hi = nv;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (cost_incl[mid] < target)
            lo = mid + 1;
        else
            hi = mid;
    }
    unit_start[u] = lo + 1 < nv ? lo + 1 : nv;
}

__global__ void ppr_row_lengths(const uint32_t *__restrict__ row_ptr, uint32_t n,
                                uint32_t *__restrict__ rowlen) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n)
        rowlen[r] = row_ptr[r + 1] - row_ptr[r];
}

__global__ void ppr_chunk_rows(const uint32_t *__restrict__ chunk_begin, uint32_t n_long,
                               uint32_t *__restrict__ chunk_row) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (uint32_t r = warp; r < n_long; r += nwarps)
        for (uint32_t k = chunk_begin[r] + lane; k < chunk_begin[r + 1]; k += 32)
            chunk_row[k] = r;
}

__global__ void ppr_seeds(const uint32_t *__restrict__ seeds_orig, const uint32_t *__restrict__ inv,
                          uint32_t k, uint32_t kp, uint32_t *__restrict__ seed, int *__restrict__ active,
                          float *__restrict__ sink_coef, float s0, int *__restrict__ bad) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= kp)
        return;
    if (j < k) {
        const uint32_t r = inv[seeds_orig[j]];
        if (r == kNone)
            atomicExch(bad, 1);
        seed[j] = r;
        active[j] = 1;
        sink_coef[j] = s0;
    } else {
        seed[j] = kNone;
        active[j] = 0;
        sink_coef[j] = 0.f;
    }
}

void run_ppr(nkg_graph *g, const nkg_pr_params &p, uint32_t k, const uint32_t *seeds_host,
             float *out, bool out_on_device, uint64_t *iters_out, nkg_stats *stats) {
    cudaStream_t s = g->stream;
    const uint32_t n = static_cast<uint32_t>(g->n);
    // Lane layout: see the head of this file.
    const uint32_t parts = k > 128 ? 2 : 1;
    uint32_t lanes = std::max<uint32_t>(1, ceil_div(k, 4 * parts));
    if (lanes > 1)
        lanes = (lanes + 1) / 2 * 2;  // whole 32-byte sectors
    const uint32_t groups = 32 / lanes;
    const uint32_t kp = 4 * lanes * parts;
    const unsigned sms = num_sms(g->device);
    NKG_CUDA(cudaEventRecord(g->ev0, s));

    // Virtual rows and their cost-balanced units.
    if (!g->rc_begin) {
        DeviceArray<uint32_t> rowlen(n), begin;
        ppr_row_lengths<<<ceil_div(n, 256), 256, 0, s>>>(g->row_ptr.get(), n, rowlen.get());
        NKG_CUDA(cudaGetLastError());
        uint32_t vlong = 0, chunk = kChunk;
        g->rc_chunks = row_chunks(rowlen.get(), n, g->arcs, sms, chunk, g->rc_long, vlong, begin, s);
        NKG_CUDA(cudaStreamSynchronize(s));
        g->rc_begin = std::move(begin);  // complete, or not there
    }
    const uint32_t n_long = g->rc_long, n_chunks = g->rc_chunks;
    const uint32_t *chunk_begin = g->rc_begin.get();
    const uint32_t nv = n_chunks + (n - n_long);
    DeviceArray<uint32_t> chunk_row(std::max<uint32_t>(n_chunks, 1));
    if (n_long)
        ppr_chunk_rows<<<sms * 4, 256, 0, s>>>(chunk_begin, n_long, chunk_row.get());
    int occ = 0;
    const size_t smem_sweep = static_cast<size_t>(kPprWarps) * 128 * sizeof(double);
    // More than 64 columns: one arc per warp and step (ppr_sweep_one).
    const auto sweep = groups > 1 ? ppr_sweep : parts == 1 ? ppr_sweep_one<1> : ppr_sweep_one<2>;
    NKG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sweep, kPprThreads,
                                                           smem_sweep * parts));
    occ = std::max(occ, 1);
    const uint32_t sweep_ctas = static_cast<uint32_t>(std::max<uint64_t>(
        1, std::min<uint64_t>(static_cast<uint64_t>(occ) * sms, (nv + kPprWarps - 1) / kPprWarps)));
    const uint32_t units = std::max<uint32_t>(
        1, std::min<uint32_t>(sweep_ctas * kPprWarps * 4, std::max<uint32_t>(nv, 1)));
    DeviceArray<uint64_t> cost(std::max<uint32_t>(nv, 1)), cost_incl(std::max<uint32_t>(nv, 1));
    DeviceArray<uint32_t> unit_start(units + 1);
    DeviceArray<uint2> vrange(std::max<uint32_t>(nv, 1));
    if (nv) {
        ppr_vrow_ranges<<<ceil_div(nv, 256), 256, 0, s>>>(g->row_ptr.get(), chunk_begin,
                                                          chunk_row.get(), n_chunks, n_long, n,
                                                          vrange.get(), cost.get());
        size_t tb = 0;
        NKG_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tb, cost.get(), cost_incl.get(),
                                               static_cast<int64_t>(nv), s));
        DeviceArray<unsigned char> tmp(tb);
        NKG_CUDA(cub::DeviceScan::InclusiveSum(tmp.get(), tb, cost.get(), cost_incl.get(),
                                               static_cast<int64_t>(nv), s));
    }
    ppr_unit_bounds<<<ceil_div(units + 1, 256), 256, 0, s>>>(cost_incl.get(), nv, units,
                                                             unit_start.get());
    // At most 16 rows of the sweep's partials per fix-up CTA.
    const uint32_t fix_ctas = std::max<uint32_t>(
        ceil_div(sweep_ctas, 16),
        std::min<uint32_t>(sms * 2, ceil_div(static_cast<uint64_t>(n_long) * parts, kPprWarps)));

    // Per-call buffers.
    DeviceArray<float> y0(static_cast<size_t>(n) * kp), y1(static_cast<size_t>(n) * kp);
    DeviceArray<float> chunk_val(static_cast<size_t>(std::max<uint32_t>(n_chunks, 1)) * kp);
    DeviceArray<uint32_t> d_seeds_orig(k), seed(kp);
    DeviceArray<int> active(kp), bad(1);
    DeviceArray<float> sink_coef(kp);
    DeviceArray<double> cta_res(static_cast<size_t>(sweep_ctas) * kp),
        cta_sink(static_cast<size_t>(sweep_ctas) * kp), fix_res(static_cast<size_t>(fix_ctas) * kp),
        fix_sink(static_cast<size_t>(fix_ctas) * kp), col_res(kp);
    DeviceArray<unsigned long long> col_iter(kp);
    DeviceArray<PprState> st(1);
    NKG_CUDA(cudaMemcpyAsync(d_seeds_orig.get(), seeds_host, k * sizeof(uint32_t),
                             cudaMemcpyHostToDevice, s));
    NKG_CUDA(cudaMemsetAsync(bad.get(), 0, sizeof(int), s));
    NKG_CUDA(cudaMemsetAsync(st.get(), 0, sizeof(PprState), s));
    NKG_CUDA(cudaMemsetAsync(col_iter.get(), 0, kp * sizeof(unsigned long long), s));
    NKG_CUDA(cudaMemsetAsync(col_res.get(), 0, kp * sizeof(double), s));
    const float x0 = 1.f / static_cast<float>(n);
    // distributeSinks: the first sweep spreads the start vector's sink mass.
    const float s0 = p.distribute_sinks ? static_cast<float>(static_cast<double>(g->sinks) / n) : 0.f;
    ppr_seeds<<<ceil_div(kp, 256), 256, 0, s>>>(d_seeds_orig.get(), g->inv.get(), k, kp,
                                                seed.get(), active.get(), sink_coef.get(), s0,
                                                bad.get());
    require(read_scalar(bad.get(), s) == 0, "a seed is not an existing node");
    ppr_init<<<ceil_div(static_cast<uint64_t>(n) * kp, 256), 256, 0, s>>>(y0.get(), g->degc.get(),
                                                                          n, kp, x0);
    NKG_CUDA(cudaGetLastError());

    PprArgs a{};
    a.row_ptr = g->row_ptr.get();
    a.col = g->col.get();
    a.degc = g->degc.get();
    a.chunk_begin = chunk_begin;
    a.vrange = vrange.get();
    a.unit_start = unit_start.get();
    a.seed = seed.get();
    a.chunk_val = chunk_val.get();
    a.active = active.get();
    a.sink_coef = sink_coef.get();
    a.cta_res = cta_res.get();
    a.cta_sink = cta_sink.get();
    a.col_res = col_res.get();
    a.col_iter = col_iter.get();
    a.st = st.get();
    a.damp = p.damp;
    a.tol = p.tol;
    a.max_iterations = p.max_iterations;
    a.n = n;
    a.n_long = n_long;
    a.n_chunks = n_chunks;
    a.units = units;
    a.kp = kp;
    a.sweep_ctas = sweep_ctas;
    a.lanes = lanes;
    a.groups = groups;
    a.parts = parts;
    a.l2 = p.norm == NKG_NORM_L2;
    a.distribute = p.distribute_sinks ? 1 : 0;

    uint64_t launches = 4;
    PprState h{};
    for (uint64_t it = 0;; it += 8) {
        for (int i = 0; i < 8; ++i) {
            a.y_in = ((it + i) & 1) ? y1.get() : y0.get();
            a.y_out = ((it + i) & 1) ? y0.get() : y1.get();
            sweep<<<sweep_ctas, kPprThreads, smem_sweep * parts, s>>>(a);
            ppr_fixup<<<fix_ctas, kPprThreads, smem_sweep, s>>>(a, fix_res.get(), fix_sink.get());
        }
        launches += 16;
        NKG_CUDA(cudaGetLastError());
        h = read_scalar(st.get(), s);
        if (h.all_done)
            break;
        check_cancel(g, "personalised PageRank run cancelled");
    }
    NKG_CUDA(cudaEventRecord(g->ev1, s));
    const float *yfin = (h.iteration & 1) ? y1.get() : y0.get();

    // Normalisation per column (PageRank.cpp:75-92), output in the caller's ids.
    const uint32_t cs_ctas = std::min<uint32_t>(sms * 2, std::max<uint32_t>((n + kPprWarps - 1) / kPprWarps, 1));
    DeviceArray<double> part_sum(static_cast<size_t>(cs_ctas) * kp), part_sink(static_cast<size_t>(cs_ctas) * kp);
    ppr_colsum<<<cs_ctas, kPprThreads, smem_sweep, s>>>(a, yfin, part_sum.get(), part_sink.get());
    std::vector<double> hs(static_cast<size_t>(cs_ctas) * kp), hk(static_cast<size_t>(cs_ctas) * kp);
    NKG_CUDA(cudaMemcpyAsync(hs.data(), part_sum.get(), hs.size() * sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    NKG_CUDA(cudaMemcpyAsync(hk.data(), part_sink.get(), hk.size() * sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    NKG_CUDA(cudaStreamSynchronize(s));
    std::vector<double> factor(kp, 1.0);
    for (uint32_t c = 0; c < kp; ++c) {
        double sum = 0.0, sk = 0.0;
        for (uint32_t i = 0; i < cs_ctas; ++i) {
            sum += hs[static_cast<size_t>(i) * kp + c];
            sk += hk[static_cast<size_t>(i) * kp + c];
        }
        factor[c] = p.normalized ? (1.0 / static_cast<double>(n)) * ((1 - p.damp) + (p.damp * sk))
                                 : sum;
        if (!(factor[c] != 0.0))
            factor[c] = 1.0;
    }
    DeviceArray<double> d_factor(kp);
    NKG_CUDA(cudaMemcpyAsync(d_factor.get(), factor.data(), kp * sizeof(double),
                             cudaMemcpyHostToDevice, s));
    DeviceArray<float> dev_out;
    float *d_out = out;
    if (!out_on_device) {
        dev_out.alloc(static_cast<size_t>(k) * g->z);
        d_out = dev_out.get();
    }
    const size_t smem_out = 32 * (kp + 1) * sizeof(float);
    ppr_output<<<ceil_div(g->z, 32), 256, smem_out, s>>>(yfin, g->degc.get(), g->inv.get(), g->z,
                                                          n, k, kp, d_factor.get(), d_out);
    NKG_CUDA(cudaGetLastError());
    launches += 2;
    NKG_CUDA(cudaEventRecord(g->ev2, s));
    if (!out_on_device)
        NKG_CUDA(cudaMemcpyAsync(out, d_out, static_cast<size_t>(k) * g->z * sizeof(float),
                                 cudaMemcpyDeviceToHost, s));
    std::vector<unsigned long long> hit(kp);
    std::vector<double> hres(kp);
    NKG_CUDA(cudaMemcpyAsync(hit.data(), col_iter.get(), kp * sizeof(unsigned long long),
                             cudaMemcpyDeviceToHost, s));
    NKG_CUDA(cudaMemcpyAsync(hres.data(), col_res.get(), kp * sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    NKG_CUDA(cudaStreamSynchronize(s));
    if (iters_out)
        for (uint32_t j = 0; j < k; ++j)
            iters_out[j] = hit[j];
    if (stats) {
        clear_stats(stats);
        float ms = 0.f;
        NKG_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev2));
        stats->ms_total = ms;
        NKG_CUDA(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
        stats->ms_iterations = ms;
        stats->iterations = h.iteration;
        double worst = 0.0;
        for (uint32_t j = 0; j < k; ++j)
            worst = std::max(worst, hres[j]);
        stats->residual = worst;
        stats->kernel_launches = launches;
        stats->fp32_sweeps = h.iteration;
        // SpMM sweep, k columns: column ids, row offsets, degrees, and per
        // column the gathered, previous and new iterate.
        stats->bytes_per_sweep_fp32 = 4 * g->arcs + 4 * (g->n + 1) + 4 * g->n + 12ull * g->n * k;
        stats->bytes_per_sweep_fp64 = 0;
    }
}

} // namespace
} // namespace nkg

extern "C" int nkg_ppr_run(nkg_graph *g, const nkg_pr_params *p, uint32_t k, const uint32_t *seeds,
                           float *scores_out, int out_on_device, uint64_t *iterations_out,
                           nkg_stats *stats) {
    using namespace nkg;
    return guarded([&] {
        require(g != nullptr && p != nullptr && seeds != nullptr && scores_out != nullptr,
                "NULL argument");
        require(k >= 1 && k <= 256, "k must be in [1, 256]");
        require(!g->weighted, "batched personalised PageRank takes unweighted graphs");
        require(p->norm == NKG_NORM_L1 || p->norm == NKG_NORM_L2, "norm must be L1 or L2");
        require(std::isfinite(p->damp) && !std::isnan(p->tol), "damp/tol must be numbers");
        for (uint32_t j = 0; j < k; ++j)
            require(seeds[j] < g->z, "seed id out of range");
        DeviceGuard guard(g->device);
        RunScope scope(g);
        run_ppr(g, *p, k, seeds, scores_out, out_on_device != 0, iterations_out, stats);
    });
}
