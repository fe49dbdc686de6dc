// PageRank of a small unweighted graph in one persistent kernel.
//
// A sweep of a graph of a few million arcs is a few microseconds of gathers;
// as a kernel of its own it costs 13 to 16 us in the captured sweep graphs
// (launch gaps, the serial batches of a lane that sums a whole row or a
// 256-arc chunk, the last-CTA reduction), whatever the graph's size. Here the
// whole run - initial vector, sweeps, stopping test, normalisation, output in
// the caller's ids - is one cooperative launch whose CTAs meet at a grid
// barrier once per sweep.
//
// Rows are read from the relabelled in-CSR (sorted by in-degree, so rows
// longer than any power of two are a prefix). A row of more than kSmallHub
// arcs is summed by a whole CTA; a shorter one by 32, 16, ..., 1 lanes of a
// warp, so that a lane sums at most kSmallBatch arcs where rows have at most
// 256 (one batch of independent gathers; the chain of a sweep is then one
// column load, one gather and the shuffles). Task t of the rows, longest
// first, is warp t's in an interleaving that gives every SM the same share.
// The columns of a warp's first task stay in its registers for the whole run.
//
// Every CTA's residual and sink partials go to a slot per CTA; after the
// barrier every CTA adds all slots in the same order and takes the same
// decision, while its other warps already gather for the next sweep. Runs are
// bit-reproducible. Where the grid does not fit or the barrier gives up, the
// run is made by the captured sweeps instead.
#pragma once

#include "common.cuh"
#include "sweep.cuh"

namespace nkg {

constexpr int kSmallThreads = 1024;
constexpr uint32_t kSmallWarps = kSmallThreads / 32;
constexpr uint32_t kSmallBatch = 8;
constexpr uint32_t kSmallHub = 2048;
constexpr int kSmallClasses = 6;  // 32, 16, 8, 4, 2, 1 lanes per row
// Sweeps per launch: between launches the host looks for a cancellation.
constexpr uint32_t kSmallSweeps = 256;
// Polls of the grid barrier before it gives up (about two seconds).
constexpr uint32_t kSmallPolls = 1u << 22;

// Rows [row[0], row[1]) are the hubs' (row[0] = 0), rows [row[c + 1],
// row[c + 2]) class c's; class c has 2^c rows per warp task and the tasks
// [task[c], task[c + 1]).
struct SmallPlan {
    uint32_t row[kSmallClasses + 2];
    uint32_t task[kSmallClasses + 1];
};

// A hub is one CTA's work and the others wait for it, so graphs with longer rows
// than this stay with the captured sweeps, which cut them into chunks for all
// SMs: hub arcs of the CTA that has most, beyond half a CTA's share of all arcs
// (by which the captured sweeps are slower elsewhere). 40 FP64 sweeps of M arcs
// and one row of H more, one launch / captured, ms: M 0.3M, H 8k 0.40 / 0.69,
// 32k 0.59 / 0.69, 128k 1.38 / 0.78, 8M 65 / 2.5; M 4M, H 32k 1.60 / 1.71, 128k
// 3.56 / 1.79, 8M 164 / 4.1; M 12M, H 32k 3.05 / 3.85, 128k 5.06 / 3.94.
constexpr uint32_t kSmallHubArcs = 28672;

// Device state of a run, and what the host reads back.
struct SmallState {
    unsigned long long iteration;
    double residual, sink_mass, sink_coef, maximum;
    int done;
    int error;
    unsigned int barrier;
    unsigned int pad;
};

template <typename T>
struct SmallArgs {
    const uint32_t *row_ptr, *col, *degc, *inv;
    const T *tele;       // personalised teleport or null
    T *y0, *y1;          // gather-form iterate (sweep.cuh), even / odd sweeps
    double *part;        // 2 x 2 x CTAs (parity, residual / sink); 3 x CTAs at the end
    double *trace, *out;
    SmallState *st;
    RunParams rp;
    SmallPlan plan;
    uint64_t z;
    uint32_t n, trace_cap;
    uint32_t cap;        // sweeps of this launch
    uint32_t polls;      // of the grid barrier before it gives up
    int first, normalized;
    double coef0;        // sink term of the first sweep
};

// Coherent load: written by other SMs before the last grid barrier.
__device__ __forceinline__ double ld_y(const double *p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_y(const float *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// All CTAs of the launch arrive, then go on; the writes before it are visible
// after it. False once the wait ran out (every CTA then gives up the same way).
__device__ __forceinline__ bool small_barrier(SmallState *st, uint32_t polls, unsigned int &target,
                                              bool *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        __threadfence();
        atomicAdd(&st->barrier, 1u);
        unsigned int v = 0;
        for (uint32_t i = 0; v < target && i < polls; ++i)
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->barrier) : "memory");
        if (v < target)
            st->error = 1;
        *s_ok = v >= target;
        __threadfence();
    }
    __syncthreads();
    return *s_ok;
}

// Row epilogue: finish_row of sweep.cuh with coherent loads of the iterate.
template <typename T>
__device__ __forceinline__ void small_row(const SmallArgs<T> &a, const T *y_in, T *y_out,
                                          T sink_coef, uint32_t r, uint32_t dc, T acc,
                                          double &res, double &sink) {
    const RunParams &rp = a.rp;
    const T yo = ld_y(y_in + r);
    if (rp.distribute)
        acc = t_add(acc, rp.personal ? t_mul(sink_coef, a.tele[r]) : sink_coef);
    T x = t_mul(acc, static_cast<T>(rp.damp));
    x = t_add(x, rp.personal ? t_mul(static_cast<T>(rp.one_minus_damp), a.tele[r])
                             : static_cast<T>(rp.tele_uniform));
    const T deg = static_cast<T>(dc);
    const T xo = dc == 0 ? yo : t_mul(yo, deg);
    const double d = static_cast<double>(xo) - static_cast<double>(x);
    res += rp.l2 ? __dmul_rn(d, d) : fabs(d);
    if (dc == 0) {
        sink += static_cast<double>(x);
        y_out[r] = x;
    } else {
        y_out[r] = x / deg;
    }
}

// Sum of y over the arcs b + first, + step, ... below e, in batches of
// independent gathers (absent arcs add nothing).
template <typename T>
__device__ __forceinline__ T small_sum(const uint32_t *col, const T *y, uint32_t k, uint32_t e,
                                       uint32_t step) {
    T acc = T(0);
    while (k < e) {
        uint32_t c[kSmallBatch];
#pragma unroll
        for (uint32_t i = 0; i < kSmallBatch; ++i)
            c[i] = k + i * step < e ? __ldg(col + k + i * step) : kNone;
        T v[kSmallBatch];
#pragma unroll
        for (uint32_t i = 0; i < kSmallBatch; ++i)
            v[i] = c[i] != kNone ? ld_y(y + c[i]) : T(0);
#pragma unroll
        for (uint32_t i = 0; i < kSmallBatch; ++i)
            acc += v[i];
        if (e - k <= kSmallBatch * step)
            break;
        k += kSmallBatch * step;
    }
    return acc;
}

// Row, lane within the row's group and group width of task t's lane.
struct SmallTask {
    uint32_t row, sub, lanes;
    bool valid;
};
__device__ __forceinline__ SmallTask small_task(const SmallPlan &p, uint32_t t, uint32_t lane) {
    int c = 0;
#pragma unroll
    for (int i = 1; i < kSmallClasses; ++i)
        c += t >= p.task[i];
    SmallTask k;
    k.lanes = 32u >> c;
    uint32_t base = p.row[1], end = p.row[2], t0 = p.task[0];
#pragma unroll
    for (int i = 1; i < kSmallClasses; ++i)
        if (c == i) {
            base = p.row[i + 1];
            end = p.row[i + 2];
            t0 = p.task[i];
        }
    k.row = base + ((t - t0) << c) + (lane >> (5 - c));
    k.sub = lane & (k.lanes - 1);
    k.valid = k.row < end;
    return k;
}

template <typename T>
__device__ __forceinline__ T group_sum(T v, uint32_t lanes) {
    for (uint32_t o = 16; o > 0; o >>= 1) {
        const T w = __shfl_down_sync(0xffffffffu, v, o);
        if (o < lanes)
            v += w;
    }
    return v;
}

template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 1) small_kernel(SmallArgs<T> a) {
    __shared__ double s_red[3][kSmallWarps];
    __shared__ double s_coef;
    __shared__ int s_done;
    __shared__ bool s_ok;
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t nctas = gridDim.x;
    const uint32_t tasks = a.plan.task[kSmallClasses], nw = nctas * kSmallWarps;
    const uint32_t t0 = wid * nctas + blockIdx.x;
    const uint64_t gid = blockIdx.x * static_cast<uint64_t>(kSmallThreads) + threadIdx.x;
    const uint64_t gsize = static_cast<uint64_t>(nctas) * kSmallThreads;
    unsigned int target = 0;  // barrier arrivals that end the next wait (thread 0)

    // The warp's first task: row bounds, degree and first columns for good.
    SmallTask k0{0, 0, 32, false};
    uint32_t b0 = 0, e0 = 0, dc0 = 0, c0[kSmallBatch];
    if (t0 < tasks) {
        k0 = small_task(a.plan, t0, lane);
        if (k0.valid) {
            b0 = a.row_ptr[k0.row];
            e0 = a.row_ptr[k0.row + 1];
            dc0 = a.degc[k0.row];
        }
    }
    const uint32_t f0 = b0 + k0.sub;
#pragma unroll
    for (uint32_t i = 0; i < kSmallBatch; ++i)
        c0[i] = f0 + i * k0.lanes < e0 ? a.col[f0 + i * k0.lanes] : kNone;

    unsigned long long it = a.st->iteration;
    if (threadIdx.x == 0) {
        s_coef = a.first ? a.coef0 : a.st->sink_coef;
        s_done = 0;
    }
    if (a.first) {
        const T x0 = static_cast<T>(a.rp.inv_n);
        for (uint64_t r = gid; r < a.n; r += gsize) {
            const uint32_t dc = a.degc[r];
            a.y0[r] = dc == 0 ? x0 : x0 / static_cast<T>(dc);
        }
        if (!small_barrier(a.st, a.polls, target, &s_ok))
            return;
    } else {
        __syncthreads();
    }

    double norm = 0.0, mass = 0.0;
    for (uint32_t k = 0;; ++k) {
        const T *y_in = (it & 1) ? a.y1 : a.y0;
        T *y_out = (it & 1) ? a.y0 : a.y1;
        // First task's gathers (thrown away when the run is over).
        T acc0 = T(0);
        if (t0 < tasks) {
            T v[kSmallBatch];
#pragma unroll
            for (uint32_t i = 0; i < kSmallBatch; ++i)
                v[i] = c0[i] != kNone ? ld_y(y_in + c0[i]) : T(0);
#pragma unroll
            for (uint32_t i = 0; i < kSmallBatch; ++i)
                acc0 += v[i];
            acc0 += small_sum(a.col, y_in, f0 + kSmallBatch * k0.lanes, e0, k0.lanes);
            acc0 = group_sum(acc0, k0.lanes);
        }
        // The stopping test of the sweep before this one (close_iteration).
        if (k > 0 && wid == 0) {
            const double *pr = a.part + (k & 1) * 2 * nctas;
            double r = 0.0, s = 0.0;
            for (uint32_t i = lane; i < nctas; i += 32) {
                r += __ldcg(pr + i);
                s += __ldcg(pr + nctas + i);
            }
            r = warp_sum(r);
            s = warp_sum(s);
            if (lane == 0) {
                norm = a.rp.l2 ? sqrt(r) : r;
                mass = s;
                s_coef = a.rp.distribute
                             ? (a.rp.personal ? s : s / static_cast<double>(a.n)) : 0.0;
                s_done = it >= a.rp.max_iterations || norm <= a.rp.tol;
                if (blockIdx.x == 0 && it - 1 < a.trace_cap)
                    a.trace[it - 1] = norm;
            }
        }
        __syncthreads();
        if (k > 0 && (s_done || k == a.cap))
            break;
        const T coef = static_cast<T>(s_coef);
        double res = 0.0, sink = 0.0;
        if (k0.valid && k0.sub == 0)
            small_row(a, y_in, y_out, coef, k0.row, dc0, acc0, res, sink);
        for (uint32_t t = t0 + nw; t < tasks; t += nw) {
            const SmallTask q = small_task(a.plan, t, lane);
            uint32_t b = 0, e = 0;
            if (q.valid) {
                b = __ldg(a.row_ptr + q.row);
                e = __ldg(a.row_ptr + q.row + 1);
            }
            T acc = small_sum(a.col, y_in, b + q.sub, e, q.lanes);
            acc = group_sum(acc, q.lanes);
            if (q.valid && q.sub == 0)
                small_row(a, y_in, y_out, coef, q.row, __ldg(a.degc + q.row), acc, res, sink);
        }
        for (uint32_t h = blockIdx.x; h < a.plan.row[1]; h += nctas) {
            const uint32_t b = __ldg(a.row_ptr + h), e = __ldg(a.row_ptr + h + 1);
            const double p = warp_sum(static_cast<double>(
                small_sum(a.col, y_in, b + threadIdx.x, e, static_cast<uint32_t>(kSmallThreads))));
            if (lane == 0)
                s_red[2][wid] = p;
            __syncthreads();
            if (wid == 0) {
                const double tot = warp_sum(s_red[2][lane]);
                if (lane == 0)
                    small_row(a, y_in, y_out, coef, h, __ldg(a.degc + h), static_cast<T>(tot), res,
                              sink);
            }
            __syncthreads();
        }
        res = warp_sum(res);
        sink = warp_sum(sink);
        if (lane == 0) {
            s_red[0][wid] = res;
            s_red[1][wid] = sink;
        }
        __syncthreads();
        if (wid == 0) {
            const double r = warp_sum(s_red[0][lane]);
            const double s = warp_sum(s_red[1][lane]);
            if (lane == 0) {
                double *pw = a.part + ((k + 1) & 1) * 2 * nctas;
                pw[blockIdx.x] = r;
                pw[nctas + blockIdx.x] = s;
            }
        }
        ++it;
        if (!small_barrier(a.st, a.polls, target, &s_ok))
            return;
    }
    if (gid == 0) {
        a.st->iteration = it;
        a.st->residual = norm;
        a.st->sink_mass = mass;
        a.st->sink_coef = s_coef;
        a.st->done = s_done;
    }
    if (!s_done)
        return;

    // PageRank.cpp:75-102: normalisation and maximum (final_reduce, final_scale).
    const T *y = (it & 1) ? a.y1 : a.y0;
    double s = 0.0, ss = 0.0, mx = -1.0 / 0.0;
    for (uint64_t r = gid; r < a.n; r += gsize) {
        const uint32_t dc = __ldg(a.degc + r);
        const T yv = ld_y(y + r);
        const double x = static_cast<double>(dc ? t_mul(yv, static_cast<T>(dc)) : yv);
        s += x;
        if (dc == 0)
            ss += x;
        mx = fmax(mx, x);
    }
    s = warp_sum(s);
    ss = warp_sum(ss);
    mx = warp_max(mx);
    if (lane == 0) {
        s_red[0][wid] = s;
        s_red[1][wid] = ss;
        s_red[2][wid] = mx;
    }
    __syncthreads();
    double *pf = a.part + 4 * static_cast<size_t>(nctas);
    if (wid == 0) {
        s = warp_sum(s_red[0][lane]);
        ss = warp_sum(s_red[1][lane]);
        mx = warp_max(s_red[2][lane]);
        if (lane == 0) {
            pf[blockIdx.x] = s;
            pf[nctas + blockIdx.x] = ss;
            pf[2 * nctas + blockIdx.x] = mx;
        }
    }
    if (!small_barrier(a.st, a.polls, target, &s_ok))
        return;
    if (wid == 0) {
        s = ss = 0.0;
        mx = -1.0 / 0.0;
        for (uint32_t i = lane; i < nctas; i += 32) {
            s += __ldcg(pf + i);
            ss += __ldcg(pf + nctas + i);
            mx = fmax(mx, __ldcg(pf + 2 * nctas + i));
        }
        s = warp_sum(s);
        ss = warp_sum(ss);
        mx = warp_max(mx);
        if (lane == 0) {
            const double n = static_cast<double>(a.n);
            s_red[0][0] = a.normalized ? (1.0 / n) * ((1 - a.rp.damp) + (a.rp.damp * ss)) : s;
            s_red[1][0] = mx;
        }
    }
    __syncthreads();
    const double factor = s_red[0][0];
    for (uint64_t o = gid; o < a.z; o += gsize) {
        const uint32_t r = __ldg(a.inv + o);
        double v = 1.0 / static_cast<double>(a.n);
        if (r != kNone) {
            const uint32_t dc = __ldg(a.degc + r);
            const T yv = ld_y(y + r);
            v = static_cast<double>(dc ? t_mul(yv, static_cast<T>(dc)) : yv) / factor;
        }
        a.out[o] = v;
        if (o == 0)
            a.st->maximum = a.normalized ? fmax(v, s_red[1][0] / factor) : 1.0;
    }
}

} // namespace nkg
