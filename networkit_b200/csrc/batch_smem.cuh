// Many-graph batch: graphs whose iterate fits into one SM's shared memory.
//
// In batch_kernel (batch.cu) the iterate of a graph is gathered through L1, at
// about one request per clock and SM once several graphs share the SM (20M
// arcs in 96 graphs: 4.8 ms, 270 G gathers/s). A graph of up to 57,000 nodes
// (FP32; 28,500 in FP64) fits into shared memory, which serves random 4-byte
// gathers at 7 per clock and SM (8-byte: 4.6). Here every CTA of a cluster
// holds the whole iterate of the cluster's graph and computes a share of its
// rows; new values go to global memory, the cluster meets once per sweep, and
// every CTA copies the new iterate back (4 n bytes, coalesced, from L2).
//
// The arcs are kept as 16-bit node numbers local to the graph, eight to a
// 16-byte load. An item is what one warp does at a time: 32 rows with a lane
// each (rows of at most 32 arcs), or 4, 2 or 1 longer rows with 8, 16 or 32
// lanes each, lane s of a group of g taking arcs [8 (i g + s), + 8) of its row
// in step i. Absent arcs name the zero entry after the last node. Items are in
// order of falling length and go round the cluster's warps.
#pragma once

namespace nkg {
namespace {

constexpr int kSmemThreads = 1024;
constexpr uint32_t kSmemWarps = kSmemThreads / 32;
// Dynamic shared memory of a CTA: the 227 KB opt-in limit less the static part.
constexpr size_t kSmemBytes = 227 * 1024 - 4 * 1024;
// Largest graph (the iterate, its zero entry, rounding to 16 bytes).
template <typename T>
constexpr uint32_t smem_max_nodes() {
    return static_cast<uint32_t>(kSmemBytes / sizeof(T)) - 8;
}
// Shared memory of a launch whose largest graph has max_n nodes.
template <typename T>
constexpr size_t smem_launch_bytes(uint32_t max_n) {
    return (static_cast<size_t>(max_n) + 8) * sizeof(T) / 16 * 16 + 16;
}
// 16 CTAs, beyond the portable 8, for batches of few graphs: one of 20,000 nodes
// and 8M arcs, 60 sweeps, FP64 1.28 ms with 8, 0.71 with 16.
constexpr int kSmemMaxCluster = 16;

struct SmemMeta {
    uint32_t base;    // first (relabelled) node id
    uint32_t ybase;   // first entry of its iterate (a multiple of 4)
    uint32_t n;
    uint32_t item0, items;
    uint32_t sinks;
    uint32_t row[3];  // rows longer than 128, 64 and 32 arcs (prefixes)
    uint32_t arcs;
    uint32_t pad[2];
};

struct SmemItem {
    uint32_t off;     // first 512-byte step
    uint32_t steps;
    uint32_t row0;    // first row, local
    uint32_t lanes;   // lanes per row: 1, 8, 16 or 32
};

template <typename T>
struct SmemArgs {
    const SmemMeta *__restrict__ meta;
    const uint32_t *__restrict__ order;      // queue position -> graph
    const SmemItem *__restrict__ item;
    const uint4 *__restrict__ arcs;          // 32 lanes x 8 node numbers per step
    const uint32_t *__restrict__ degc;
    const uint32_t *__restrict__ perm;
    T *y0, *y1;                              // new iterates, even / odd sweeps
    double *out;
    unsigned long long *iterations;
    double *residual;
    unsigned long long *times;
    unsigned int *queue;
    unsigned int *floor_stops;
    const BatchParams *prm;
    uint32_t count;
};

struct SmemShared {
    double part[2][3];
    double s_red[3][kSmemWarps];
    double sumx, sink, res, sink_coef;
    uint32_t graph;
    int done;
};

template <typename T>
__device__ __forceinline__ T smem_step(const T *ys, uint4 w) {
    const T a0 = ys[w.x & 0xffffu], a1 = ys[w.x >> 16];
    const T a2 = ys[w.y & 0xffffu], a3 = ys[w.y >> 16];
    const T a4 = ys[w.z & 0xffffu], a5 = ys[w.z >> 16];
    const T a6 = ys[w.w & 0xffffu], a7 = ys[w.w >> 16];
    return ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
}

// 16-byte read that stays out of L1 (column streams; iterates other CTAs wrote).
__device__ __forceinline__ uint4 ld_cg_v4(const void *p) {
    return __ldcg(static_cast<const uint4 *>(p));
}

template <typename T>
__global__ void __launch_bounds__(kSmemThreads, 1) batch_smem_kernel(SmemArgs<T> a) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ SmemShared sh;
    T *ys = reinterpret_cast<T *>(s_dyn);
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned crank = cluster.block_rank(), csize = cluster.num_blocks();
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // Consecutive items go to different CTAs, so every CTA gets the same mix.
    const uint32_t cw = wid * csize + crank, nw = csize * kSmemWarps;
    const BatchParams prm = *a.prm;
    const T damp = static_cast<T>(prm.damp);
    constexpr uint32_t kVec = 16 / sizeof(T);

    for (;;) {
        if (crank == 0 && threadIdx.x == 0)
            sh.graph = atomicAdd(a.queue, 1u);
        cluster.sync();
        const uint32_t q = *cluster.map_shared_rank(&sh.graph, 0);
        if (q >= a.count) {
            cluster.sync();  // no CTA exits while another still reads its shared memory
            break;
        }
        const uint32_t gi = a.order[q];
        const SmemMeta m = a.meta[gi];
        if (crank == 0 && threadIdx.x == 0)
            a.times[2 * gi] = global_ns();
        const T tele = static_cast<T>((1.0 - prm.damp) / static_cast<double>(m.n));
        const T x0 = static_cast<T>(1.0 / static_cast<double>(m.n));
        for (uint32_t i = threadIdx.x; i < m.n; i += kSmemThreads) {
            const uint32_t dc = __ldg(a.degc + m.base + i);
            ys[i] = dc ? x0 / static_cast<T>(dc) : x0;
        }
        if (threadIdx.x == 0)
            ys[m.n] = T(0);
        T sink_coef = static_cast<T>(
            prm.distribute ? static_cast<double>(m.sinks) * (1.0 / static_cast<double>(m.n)) /
                                 static_cast<double>(m.n)
                           : 0.0);
        double res_prev = 0.0;
        unsigned long long it = 0;
        __syncthreads();
        for (;;) {
            T *yout = ((it & 1) ? a.y1 : a.y0) + m.ybase;
            double res = 0.0, sumx = 0.0, sink = 0.0;
            SmemItem x{};
            uint4 w{};
            if (cw < m.items) {
                x = a.item[m.item0 + cw];
                w = ld_cg_v4(a.arcs + static_cast<size_t>(x.off) * 32 + lane);
            }
            for (uint32_t k = cw; k < m.items;) {
                // The next item's head is loaded while this one is summed.
                const uint32_t kn = k + nw;
                SmemItem xn{};
                if (kn < m.items)
                    xn = a.item[m.item0 + kn];
                const uint4 *src = a.arcs + static_cast<size_t>(x.off) * 32 + lane;
                T acc = T(0);
                for (uint32_t i = 1; i < x.steps; ++i) {
                    const uint4 wn = ld_cg_v4(src + static_cast<size_t>(i) * 32);
                    acc += smem_step(ys, w);
                    w = wn;
                }
                uint4 wn{};
                if (kn < m.items)
                    wn = ld_cg_v4(a.arcs + static_cast<size_t>(xn.off) * 32 + lane);
                acc += smem_step(ys, w);
                for (uint32_t o = x.lanes >> 1; o > 0; o >>= 1)
                    acc += __shfl_xor_sync(0xffffffffu, acc, o);
                const uint32_t group = x.lanes == 1 ? lane : lane / x.lanes;
                const uint32_t i = x.row0 + group;
                // Rows of the item's class end with the class or the graph.
                const uint32_t end = x.lanes == 1 ? m.n : x.lanes == 8 ? m.row[2]
                                                      : x.lanes == 16  ? m.row[1]
                                                                       : m.row[0];
                if (i < end && (lane & (x.lanes - 1)) == 0) {
                    const uint32_t dc = __ldg(a.degc + m.base + i);
                    const T deg = static_cast<T>(dc);
                    if (prm.distribute)
                        acc = t_add(acc, sink_coef);
                    const T v = t_add(t_mul(acc, damp), tele);
                    const T yo = ys[i];
                    const T xo = dc ? t_mul(yo, deg) : yo;
                    const double d = static_cast<double>(xo) - static_cast<double>(v);
                    res += prm.l2 ? d * d : fabs(d);
                    sumx += static_cast<double>(v);
                    if (dc) {
                        yout[i] = v / deg;
                    } else {
                        yout[i] = v;
                        sink += static_cast<double>(v);
                    }
                }
                x = xn;
                w = wn;
                k = kn;
            }
            res = warp_sum(res);
            sumx = warp_sum(sumx);
            sink = warp_sum(sink);
            if (lane == 0) {
                sh.s_red[0][wid] = res;
                sh.s_red[1][wid] = sumx;
                sh.s_red[2][wid] = sink;
            }
            __syncthreads();
            const int slot = static_cast<int>(it & 1);
            if (wid == 0) {
                res = warp_sum(sh.s_red[0][lane]);
                sumx = warp_sum(sh.s_red[1][lane]);
                sink = warp_sum(sh.s_red[2][lane]);
                if (lane == 0) {
                    sh.part[slot][0] = res;
                    sh.part[slot][1] = sumx;
                    sh.part[slot][2] = sink;
                }
            }
            __threadfence();
            cluster.sync();
            // Every CTA adds the partials in the same order and takes the same
            // decision, while the new iterate is copied in.
            if (wid == 0) {
                double t[3] = {0.0, 0.0, 0.0};
                if (lane < csize) {
                    const double *pp = cluster.map_shared_rank(&sh.part[slot][0], lane);
                    t[0] = pp[0];
                    t[1] = pp[1];
                    t[2] = pp[2];
                }
                t[0] = warp_sum(t[0]);
                t[1] = warp_sum(t[1]);
                t[2] = warp_sum(t[2]);
                if (lane == 0) {
                    const double norm = prm.l2 ? sqrt(t[0]) : t[0];
                    const unsigned long long done_it = it + 1;
                    int done = (done_it >= prm.max_iterations || norm <= prm.tol) ? 1 : 0;
                    int at_floor = 0;
                    if (sizeof(T) == 4 && !done && it >= 1 && norm > 0.9 * res_prev) {
                        done = 1;
                        at_floor = 1;
                    }
                    sh.done = done;
                    sh.res = norm;
                    sh.sumx = t[1];
                    sh.sink = t[2];
                    sh.sink_coef = prm.distribute ? t[2] / static_cast<double>(m.n) : 0.0;
                    if (done && crank == 0) {
                        a.times[2 * gi + 1] = global_ns();
                        a.iterations[gi] = done_it;
                        a.residual[gi] = norm;
                        if (at_floor)
                            atomicAdd(a.floor_stops, 1u);
                    }
                }
            }
            const uint32_t vecs = (m.n + kVec - 1) / kVec;
            uint4 *dst = reinterpret_cast<uint4 *>(ys);
#pragma unroll 4
            for (uint32_t i = threadIdx.x; i < vecs; i += kSmemThreads)
                dst[i] = ld_cg_v4(reinterpret_cast<const uint4 *>(yout) + i);
            __syncthreads();
            // The copy rounds up to 16 bytes: put the zero entry back.
            if (threadIdx.x == 0)
                ys[m.n] = T(0);
            res_prev = sh.res;
            sink_coef = static_cast<T>(sh.sink_coef);
            ++it;
            const bool done = sh.done;
            __syncthreads();
            if (done)
                break;
        }
        // Scores of the final iterate (PageRank.cpp:75-92), in caller ids.
        const double factor =
            prm.normalized ? (1.0 / static_cast<double>(m.n)) * ((1.0 - prm.damp) + prm.damp * sh.sink)
                           : sh.sumx;
        for (uint32_t i = crank * kSmemThreads + threadIdx.x; i < m.n; i += csize * kSmemThreads) {
            const uint32_t dc = __ldg(a.degc + m.base + i);
            const T yv = ys[i];
            const double v = dc ? static_cast<double>(t_mul(yv, static_cast<T>(dc)))
                                : static_cast<double>(yv);
            a.out[__ldg(a.perm + m.base + i)] = v / factor;
        }
    }
}

// Rows longer than 128, 64 and 32 arcs of every graph, and its items (0 for
// graphs of more than max_n nodes).
__global__ void smem_count(SmemMeta *__restrict__ meta, uint32_t count, uint32_t max_n,
                           const uint32_t *__restrict__ rowlen) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= count)
        return;
    SmemMeta m = meta[g];
    m.items = 0;
    if (m.n <= max_n) {
        for (int c = 0; c < 3; ++c) {
            uint32_t lo = 0, hi = m.n;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (rowlen[m.base + mid] > (128u >> c))
                    lo = mid + 1;
                else
                    hi = mid;
            }
            m.row[c] = lo;
        }
        m.items = m.row[0] + (m.row[1] - m.row[0] + 1) / 2 + (m.row[2] - m.row[1] + 3) / 4 +
                  (m.n - m.row[2] + 31) / 32;
    }
    meta[g] = m;
}

// Row group and length of every item of a graph (one CTA per graph); `steps`
// receives the item's 512-byte steps.
__global__ void smem_items(const SmemMeta *__restrict__ meta, uint32_t count,
                           const uint32_t *__restrict__ rowlen, SmemItem *__restrict__ item,
                           uint32_t *__restrict__ steps, uint32_t *__restrict__ item_graph) {
    for (uint32_t g = blockIdx.x; g < count; g += gridDim.x) {
        const SmemMeta m = meta[g];
        const uint32_t i0 = m.row[0], i1 = i0 + (m.row[1] - m.row[0] + 1) / 2,
                       i2 = i1 + (m.row[2] - m.row[1] + 3) / 4;
        for (uint32_t k = threadIdx.x; k < m.items; k += blockDim.x) {
            SmemItem x;
            uint32_t end, rows;
            if (k < i0) {
                x.lanes = 32, rows = 1, x.row0 = k, end = m.row[0];
            } else if (k < i1) {
                x.lanes = 16, rows = 2, x.row0 = m.row[0] + 2 * (k - i0), end = m.row[1];
            } else if (k < i2) {
                x.lanes = 8, rows = 4, x.row0 = m.row[1] + 4 * (k - i1), end = m.row[2];
            } else {
                x.lanes = 1, rows = 32, x.row0 = m.row[2] + 32 * (k - i2), end = m.n;
            }
            uint32_t len = 0;
            for (uint32_t r = x.row0; r < min(end, x.row0 + rows); ++r)
                len = max(len, rowlen[m.base + r]);
            const uint32_t per = 8 * x.lanes;
            x.steps = max(1u, (len + per - 1) / per);
            x.off = 0;
            item[m.item0 + k] = x;
            steps[m.item0 + k] = x.steps;
            item_graph[m.item0 + k] = g;
        }
    }
}

// Offsets into the items and the arcs of every item (one warp per item).
__global__ void smem_fill(const SmemMeta *__restrict__ meta, const uint32_t *__restrict__ item_graph,
                          uint32_t items, const uint32_t *__restrict__ off,
                          const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ col,
                          SmemItem *__restrict__ item, uint4 *__restrict__ arcs) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t k = warp; k < items; k += nwarps) {
        const SmemMeta m = meta[item_graph[k]];
        SmemItem x = item[k];
        x.off = off[k];
        __syncwarp();
        if (lane == 0)
            item[k].off = x.off;
        const uint32_t group = lane / x.lanes, sub = lane & (x.lanes - 1);
        const uint32_t i = x.row0 + group;
        const uint32_t end = x.lanes == 1 ? m.n : x.lanes == 8 ? m.row[2]
                                              : x.lanes == 16  ? m.row[1]
                                                               : m.row[0];
        uint32_t b = 0, e = 0;
        if (i < end) {
            b = row_ptr[m.base + i];
            e = row_ptr[m.base + i + 1];
        }
        for (uint32_t s = 0; s < x.steps; ++s) {
            uint32_t v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t p = b + 8 * (s * x.lanes + sub) + 2 * j;
                const uint32_t lo = p < e ? col[p] - m.base : m.n;
                const uint32_t hi = p + 1 < e ? col[p + 1] - m.base : m.n;
                v[j] = lo | (hi << 16);
            }
            arcs[(static_cast<size_t>(x.off) + s) * 32 + lane] = make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
}

} // namespace
} // namespace nkg
