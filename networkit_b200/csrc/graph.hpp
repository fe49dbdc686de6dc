// Device-resident graph handle (the opaque nkg_graph of nkgpu.h).
#pragma once

#include <atomic>
#include <memory>

#include "common.cuh"
#include "hot.cuh"
#include "small.cuh"
#include "sweep.cuh"

namespace nkg {

// Sweeps per captured CUDA graph (even, so every graph starts on buffer 0).
constexpr int kSweepsPerGraph = 8;
// Work units per resident warp of the sweep kernel.
constexpr uint32_t kUnitsPerWarp = 8;
// Work units per resident warp of the queued PageRank sweep. Measured on
// R-MAT scale 24 (FP64 sweep, B200): 4 / 8 / 12 / 16 / 24 / 32 / 64 units per
// warp ran 0.941 / 0.880 / 0.876 / 0.875 / 0.889 / 0.900 / 0.975 ms, against
// 0.956 ms for 8 static units per warp. Fewer units leave a longer tail;
// more units pay the ticket round trip and a cold start more often.
constexpr uint32_t kQueueUnitsPerWarp = 16;
// Cost of a slice in units of one slot step, besides its length (the
// epilogue of its 32 rows).
constexpr uint32_t kSliceOverhead = 3;

// Work buffers of the FP32 refinement solve, kept between runs.
struct RefineWork {
    DeviceArray<float> x, r, rhat, p, v, s, t, g;  // g: n+1 (gather form, g[n] = 0)
    DeviceArray<double> x64, part, fix_part;
    DeviceArray<double> unit_part;                  // queued product: 2 per unit
    DeviceArray<unsigned char> sc;                  // BiScalars
};

// Buffers of the one-launch run of a small graph (small.cuh), kept between runs.
struct SmallWork {
    SmallPlan plan{};
    unsigned ctas = 0;     // 0: not set up
    bool declined = false; // this graph's runs are captured sweeps
    uint32_t polls = kSmallPolls;
    unsigned test_ctas = 0;  // nkg_test_small_run: CTAs whatever the graph's rows are
    DeviceArray<double> y0, y1, part;
    DeviceArray<SmallState> st;
    PinnedHost<SmallState> host;
};

// Sliced layout (SELL-32 with chunked long rows, see sweep.cuh) of one
// adjacency: the in-adjacency for the forward sweeps, the out-adjacency for
// the adjoint.
struct SellLayout {
    uint32_t chunk = kChunk;            // arcs per chunk of a split row (chunk_for)
    uint32_t n_long = 0, n_vlong = 0, n_chunks = 0, s_chunk = 0, slices = 0;
    uint64_t slots = 0;
    DeviceArray<uint32_t> chunk_begin;  // n_long+1
    DeviceArray<uint32_t> slice_off;    // slices+1
    DeviceArray<uint64_t> slice_cost;   // slices, inclusive prefix of slice costs
    DeviceArray<uint32_t> col_sell;     // slots
    DeviceArray<double> w_sell64;       // slots (weighted)
    // Source blocks (hot.cuh; unweighted in-adjacency of large graphs): rows
    // [0, n_hot) have segments, whose sums are chunk sums of the row (its
    // first chunk sums, chunk_begin has n_hot + 1 entries); the chunks of the
    // slices above are then of the other arcs, stored chunk i's sum going to
    // chunk_slot[i] (s_chunk * 32 entries; empty: i).
    uint32_t n_hot = 0, n_sums = 0;
    DeviceArray<uint32_t> chunk_slot;
    HotBlocks hot_blocks{};
    uint32_t hot_slices = 0;
    uint64_t hot_steps = 0;
    uint64_t hot_n = 0, hot_sums = 0;   // arcs of the segments, sums of their chunks
    DeviceArray<uint4> hot_arcs;        // 32 lanes x 8 arcs per step
    DeviceArray<uint32_t> hot_off;      // hot_slices + 1
    DeviceArray<uint32_t> hot_slot;     // 32 per slice
    DeviceArray<uint64_t> hot_cost;     // hot_slices each for FP64 and FP32, inclusive prefixes
    // Entries of a chunk-sum buffer.
    size_t chunk_sums() const { return std::max<size_t>(static_cast<size_t>(s_chunk) * 32, n_sums); }
};

// The launches of hot_kernel over one layout in one precision; launch() does
// nothing (and returns 0) where the layout has no blocks.
template <typename T>
struct HotRun {
    unsigned ctas = 0;
    DeviceArray<uint32_t> cta_start;
    void setup(const SellLayout &L, unsigned sms, cudaStream_t s);
    template <int MODE = 0>
    unsigned launch(const SellLayout &L, const T *y, T *sums, uint32_t n, T pad, T alpha,
                    const int *skip, cudaStream_t s) const {
        if (!ctas)
            return 0;
        HotArgs<T> a{};
        a.arcs = L.hot_arcs.get();
        a.off = L.hot_off.get();
        a.slot = L.hot_slot.get();
        a.cta_start = cta_start.get();
        a.y = y;
        a.sums = sums;
        a.skip = skip;
        a.blocks = L.hot_blocks;
        a.n = n;
        a.pad = pad;
        a.alpha = alpha;
        NKG_CUDA(cudaFuncSetAttribute(hot_kernel<T, MODE>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(hot_bytes<T>())));
        hot_kernel<T, MODE><<<ctas, kHotKernelThreads, hot_bytes<T>(), s>>>(a);
        return 1;
    }
};

// Rows of more than `chunk` arcs (kChunk or kSmallChunk) cut into chunks of that
// many in CSR order: their number, those of more than kShortChunks chunks, the
// first chunk of each (n_long + 1 entries). Returns the number of chunks. Where
// kSmallChunk would split most rows just past their end (rows of 9/8 to 3/2 of it
// on average, at most kChunk) and the rows alone give 5/6 of the resident lanes a
// row each, chunk becomes kChunk: the fix-up of those rows then costs more than
// the shorter lanes save. 40 FP64 iterations, ids in order, split / whole, ms: 80
// arcs a row 200,000 rows 1.85 / 1.58, 400,000 2.91 / 2.42, 175,000 1.60 / 1.69,
// 25,000 0.77 / 0.95; 66 arcs, 250,000 rows 1.67 / 1.77; 120 arcs, 200,000 rows
// 2.05 / 1.95 (FP32 1.56 / 1.69); 160 arcs 2.38 / 2.53.
uint32_t row_chunks(const uint32_t *rowlen, uint32_t n, uint64_t arcs, unsigned sms,
                    uint32_t &chunk, uint32_t &n_long, uint32_t &n_vlong,
                    DeviceArray<uint32_t> &chunk_begin, cudaStream_t s);

// Build the sliced layout of a CSR whose n rows are sorted by length,
// descending; the weight of entry k is w[w_index[k]] (w[k] without an index,
// no weights when w is null). Padding slots hold pad_col (kNone: n, the zero
// entry of an iterate of n + 1). `blocks`: unweighted, columns numbered as the
// rows are; the layout may get source blocks. `scratch`: an array of `arcs`
// entries that is no longer needed, or null.
void build_sell(SellLayout &L, uint32_t n, uint64_t arcs, const uint32_t *row_ptr,
                const uint32_t *col, const double *w, const uint32_t *w_index, const uint32_t *rowlen, int device,
                cudaStream_t s, uint32_t pad_col = kNone, bool blocks = false,
                DeviceArray<uint32_t> *scratch = nullptr);
// map[slot] = index[k] for the CSR entry k each slot of L holds (kNone for
// padding slots).
void build_slot_map(const SellLayout &L, uint32_t n, const uint32_t *row_ptr, const uint32_t *index,
                    uint32_t *map, int device, cudaStream_t s);
// Cost-balanced unit boundaries over the slices of L (units+1 entries).
void sell_units(const SellLayout &L, uint32_t units, uint32_t *unit_start, cudaStream_t s);
void convert_to_float(const double *in, float *out, uint64_t m, int device, cudaStream_t s);

struct AdjointState;
void destroy_adjoint(AdjointState *a);
struct AdjointDeleter {
    void operator()(AdjointState *a) const { destroy_adjoint(a); }
};

// Per-precision work buffers and the captured sweep graph.
template <typename T>
struct Plane {
    DeviceArray<T> y[2];         // ping-pong iterate in gather form (n+1, y[n] = 0)
    DeviceArray<T> chunk_val;    // per chunk slot
    DeviceArray<T> w_sell;       // slot weights in this precision (weighted)
    DeviceArray<T> degw;         // weighted degree in this precision (weighted)
    DeviceArray<T> tele;         // personalised teleport, relabelled
    DeviceArray<uint32_t> unit_start;
    uint32_t units = 0;
    cudaGraphExec_t exec[2] = {nullptr, nullptr};  // [personal]
    unsigned sweep_ctas = 0;
    unsigned fix_ctas = 0;
    uint32_t hot = 0;            // ids in the shared-memory tier (0: none)
    // The tier kernel's own grid and work units; the fields above stay those
    // of the regular shape, which the FP32 product of the refinement solve
    // also uses.
    DeviceArray<uint32_t> hot_unit_start;
    uint32_t hot_units = 0;
    unsigned hot_ctas = 0;
    int hot_threads = 0;         // kHotThreads or kHotThreadsPair
    // Queued sweep (warps take units from a device counter): its units and
    // their residual / sink partials (2 x q_units). q_units 0: the static
    // assignment of unit_start (the shared-memory tier).
    DeviceArray<uint32_t> q_unit_start;
    DeviceArray<double> q_part;
    uint32_t q_units = 0;
    bool ready = false;          // sweep_setup is done
    HotRun<T> hot_run;           // source blocks (hot.cuh), before every sweep
    // The sweep's last CTA closes each iteration (no fix-up launch): graphs
    // with no split rows and at most kCloseInSweepUnits units.
    bool close_in_sweep = false;
};

} // namespace nkg

struct nkg_graph {
    nkg_graph() = default;
    nkg_graph(const nkg_graph &) = delete;
    nkg_graph &operator=(const nkg_graph &) = delete;
    ~nkg_graph();
    int device = 0;
    cudaStream_t stream = nullptr;
    uint64_t z = 0, n = 0, arcs = 0, sinks = 0;
    bool weighted = false, directed = false;
    double ms_create = 0.0;
    int row_order = 0;  // relabelling used: 0 in-degree, 1 in-degree buckets

    nkg::DeviceArray<uint32_t> perm;     // new id -> original id (n)
    nkg::DeviceArray<uint32_t> inv;      // original id -> new id (z), kNone if absent
    nkg::DeviceArray<uint32_t> row_ptr;  // n+1, in-CSR in new ids
    nkg::DeviceArray<uint32_t> col;      // arcs
    nkg::DeviceArray<uint32_t> degc;     // out-degree count (n)
    nkg::DeviceArray<double> w64src;     // CSR arc weights (FP64, relabelled order)
    nkg::DeviceArray<double> degw64src;  // weighted degree (FP64)

    nkg::DeviceArray<uint64_t> row_src; // n: offset of new row r in the caller's in-CSR

    // Sliced layout of the sweep (the in-adjacency).
    nkg::SellLayout fw;
    // Chunks of the long rows in CSR order for the sweeps that read the CSR
    // (personalised PageRank), built on first use.
    uint32_t rc_long = 0, rc_chunks = 0;
    nkg::DeviceArray<uint32_t> rc_begin;
    int sweep_shape = 0;
    bool arc_sorted = false;
    bool w64src_stale = false;  // w64src predates nkg_graph_set_weights

    // Out-adjacency layout and buffers of the adjoint (built on first use).
    std::unique_ptr<nkg::AdjointState, nkg::AdjointDeleter> adj;

    nkg::Plane<double> p64;
    nkg::Plane<float> p32;
    nkg::RefineWork refine_work;

    nkg::DeviceArray<double> cta_res, cta_sink, fix_res, fix_sink;
    nkg::DeviceArray<double> out_buf;    // scores staging for host output (z)
    nkg::DeviceArray<double> red;        // scratch for finalisation reductions
    nkg::DeviceArray<unsigned int> red_ticket;
    nkg::DeviceArray<nkg::RunParams> rp;
    nkg::DeviceArray<nkg::IterState> st;
    nkg::PinnedHost<nkg::IterState> st_host;
    nkg::PinnedHost<double> scalars_host;

    nkg::DeviceArray<double> trace;      // residual of sweep i at [i] (kTraceCapacity)
    int hot_tier_kb = -1;                // nkg_graph_options.hot_tier_kb
    nkg::SmallWork small;

    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr;
    std::atomic<int> cancel{0};
    bool has_run = false;
};

namespace nkg {
// Cancellation (nkg_cancel): a request stays set until a run on the handle
// ends, so one issued just before a run starts stops that run. Every run
// holds a RunScope, which clears the request when the run ends (normally or
// by an error); the checks between chunks of sweeps only read it.
struct RunScope {
    nkg_graph *g;
    explicit RunScope(nkg_graph *h) : g(h) {}
    RunScope(const RunScope &) = delete;
    RunScope &operator=(const RunScope &) = delete;
    ~RunScope() { g->cancel.store(0); }
};
inline void check_cancel(const nkg_graph *g, const char *what) {
    if (g->cancel.load())
        throw Error(NKG_ERR_CANCELLED, what);
}

// A graph from an in-CSR already in device memory (nkgpu.cu): the shell on the
// options' device (its stream is the one to build on), then the regular upload
// steps from the device arrays (host copy of the existence mask, nullable).
std::unique_ptr<nkg_graph> device_graph_shell(const nkg_graph_options *opt, uint64_t z,
                                              bool weighted, int directed);
nkg_graph *device_graph_build(std::unique_ptr<nkg_graph> g, uint64_t arcs,
                              DeviceArray<uint64_t> &d_ptr, DeviceArray<uint32_t> &d_col,
                              DeviceArray<double> &d_w, DeviceArray<double> &d_wdeg,
                              DeviceArray<uint8_t> &d_ex, const uint8_t *exists_host,
                              const nkg_graph_options *opt);

// Most sweeps whose residual a run records for nkg_stats.residual_trace.
constexpr uint32_t kTraceCapacity = 65536;

// The out-adjacency layout of the adjoint (adjoint.cu), built on first use.
AdjointState &adjoint_ensure(nkg_graph *g);
// Read-only view of that layout for other kernels: rows are the nodes in
// out-degree order (tinv: relabelled id -> row), columns row numbers.
struct OutLayoutView {
    const SellLayout *tl;
    const uint32_t *tinv;
};
OutLayoutView adjoint_out_layout(nkg_graph *g);
// Replace the arc weights in place (device arrays in the caller's order;
// wdeg null: summed on the device over every node's out-arcs).
void set_weights_device(nkg_graph *g, const double *w, const double *wdeg);
} // namespace nkg
