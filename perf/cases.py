"""Performance cases of the framework: the calls a user makes, over their range.

A case is a dict of plain values. `listed()` gives the fixed cases, `draw(rng)`
one more of the same ranges, `prepare` what a program holds before the call,
`run` one call through the public entry points, `work` the bytes and
operations the call cannot do without, `exact` the same outputs in 64-bit
torch, and `tolerance` how far two correct implementations may be apart.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from networkit_b200 import _capi, autograd, generators, graphio
from networkit_b200.graph import InCSR

DAMP = 0.85
RMAT = (0.57, 0.19, 0.19)
L1, L2 = 0, 1
PRECISION = {"fp64": _capi.NKG_PREC_FP64, "refine": _capi.NKG_PREC_FP32_REFINE,
             "fp32": _capi.NKG_PREC_FP32}


def listed():
    return [
        # A graph of wiki-Vote's size, scores back on the host with the class's
        # default tolerance: the smallest call, all latency.
        {"name": "small_host", "kind": "pagerank", "family": "rmat", "n": 7115, "deg": 16,
         "tol": 1e-8, "norm": L2, "sinks": False, "precision": "fp64", "weighted": False,
         "out": "host"},
        # G(1e5, average degree 10), sinks redistributed: the benchmark's plain
        # configuration.
        {"name": "er_1e5", "kind": "pagerank", "family": "er", "n": 100_000, "deg": 10,
         "tol": 1e-8, "norm": L2, "sinks": True, "precision": "fp64", "weighted": False,
         "out": "device"},
        # The headline run: directed R-MAT scale 24 to 1e-10 in FP64.
        {"name": "rmat24_fp64", "kind": "pagerank", "family": "rmat", "n": 1 << 24, "deg": 16,
         "tol": 1e-10, "norm": L1, "sinks": False, "precision": "fp64", "weighted": False,
         "out": "device"},
        # The same graph through the FP32 bulk solve with FP64 refinement.
        {"name": "rmat24_refine", "kind": "pagerank", "family": "rmat", "n": 1 << 24, "deg": 16,
         "tol": 1e-10, "norm": L1, "sinks": False, "precision": "refine", "weighted": False,
         "out": "device"},
        # Training step of the differentiable form on a weighted graph.
        {"name": "rmat22_grad", "kind": "grad", "family": "rmat", "n": 1 << 22, "deg": 16,
         "tol": 1e-10, "sinks": False, "precision": "refine"},
        # Batched personalised PageRank at the benchmark's size ...
        {"name": "ppr_ba4m_256", "kind": "ppr", "n": 4_000_000, "m": 8, "k": 256, "tol": 1e-7},
        # ... and an ordinary request: few seeds, ragged sizes.
        {"name": "ppr_ba300k_37", "kind": "ppr", "n": 300_001, "m": 5, "k": 37, "tol": 1e-7},
        # Many uneven geometric graphs in one launch.
        {"name": "batch_96", "kind": "batch", "count": 96, "low": 1000, "high": 50_000,
         "deg": 16, "tol": 1e-8},
        # One community per seed on a geometric graph (PageRankNibble).
        {"name": "nibble_2048", "kind": "local", "n": 200_000, "deg": 16, "seeds": 2048,
         "alpha": 0.1, "eps": 1e-5},
        # Eigenvector centrality and both Katz directions, scores on the host.
        {"name": "centralities", "kind": "centrality", "family": "rmat", "n": 2_000_003,
         "deg": 16},
        # End to end: a host CSR uploaded, solved, the scores back on the host.
        {"name": "upload_run_rmat22", "kind": "upload", "family": "rmat", "n": 3_800_017,
         "deg": 16, "tol": 1e-8, "norm": L1},
        # A NetworkitBinaryGraph file read from its path and ranked.
        {"name": "file_run", "kind": "file", "family": "rmat", "n": 1 << 20, "deg": 16,
         "chunks": 32, "tol": 1e-8, "norm": L2},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["pagerank", "pagerank", "pagerank", "grad", "ppr", "batch", "local",
                       "centrality", "upload", "file"])
    if kind == "pagerank":
        norm = rng.choice([L1, L2])
        return {"kind": kind, "family": rng.choice(["rmat", "rmat", "er", "ba"]),
                "n": _log_int(rng, 1000, 12_000_000), "deg": rng.randint(4, 20),
                "tol": 10.0 ** -rng.randint(6, 10), "norm": norm,
                "sinks": rng.random() < 0.5,
                "precision": rng.choice(["fp64", "fp64", "refine"]) if norm == L1 else "fp64",
                "weighted": rng.random() < 0.25, "out": rng.choice(["device", "host"])}
    if kind == "grad":
        return {"kind": kind, "family": rng.choice(["rmat", "er"]),
                "n": _log_int(rng, 2000, 3_000_000), "deg": rng.randint(4, 16), "tol": 1e-10,
                "sinks": rng.random() < 0.5, "precision": rng.choice(["refine", "fp64"])}
    if kind == "ppr":
        return {"kind": kind, "n": _log_int(rng, 5000, 2_000_000), "m": rng.randint(3, 10),
                "k": _log_int(rng, 1, 256), "tol": 1e-7}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 96), "low": 500,
                "high": _log_int(rng, 2000, 60_000), "deg": rng.randint(6, 20), "tol": 1e-8}
    if kind == "local":
        return {"kind": kind, "n": _log_int(rng, 20_000, 300_000), "deg": rng.randint(6, 20),
                "seeds": _log_int(rng, 1, 2048), "alpha": rng.choice([0.1, 0.15, 0.3]),
                "eps": rng.choice([1e-4, 1e-5])}
    if kind == "centrality":
        return {"kind": kind, "family": rng.choice(["rmat", "er"]),
                "n": _log_int(rng, 2000, 3_000_000), "deg": rng.randint(4, 16)}
    if kind == "upload":
        return {"kind": kind, "family": rng.choice(["rmat", "er"]),
                "n": _log_int(rng, 2000, 3_000_000), "deg": rng.randint(4, 16), "tol": 1e-8,
                "norm": L1}
    return {"kind": kind, "family": "rmat", "n": _log_int(rng, 5000, 1_000_000),
            "deg": rng.randint(4, 16), "chunks": rng.choice([1, 7, 32]), "tol": 1e-8,
            "norm": L2}


# ---------------------------------------------------------------------------
# Graphs, drawn on the GPU from a seed.


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _edges_rmat(n, deg, gen):
    """Directed R-MAT on n nodes (ids past n, duplicates, self-loops dropped)."""
    scale = max(1, math.ceil(math.log2(n)))
    m = n * deg
    a, b, c = RMAT
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=gen)
        src.mul_(2).add_(r >= a + b)
        dst.mul_(2).add_(((r >= a) & (r < a + b)) | (r >= a + b + c))
    del r
    keep = (src < n) & (dst < n) & (src != dst)
    key = torch.unique(src[keep] * n + dst[keep])
    return key // n, key % n


def _edges_er(n, deg, gen):
    m = n * deg // 2
    s = torch.randint(0, n, (m,), device="cuda", generator=gen)
    d = torch.randint(0, n, (m,), device="cuda", generator=gen)
    lo, hi = torch.minimum(s, d), torch.maximum(s, d)
    key = torch.unique((lo * n + hi)[lo != hi])
    return key // n, key % n


def _edges_ba(n, m, gen):
    """Preferential attachment: every edge's second end copies a random earlier
    end of the edge list (resolved by pointer jumping); duplicates dropped."""
    e = n * m
    pick = (torch.rand(e, device="cuda", generator=gen, dtype=torch.float64) *
            (2 * torch.arange(e, device="cuda") + 1)).to(torch.int64)
    at = pick.clone()
    while True:  # odd positions refer to an earlier edge's own pick
        odd = (at & 1) == 1
        if not bool(odd.any()):
            break
        at = torch.where(odd, pick[at >> 1], at)
    s = torch.arange(e, device="cuda") // m
    d = (at >> 1) // m
    lo, hi = torch.minimum(s, d), torch.maximum(s, d)
    key = torch.unique((lo * n + hi)[lo != hi])
    return key // n, key % n


def _edges(case, seed):
    """(src, dst, weights or None, directed) of the case's graph."""
    # A training step keeps its graph: there the seed draws the weights only.
    gen = _generator(7 if case["kind"] == "grad" else seed)
    family = case.get("family", "ba")
    if family == "rmat":
        s, d = _edges_rmat(case["n"], case["deg"], gen)
    elif family == "er":
        s, d = _edges_er(case["n"], case["deg"], gen)
    else:
        s, d = _edges_ba(case["n"], case.get("m", max(2, case.get("deg", 16) // 2)), gen)
    w = None
    if case.get("weighted") or case["kind"] == "grad":
        if case["kind"] == "grad":
            gen = _generator(seed)
        w = 1.0 - 0.9 * torch.rand(s.shape[0], device="cuda", dtype=torch.float64, generator=gen)
    return s, d, w, family == "rmat"


def _arcs(case, seed):
    """Arcs (source -> target) of the adjacency, both ways for undirected edges."""
    s, d, w, directed = _edges(case, seed)
    if directed:
        return s, d, w, True
    return (torch.cat([s, d]), torch.cat([d, s]), None if w is None else torch.cat([w, w]), False)


def _host_csr(case, seed):
    n = case["n"]
    s, d, w, directed = _arcs(case, seed)
    order = torch.argsort(d * n + s)
    counts = torch.bincount(d, minlength=n)
    in_ptr = np.zeros(n + 1, np.uint64)
    in_ptr[1:] = torch.cumsum(counts, 0).cpu().numpy().astype(np.uint64)
    in_col = s[order].to(torch.int32).cpu().numpy().view(np.uint32)
    outdeg = torch.bincount(s, minlength=n)
    in_w, wdeg = None, outdeg.to(torch.float64)
    if w is not None:
        in_w = w[order].cpu().numpy()
        wdeg = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, s, w)
    return InCSR(n, n, in_ptr, in_col, in_w, wdeg.cpu().numpy(),
                 outdeg.to(torch.int32).cpu().numpy().view(np.uint32), None, directed)


def _device_graph(case, seed):
    s, d, w, directed = _edges(case, seed)
    s32, d32 = s.to(torch.int32), d.to(torch.int32)
    m = s.shape[0]
    del s, d
    torch.cuda.synchronize()
    return _capi.DeviceGraph.from_device_edges(case["n"], m, s32.data_ptr(), d32.data_ptr(),
                                               0 if w is None else w.data_ptr(),
                                               directed=directed, device=0)


def _seeds(case, seed, n, k):
    return np.sort(np.random.default_rng(seed + 1).choice(n, k, replace=False))


def _batch_sizes(case):
    rng = np.random.default_rng(case["count"])
    return np.round(np.exp(rng.uniform(math.log(case["low"]), math.log(case["high"]),
                                       case["count"]))).astype(np.uint64)


# ---------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "pagerank":
        st["graph"] = _device_graph(case, seed)
        st["params"] = _capi.DeviceGraph.params(DAMP, case["tol"], case["norm"], False,
                                                case["sinks"], PRECISION[case["precision"]],
                                                _capi.UINT64_MAX)
        if case["out"] == "device":
            st["out"] = torch.empty(case["n"], dtype=torch.float64, device="cuda")
    elif kind == "grad":
        csr = _host_csr(case, seed)
        st["graph"] = autograd.DifferentiableGraph(csr, device=0)
        st["w"] = torch.from_numpy(csr.in_w).cuda().requires_grad_(True)
        t = torch.rand(case["n"], dtype=torch.float64, device="cuda", generator=_generator(seed + 2))
        st["t"] = (t / t.sum()).requires_grad_(True)
        st["g"] = torch.randn(case["n"], dtype=torch.float64, device="cuda",
                              generator=_generator(seed + 3))
    elif kind == "ppr":
        st["graph"] = _device_graph(case, seed)
        st["seeds"] = _seeds(case, seed, case["n"], case["k"]).astype(np.uint32)
        st["params"] = _capi.DeviceGraph.params(DAMP, case["tol"], L1, False, False,
                                                _capi.NKG_PREC_FP32, 1000)
        st["out"] = torch.empty((case["k"], case["n"]), dtype=torch.float32, device="cuda")
    elif kind == "batch":
        csr, offs = generators.hyperbolic_batch(_batch_sizes(case), float(case["deg"]), 3.0,
                                                seed=seed)
        st["batch"] = _capi.DeviceBatch(csr, offs, device=0)
        st["batch"].set_tuning(8, 256, 128)  # the shape the tuner picks on the benchmark's batch
        st["params"] = _capi.PRParams(DAMP, case["tol"], L1, 0, 0, _capi.NKG_PREC_FP32, 10000)
        st["out"] = torch.empty(int(offs[-1]), dtype=torch.float64, device="cuda")
    elif kind == "local":
        g = generators.hyperbolic(case["n"], float(case["deg"]), 3.0, seed=seed)
        st["local"] = _capi.DeviceLocal(g.z, g.in_ptr, g.in_col, None, None, False, device=0)
        st["seeds"] = _seeds(case, seed, case["n"], case["seeds"])
        st["max_pushes"] = int(1.0 / (case["alpha"] * case["eps"])) + 2000
        # the program's own result arrays, the same size whatever the seeds
        st["nodes"], st["members"] = (np.zeros(case["seeds"] * 8000, np.uint32) for _ in range(2))
        st["values"] = np.zeros(case["seeds"] * 8000)
    elif kind == "centrality":
        st["graph"] = _device_graph(case, seed)
    elif kind == "upload":
        csr = _host_csr(case, seed)
        # page-locked, as a program that uploads graph after graph keeps them
        csr.in_ptr = torch.from_numpy(csr.in_ptr.view(np.int64)).pin_memory().numpy().view(np.uint64)
        csr.in_col = torch.from_numpy(csr.in_col.view(np.int32)).pin_memory().numpy().view(np.uint32)
        st["csr"] = csr
        st["out"] = torch.empty(case["n"], dtype=torch.float64).pin_memory().numpy()
        st["params"] = _capi.DeviceGraph.params(DAMP, case["tol"], case["norm"], False, False,
                                                _capi.NKG_PREC_FP64, _capi.UINT64_MAX)
    else:
        csr = _host_csr(case, seed)
        out_ptr, out_col, _ = csr.out_csr()
        handle, path = tempfile.mkstemp(suffix=".nkbg")
        os.close(handle)
        graphio.write_nkbg(path, csr.z, out_ptr, out_col, None, csr.in_ptr, csr.in_col, None,
                           directed=True, chunks=case["chunks"])
        st["file"] = _File(path)
        st["params"] = _capi.DeviceGraph.params(DAMP, case["tol"], case["norm"], False, False,
                                                _capi.NKG_PREC_FP64, _capi.UINT64_MAX)
    return st


class _File:
    """A file that goes away with the state that holds it."""

    def __init__(self, path):
        self.path = path

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "pagerank":
        g, p = st["graph"], st["params"]
        if case["out"] == "device":
            g.run_device(p, st["out"].data_ptr())
            return st["out"]
        return g.run(p)[0]
    if kind == "grad":
        st["w"].grad = st["t"].grad = None
        s = autograd.pagerank(st["graph"], st["w"], st["t"], DAMP, case["tol"], case["sinks"],
                              "fp64" if case["precision"] == "fp64" else "fp32_refine")
        s.backward(st["g"])
        return s.detach(), st["w"].grad, st["t"].grad
    if kind == "ppr":
        st["graph"].ppr(st["seeds"], st["params"], st["out"].data_ptr())
        return st["out"]
    if kind == "batch":
        st["batch"].run(st["params"], st["out"].data_ptr())
        return st["out"]
    if kind == "local":
        sup, sets, _ = st["local"].run(st["seeds"], case["alpha"], case["eps"], nibble=True,
                                       max_pushes=st["max_pushes"])
        total, members = sum(len(s[0]) for s in sup), sum(len(s) for s in sets)
        np.concatenate([s[0] for s in sup], out=st["nodes"][:total])
        np.concatenate([s[1] for s in sup], out=st["values"][:total])
        np.concatenate(sets, out=st["members"][:members])
        return st["nodes"], st["values"], st["members"], np.array([len(s) for s in sets])
    if kind == "centrality":
        g = st["graph"]
        return (g.eigenvector(1e-9)[0], g.katz(0.0, 0.1, 1e-8, 0)[0], g.katz(0.0, 0.1, 1e-8, 1)[0])
    if kind == "upload":
        g = _capi.DeviceGraph(st["csr"], device=0)
        g.run(st["params"], out=st["out"])
        g.close()
        return st["out"]
    g = _capi.DeviceGraph.from_nkbg_file(st["file"].path, device=0)
    scores = g.run(st["params"])[0]
    g.close()
    return scores


# ---------------------------------------------------------------------------


def _arc_count(case):
    directed = case.get("family") == "rmat"
    return case["n"] * case["deg"] if case.get("family") in ("rmat", "er") else (
        2 * case["n"] * case.get("m", max(2, case.get("deg", 16) // 2)) if not directed else 0)


def _sweeps(case):
    """Power iterations to the tolerance, from the family's typical contraction."""
    if case["kind"] in ("pagerank", "grad") and case["precision"] == "refine":
        return 14  # Krylov steps of two half-width products: 14 FP64-equivalent sweeps
    rate = {"rmat": 0.8, "er": 0.5}.get(case.get("family", "ba"), 0.5)
    tol = case["tol"] * (math.sqrt(case["n"]) if case.get("norm", L1) == L2 else 1.0)
    return max(4, int(math.log(min(tol, 0.1)) / math.log(rate)))


def work(case):
    kind = case["kind"]
    if kind in ("pagerank", "upload", "file"):
        m, n, k = _arc_count(case), case["n"], _sweeps(case)
        per = (12 if case.get("weighted") else 4) * m + 32 * n
        extra = {"pagerank": 8 * n, "upload": 8 * m + 24 * n, "file": 16 * m + 24 * n}[kind]
        return {"bytes": float(k * per + extra), "flops": float(2 * k * m)}
    if kind == "grad":
        m, n, k = _arc_count(case), case["n"], _sweeps(case)
        # weights in, their gradient out, a forward and an adjoint solve
        return {"bytes": float(2 * k * (12 * m + 32 * n) + 40 * m), "flops": float(4 * k * m)}
    if kind == "ppr":
        m, n, k, s = 2 * case["n"] * case["m"], case["n"], case["k"], 23
        return {"bytes": float(s * (4 * m + 12 * n * k)), "flops": float(2 * s * m * k)}
    if kind == "batch":
        n = case["count"] * (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        m, s = n * case["deg"], 65
        return {"bytes": s * (4 * m + 20 * n), "flops": 2 * s * m}
    if kind == "local":
        # pushes of alpha * eps * volume each; about 90,000 arc visits a seed at 1e-5
        visits = case["seeds"] * 0.9 / case["eps"] * 0.1 / case["alpha"]
        return {"bytes": 24.0 * visits, "flops": 4.0 * visits}
    m, n = _arc_count(case), case["n"]
    return {"bytes": float(35 * (4 * m + 20 * n)), "flops": float(35 * 2 * m)}


def tolerance(case):
    kind = case["kind"]
    if kind == "local":
        return "exact"
    if kind == "grad" or case.get("precision") == "refine":
        return {"rel": 1e-8, "max": 1e-6}
    if kind in ("ppr", "batch"):
        return {"rel": 5e-6, "max": 2e-4}
    return {"rel": 1e-12, "max": 1e-10}


# ---------------------------------------------------------------------------
# The same outputs in 64-bit torch.


def _matrix(rows, cols, vals, n):
    order = torch.argsort(rows * n + cols)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return torch.sparse_csr_tensor(ptr, cols[order], vals[order], (n, n), check_invariants=False)


def _solve(A, sink, tele, x, damp, tol, l2, sinks):
    """Jacobi sweeps of PageRank to the stopping test; not normalised."""
    while True:
        y = A @ x
        if sinks:
            y = y + (x * sink).sum() * tele
        y = damp * y + (1.0 - damp) * tele
        d = y - x
        x = y
        if (d.norm() if l2 else d.abs().sum()) <= tol:
            return x


def _exact_pagerank(case, seed, tol, tele=None):
    n = case["n"]
    s, d, w, _ = _arcs(case, seed)
    if w is None:
        w = torch.ones(s.shape[0], dtype=torch.float64, device="cuda")
    wdeg = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, s, w)
    sink = (torch.bincount(s, minlength=n) == 0).to(torch.float64)
    A = _matrix(d, s, w / wdeg[s], n)
    x = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    if tele is None:
        tele = x
    x = _solve(A, sink, tele, x.clone(), DAMP, tol, case.get("norm", L1) == L2,
               case.get("sinks", False))
    return x, (s, d, w, wdeg, sink)


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "local":
        return None
    if kind in ("pagerank", "upload", "file"):
        # the refined solve returns the fixed point, the others the iterate at tol
        tol = 1e-14 if case.get("precision") == "refine" else case["tol"]
        x, _ = _exact_pagerank(case, seed, tol)
        return x / x.sum()
    if kind == "grad":
        t = torch.rand(n, dtype=torch.float64, device="cuda", generator=_generator(seed + 2))
        t = t / t.sum()
        g = torch.randn(n, dtype=torch.float64, device="cuda", generator=_generator(seed + 3))
        x, (s, d, w, wdeg, sink) = _exact_pagerank(case, seed, 1e-14, t)
        total, mass = x.sum(), (x * sink).sum()
        p = x / total
        rhs = (g - (g * p).sum()) / total
        B = _matrix(s, d, w / wdeg[s], n)
        lam = rhs.clone()
        for _ in range(400):
            c = B @ lam
            if case["sinks"]:
                c = c + sink * (t * lam).sum()
            new = rhs + DAMP * c
            done = (new - lam).abs().sum() <= 1e-13 * rhs.abs().sum()
            lam = new
            if done:
                break
        c = B @ lam
        order = torch.argsort(d * n + s)
        s, d = s[order], d[order]
        gw = DAMP * (x[s] / wdeg[s]) * (lam[d] - c[s])
        gt = ((DAMP * mass if case["sinks"] else 0.0) + 1.0 - DAMP) * lam
        return p, gw, gt
    if kind == "ppr":
        k = case["k"]
        s, d, _, _ = _arcs(case, seed)
        deg = torch.bincount(s, minlength=n).to(torch.float64)
        A = _matrix(d, s, 1.0 / deg[s], n)
        at = torch.from_numpy(_seeds(case, seed, n, k)).cuda()
        out = torch.empty((k, n), dtype=torch.float64, device="cuda")
        for j in range(0, k, 32):  # 32 columns at a time
            col = torch.arange(min(32, k - j), device="cuda")
            X = torch.full((n, col.shape[0]), 1.0 / n, dtype=torch.float64, device="cuda")
            for _ in range(200):
                Y = DAMP * (A @ X)
                Y[at[j:j + 32], col] += 1.0 - DAMP
                res = (Y - X).abs().sum(0).max()
                X = Y
                if res <= case["tol"]:
                    break
            out[j:j + 32] = (X / X.sum(0)).t()
        return out
    if kind == "batch":
        csr, offs = generators.hyperbolic_batch(_batch_sizes(case), float(case["deg"]), 3.0,
                                                seed=seed)
        z = int(offs[-1])
        ptr = torch.from_numpy(csr.in_ptr.view(np.int64)).cuda()
        col = torch.from_numpy(csr.in_col.astype(np.int64)).cuda()
        deg = torch.bincount(col, minlength=z).to(torch.float64)
        A = torch.sparse_csr_tensor(ptr, col, 1.0 / deg[col], (z, z), check_invariants=False)
        sizes = torch.from_numpy(np.diff(offs.astype(np.int64))).cuda()
        graph = torch.repeat_interleave(torch.arange(sizes.shape[0], device="cuda"), sizes)
        tele = 1.0 / sizes.to(torch.float64)[graph]
        x = tele.clone()
        for _ in range(150):  # far past the single-precision floor
            x = DAMP * (A @ x) + (1.0 - DAMP) * tele
        total = torch.zeros(sizes.shape[0], dtype=torch.float64, device="cuda")
        total.index_add_(0, graph, x)
        return x / total[graph]
    # centrality
    s, d, _, _ = _arcs(case, seed)
    one = torch.ones(s.shape[0], dtype=torch.float64, device="cuda")
    A, B = _matrix(d, s, one, n), _matrix(s, d, one, n)
    x, old = torch.ones(n, dtype=torch.float64, device="cuda"), 0.0
    while True:
        x = A @ x
        length = float(x.norm())
        x = x / length
        if abs(length - old) <= 1e-9:
            break
        old = length
    found = [x]
    alpha = 1.0 / (1.0 + float(torch.bincount(s, minlength=n).max()))
    for M in (A, B):
        x, old = torch.ones(n, dtype=torch.float64, device="cuda"), 0.0
        while True:
            x = alpha * (M @ (1.0 + x)) + 0.1
            length = float(x.norm())
            if abs(length - old) <= 1e-8:
                break
            old = length
        found.append(x / length)
    return tuple(found)
