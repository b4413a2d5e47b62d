"""Cases for timing the engine through its public Python and C entry points.

A case is a dict of plain values; `listed()` gives the standing set, `draw()`
one more case of the same ranges.  `prepare(case, seed)` makes what a program
has before the call (a CSR in device memory, a host CSR, the entries of a
matrix file, an engine handle), `run(state)` is the call itself.

Graph families (the ones of the tests and of bench.py):
  planted  seeded planted partitions, the family of the small-graph tests, the
           CLI tests and the batched workload;
  rmat     R-MAT graphs, the family the headline number is quoted on;
  lfr      LFR-like graphs, the family the learned mode is trained on.
Weights: "unit"; "uniform" in [0.5, 1.5) on a 2^-24 grid (fixed-point values
below 2^32); "fine" = exponentially distributed float32 values using their
whole mantissa, as similarity scores do (fixed-point values above 2^32).
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    name = "gpu_louvain_b200"
    if name not in sys.modules:
        d = os.path.join(os.getcwd(), "gpu-louvain_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def _run(name, family, weights, source, min_gain=1e-6, **size):
    return dict(name=name, kind="run", family=family, weights=weights, source=source, min_gain=min_gain, **size)


def listed():
    return [
        # the smallest calls: one small graph from host arrays to its map, as
        # the command line tool and a script over many files do it
        _run("planted_2k_host", "planted", "unit", "host", 0.01, V=2000, blocks=16, d_in=12.0, d_out=2.0),
        # the small graph of the tests with an odd vertex count, already on the GPU
        _run("planted_10k", "planted", "uniform", "device", V=10007, blocks=64, d_in=16.0, d_out=2.0),
        # a mid-sized network with power-law degrees and communities, from host arrays
        _run("lfr_300k_host", "lfr", "unit", "host", V=300007, mu=0.3),
        # the largest configuration that the tests compare with the CPU, on the GPU
        _run("rmat20", "rmat", "uniform", "device", scale=20, edge_factor=16),
        # real-valued weights: 64-bit sums at every level
        _run("rmat21_fine", "rmat", "fine", "device", scale=21, edge_factor=16),
        # the headline run
        _run("rmat24", "rmat", "uniform", "device", scale=24, edge_factor=16),
        # a matrix file's entries to the map: the graph is built on the GPU
        dict(name="entries_rmat18", kind="entries", family="rmat", weights="uniform", min_gain=1e-6, scale=18,
             edge_factor=16),
        # the level loop driven operator by operator on a kept handle
        dict(name="operators_rmat16", kind="operators", family="rmat", weights="unit", min_gain=1e-6, scale=16,
             edge_factor=16),
        # learned active-set sweeps on a graph of the family they are meant for
        dict(name="learned_lfr_1m", kind="learned", family="lfr", weights="unit", min_gain=1e-6, V=1000003, mu=0.35),
        # the batched workload's graphs (sizes over its whole range)
        dict(name="batch_256", kind="batch", weights="unit", min_gain=1e-6, graphs=256, V_min=100, V_max=50000),
        # a batch of many small graphs (ego networks, molecules, sessions)
        dict(name="batch_2048_small", kind="batch", weights="uniform", min_gain=1e-6, graphs=2048, V_min=100,
             V_max=1500),
        # the value of a partition without any allocation
        dict(name="modularity_noalloc", kind="modularity", family="planted", weights="uniform", V=200003, blocks=256,
             d_in=16.0, d_out=2.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_planted(rng, lo, hi):
    V = _log(rng, lo, hi)
    return dict(family="planted", V=V, blocks=min(rng.randint(4, 256), V), d_in=round(rng.uniform(8.0, 24.0), 3),
                d_out=round(rng.uniform(1.0, 4.0), 3))


def draw(rng):
    weights = rng.choice(["unit", "uniform", "fine"])
    gain = rng.choice([1e-6, 1e-6, 1e-4, 0.01])
    kind = rng.choice(["run", "run", "run", "run", "entries", "operators", "learned", "batch", "modularity"])
    c = dict(kind=kind, weights=weights, min_gain=gain)
    if kind == "run":
        c["source"] = rng.choice(["host", "device"])
        family = rng.choice(["planted", "planted", "lfr", "rmat"])
        if family == "planted":
            c.update(_draw_planted(rng, 500, 300000))
        elif family == "lfr":
            c.update(family="lfr", V=_log(rng, 20000, 600000), mu=round(rng.uniform(0.2, 0.5), 3))
        else:
            c.update(family="rmat", scale=rng.randint(12, 22), edge_factor=rng.randint(6, 16), source="device")
    elif kind in ("entries", "operators"):
        if rng.random() < 0.5:
            c.update(family="rmat", scale=rng.randint(12, 18), edge_factor=rng.randint(6, 16))
        else:
            c.update(_draw_planted(rng, 1000, 200000))
    elif kind == "learned":
        c.update(family="lfr", weights="unit", min_gain=1e-6, V=_log(rng, 100000, 1000000),
                 mu=round(rng.uniform(0.2, 0.5), 3))
    elif kind == "batch":
        lo = _log(rng, 50, 1000)
        hi = _log(rng, 4 * lo, 50000)
        c.update(weights=rng.choice(["unit", "uniform"]), V_min=lo, V_max=hi,
                 graphs=max(4, min(2048, _log(rng, 16, 4000000 // hi))))
    else:
        c = dict(kind=kind, weights=weights, **_draw_planted(rng, 1000, 1 << 20))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _Memory:
    """Device memory of the library seen as an array by torch."""

    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 2}


def _tensor(ptr, n, kind):
    t = torch.int32 if kind == "<i4" else torch.float32
    return torch.as_tensor(_Memory(ptr, n, kind), device="cuda").clone() if n else torch.empty(0, dtype=t,
                                                                                               device="cuda")


def _fine(rp, cl, seed):
    """Exponentially distributed weights, the same for both directions of an edge."""
    V = rp.numel() - 1
    row = torch.repeat_interleave(torch.arange(V, dtype=torch.int32, device=rp.device), (rp[1:] - rp[:-1]).long(),
                                  output_size=cl.numel())
    x = torch.minimum(row, cl).long() * 0x2545F491 + torch.maximum(row, cl).long() * 0x9E3779B1
    del row
    x = (x + (seed % 65521) * 0x632BE5AB) & ((1 << 62) - 1)
    for m in (0x45D9F3B5, 0x119DE1F3):
        x ^= x >> 29
        x = (x * m) & ((1 << 62) - 1)
    x ^= x >> 31
    u = ((x & ((1 << 40) - 1)).double() + 0.5) / float(1 << 40)
    return (-torch.log(u)).float()


def _device_csr(case, seed):
    """(rowptr, col, w) on the GPU."""
    L = _package()
    base = "uniform" if case["weights"] == "uniform" else "unit"
    if case["family"] == "rmat":
        g = L.gen_rmat_device(case["scale"], case["edge_factor"], seed, weights=base)
        rp, cl, w = _tensor(g.rowptr, g.V + 1, "<i4"), _tensor(g.col, g.E, "<i4"), _tensor(g.w, g.E, "<f4")
        torch.cuda.synchronize()
        g.free()
    else:
        if case["family"] == "lfr":
            g, _ = L.gen_lfr(case["V"], case["mu"], seed)
        else:
            g = L.gen_planted(case["V"], case["blocks"], case["d_in"], case["d_out"], seed, base)
        rp, cl, w = (torch.from_numpy(x).cuda() for x in (g.rowptr, g.col, g.w))
        if case["family"] == "lfr" and base == "uniform":   # the LFR generator draws unit weights
            w = 0.5 + torch.floor(torch.remainder(_fine(rp, cl, seed), 1.0) * float(1 << 22)) / float(1 << 22)
    if case["weights"] == "fine":
        w = _fine(rp, cl, seed)
    return rp, cl, w


def _host_graph(case, seed):
    rp, cl, w = _device_csr(case, seed)
    return _package().Graph(rp.cpu().numpy(), cl.cpu().numpy(), w.cpu().numpy())


def _pointers(csr):
    rp, cl, w = csr
    return rp.data_ptr(), cl.data_ptr(), w.data_ptr(), rp.numel() - 1, cl.numel()


def _batch_params(case, seed):
    # the sizes follow from the case, the graphs from the seed
    r = np.random.default_rng([case["graphs"], case["V_min"], case["V_max"]])
    out = []
    for i in range(case["graphs"]):
        V = int(round(math.exp(r.uniform(math.log(case["V_min"]), math.log(case["V_max"])))))
        out.append((V, min(int(r.integers(4, 257)), V), float(r.uniform(8.0, 24.0)), float(r.uniform(1.0, 4.0)),
                    seed * 1000003 + i))
    return out


def _partition(V, blocks, seed):
    """The planted blocks with a tenth of the vertices elsewhere."""
    r = np.random.default_rng([seed, 7])
    c = (np.arange(V, dtype=np.int64) * blocks // V).astype(np.int32)
    at = r.integers(0, V, V // 10)
    c[at] = r.integers(0, blocks, V // 10)
    return c


def prepare(case, seed):
    L = _package()
    L.lib()
    kind = case["kind"]
    s = {"case": case, "kind": kind, "L": L}
    if kind == "run" and case["source"] == "host":
        s["graph"] = _host_graph(case, seed)
    elif kind in ("run", "learned"):
        s["csr"] = _device_csr(case, seed)
        if kind == "learned":
            s["model"] = L.load_active_model()
            s["settings"] = L.read_active_model()[2]
    elif kind == "entries":
        u, v, w = _host_graph(case, seed).edges()
        order = np.random.default_rng([seed, 3]).permutation(len(u))   # a file need not be sorted
        s["V"] = 1 << case["scale"] if case["family"] == "rmat" else case["V"]
        s["entries"] = tuple(np.ascontiguousarray(x[order]) for x in (u, v, w))
    elif kind == "operators":
        s["csr"] = _device_csr(case, seed)
        torch.cuda.synchronize()
        s["engine"] = L.Louvain(device_csr=_pointers(s["csr"]))
    elif kind == "batch":
        rp, cl, w, gp = L.gen_planted_batch(_batch_params(case, seed), case["weights"])
        s["csr"] = tuple(torch.from_numpy(x).cuda() for x in (rp, cl, w))
        s["graph_ptr"] = gp
    elif kind == "modularity":
        s["csr"] = _device_csr(case, seed)
        s["comm"] = torch.from_numpy(_partition(case["V"], case["blocks"], seed)).cuda()
        s["q"], s["err"] = C.c_double(), C.create_string_buffer(256)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
LEVELS = 64   # rows of the per-level outputs (a run has about five levels)


def _whole(engine, min_gain):
    q = engine.run(min_gain)
    m, n = engine.original_to_community()
    engine.close()
    return {"modularity": q, "map": m, "communities": n}


def run(s):
    L, case, kind = s["L"], s["case"], s["kind"]
    if kind == "run":
        if case["source"] == "host":
            return _whole(L.Louvain(s["graph"]), case["min_gain"])
        return _whole(L.Louvain(device_csr=_pointers(s["csr"])), case["min_gain"])
    if kind == "learned":
        e = L.Louvain(device_csr=_pointers(s["csr"]), active_set=True, active_full_every=s["settings"]["full_every"],
                      active_start=s["settings"]["active_start"], active_min_recall=s["settings"]["min_recall"])
        e.set_active_model(*s["model"])
        return _whole(e, case["min_gain"])
    if kind == "entries":
        g = L.csr_from_entries_device(s["V"], *s["entries"])
        out = _whole(L.Louvain(device_csr=(g.rowptr, g.col, g.w, g.V, g.E)), case["min_gain"])
        g.free()
        return out
    if kind == "operators":
        e = s["engine"]
        e.reset()
        qs, sizes = np.zeros(LEVELS), np.zeros((LEVELS, 2), np.int64)
        level = 0
        while e.optimise_modularity(case["min_gain"]):
            qs[level] = e.calculate_modularity()
            e.aggregate_communities()
            sizes[level] = e.level_info()[:2]
            level += 1
        m, n = e.original_to_community()
        return {"modularity": e.calculate_modularity(), "level_modularity": qs, "level_sizes": sizes, "map": m,
                "communities": n}
    if kind == "batch":
        rp, cl, w = s["csr"]
        with L.Batch(graph_ptr=s["graph_ptr"], device_csr=(rp.data_ptr(), cl.data_ptr(), w.data_ptr()),
                     num_vertices=rp.numel() - 1, num_entries=cl.numel()) as b:
            b.run(case["min_gain"])
            return b.results()
    rp, cl, w = s["csr"]
    rc = L.lib().lv_modularity_noalloc(rp.data_ptr(), cl.data_ptr(), w.data_ptr(), rp.numel() - 1, cl.numel(),
                                       s["comm"].data_ptr(), None, C.byref(s["q"]), s["err"], 256)
    if rc != L.LV_OK:
        raise L.LouvainError(rc, s["err"].value.decode())
    return s["q"].value


# ---------------------------------------------------------------------------
# sizes and values
# ---------------------------------------------------------------------------
def _size(case):
    """(vertices, CSR entries) of the case's graph, duplicates aside."""
    if case["kind"] == "batch":
        lo, hi = math.log(case["V_min"]), math.log(case["V_max"])
        V = case["graphs"] * ((case["V_max"] - case["V_min"]) / (hi - lo) if hi > lo else case["V_min"])
        return V, V * 18.5
    if case["family"] == "rmat":
        V = 1 << case["scale"]
        return V, 1.9 * V * case["edge_factor"]
    if case["family"] == "lfr":
        return case["V"], 20.0 * case["V"]
    return case["V"], case["V"] * (case["d_in"] + case["d_out"])


def work(case):
    """The CSR (or the entries) read once, the map or the value written once."""
    V, E = _size(case)
    out = 8.0 if case["kind"] == "modularity" else 4.0 * V
    given = 12.0 * E / 2 if case["kind"] == "entries" else 4.0 * (V + 1) + 8.0 * E
    given += 4.0 * V if case["kind"] == "modularity" else 0.0
    return {"bytes": given + out, "flops": 0.0}


def exact(case, seed):
    """The modularity of the given partition in 64-bit arithmetic; the other
    kinds search for a partition, which has no value to hold it to."""
    if case["kind"] != "modularity":
        return None
    rp, cl, w = (x.cpu().numpy() for x in _device_csr(case, seed))
    c = _partition(case["V"], case["blocks"], seed)
    row = np.repeat(np.arange(case["V"]), np.diff(rp))
    w = w.astype(np.float64)
    total = w.sum()
    inside = w[c[row] == c[cl]].sum()
    sums = np.bincount(c[row], weights=w, minlength=case["blocks"])
    return float(inside / total - np.square(sums / total).sum())
