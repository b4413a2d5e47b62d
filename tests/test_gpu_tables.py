"""Late sweeps from neighbour-community tables: that they run where they may and
do not where they must not, and that every way through them (tables built by a
warp and by a CTA, giants, rows with too many communities, tables gone stale, a
pool used up) decides as the host loop does, which always sums rows."""
import numpy as np
import pytest

from test_gpu_scale import _table_graphs
from test_sym_mix import PAIRS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs(lvb):
    return _table_graphs(lvb)


def _build(lvb, u, v, w, V):
    n = u != v
    rows, cols = np.concatenate([u, v[n]]), np.concatenate([v, u[n]])
    ww = np.concatenate([w, w[n]]).astype(np.float32)
    o = np.lexsort((cols, rows))
    rp = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=V), out=rp[1:])
    return lvb.Graph(rp, cols[o].astype(np.int32), ww[o])


def _run(lvb, g, limit=0, start=None, gain=1e-7, **kw):
    with lvb.Louvain(g, **kw) as e:
        e.set_test_limits(0, limit)
        if start is not None:
            e.set_communities(start)
            e.optimise_modularity(gain)
            out = e.calculate_modularity(), e.communities()
        else:
            out = e.run(gain), e.original_to_community()[0]
        st = e.stats()
        return out + (st["sweeps"], st["moves"]), e.table_stats()


def _same(a, b):
    assert a[0] == b[0] and a[2:] == b[2:] and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("name", ["planted", "fine", "rmat18"])
def test_tables_run_and_a_small_pool_does(lvb, graphs, name):
    g = graphs[name]
    want, st = _run(lvb, g, sweep_graph=False)
    assert st["sweeps"] == 0
    got, st = _run(lvb, g)
    _same(got, want)
    assert st["sweeps"] > 0 and st["slots"] > 0 and not st["pool_full"]
    for limit in (1, 4096, g.E // 100):
        got, st = _run(lvb, g, limit)
        _same(got, want)
        assert st["sweeps"] > 0 and st["pool_full"] and st["slots"] <= limit * 3   # three levels at most


def test_tables_do_not_run_on_zero_weights_or_asymmetric_entries(lvb, graphs):
    base = graphs["planted"]
    w = base.w.copy()
    w[::100] *= 2.0
    # one edge of two weights each that a weaker mix took for symmetric
    row = np.repeat(np.arange(base.V), np.diff(base.rowptr))
    a, b, k = np.array(PAIRS).T
    rows, cols = np.concatenate([row, a, b]), np.concatenate([base.col, b, a])
    ww = np.concatenate([base.w, 2.0 ** (k - 24), 2.0 ** (k - 23)]).astype(np.float32)
    o = np.lexsort((cols, rows))
    rp = np.zeros(base.V + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=base.V), out=rp[1:])
    for g in (graphs["zero"], lvb.Graph(base.rowptr, base.col, w),
              lvb.Graph(rp, cols[o].astype(np.int32), ww[o])):
        want, _ = _run(lvb, g, sweep_graph=False, max_sweeps=40)
        got, st = _run(lvb, g, max_sweeps=40)
        _same(got, want)
        assert st["sweeps"] == 0


@pytest.fixture(scope="module")
def gadgets(lvb, graphs):
    """A settled planted graph (of its own communities) and, beside it:
    - 64 chains c0 .. c6: c1 .. c6 start in community A, whose core they are
      tied to; a chain vertex follows the one before it, one step per sweep,
      out of A into the community of its chain's c0;
    - hub s, tied to every chain's c3: its table, built while all are in A,
      meets 64 new communities a sweep later;
    - 9000 settled pairs: hub n is tied to all of them, hub m to 1000;
    - hub g, tied to 9500 planted vertices (beyond the giant degree)."""
    base = graphs["planted"]
    with lvb.Louvain(base) as e:
        e.run(1e-7)
        c = e.original_to_community()[0]
    first = np.full(c.max() + 1, base.V, np.int64)
    np.minimum.at(first, c, np.arange(base.V))
    u, v, w = (list(x) for x in base.edges())
    comm = list(first[c])
    V = base.V

    def vertex(community=None):
        nonlocal V
        comm.append(V if community is None else community)
        V += 1
        return V - 1

    def edge(x, y, weight):
        u.append(x), v.append(y), w.append(weight)

    core = vertex()
    core2 = vertex(core)
    edge(core, core2, 8.0)
    s = vertex()
    for _ in range(64):
        c0 = vertex()
        edge(c0, vertex(c0), 4.0)
        last = c0
        for i in range(1, 7):
            x = vertex(core)
            edge(last, x, 4.0 ** -i)
            edge(core, x, 4.0 ** -i / 2)
            if i == 3:
                edge(s, x, 2.0 ** -16)
            last = x
    n, m, big = vertex(), vertex(), vertex()
    for i in range(9000):
        p = vertex()
        edge(p, vertex(p), 1.0)
        edge(n, p, 2.0 ** -10)
        if i < 1000:
            edge(m, p, 2.0 ** -10)
    for x in range(9500):
        edge(big, x, 2.0 ** -12)
    g = _build(lvb, np.array(u), np.array(v), np.array(w), V)
    return g, np.array(comm, np.int32)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("giant_degree", [0, 1024])
def test_every_way_through_the_tables(lvb, gadgets, wide, giant_degree):
    g, start = gadgets
    kw = {"start": start, "gain": 0.0, "wide_weights": wide, "giant_degree": giant_degree}
    want, _ = _run(lvb, g, sweep_graph=False, **kw)
    assert want[2] >= 6   # a chain takes as many sweeps
    got, st = _run(lvb, g, **kw)
    _same(got, want)
    assert st["sweeps"] >= 4
    assert st["stale"] and st["without"] >= 1 and not st["pool_full"]
    got, st = _run(lvb, g, 20000, **kw)
    _same(got, want)
    assert st["pool_full"]
