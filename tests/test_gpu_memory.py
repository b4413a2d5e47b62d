"""Device memory that runs out at any allocation of a handle: a call either
fails with LV_ERR_NOMEM or, where the buffer only makes later sweeps faster,
gives the usual result; the handle, reset, then runs as if nothing had been.
The failures are made on the host (lv_set_test_limits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAIN = 1e-7


def _graph(lvb, name):
    if name == "small":      # one launch
        return lvb.gen_planted(2000, 16, 12.0, 2.0, 1, "uniform"), {}
    if name == "levels":
        return lvb.gen_planted(10007, 64, 14.0, 3.0, 2, "uniform"), {}
    if name == "giants":     # rows beyond the giant degree
        return lvb.gen_rmat(15, 16, 3), {"giant_degree": 1024}
    if name == "tables":     # late sweeps from tables
        return lvb.gen_planted(10000, 24, 300.0, 15.0, 3, "uniform"), {}
    if name == "learned":    # the proposals' buffers
        return lvb.gen_lfr(70000, 0.4, 5)[0], {"active_set": True, "active_start": 0.2, "active_min_recall": 0.5}
    if name == "traced":
        return lvb.gen_planted(3000, 24, 14.0, 3.0, 5, "uniform"), {"trace_sample": 0.5}


def _engine(lvb, g, kw):
    e = lvb.Louvain(g, **kw)
    if kw.get("active_set"):
        e.set_active_model(*lvb.load_active_model())
    return e


def _result(e):
    q = e.run(GAIN)
    m, n = e.original_to_community()
    return q, n, m


@pytest.mark.parametrize("name", ["small", "levels", "giants", "tables", "learned", "traced"])
def test_failing_allocations(lvb, name):
    g, kw = _graph(lvb, name)
    with _engine(lvb, g, kw) as e:
        want = _result(e)
    refused = 0
    for n in range(1, 80):
        with _engine(lvb, g, kw) as e:
            e.set_test_limits(n)
            for again in (False, True):   # the second time with the hook off
                try:
                    got = _result(e)
                    assert got[:2] == want[:2] and np.array_equal(got[2], want[2]), n
                except lvb.LouvainError as x:
                    assert x.status == lvb.LV_ERR_NOMEM and not again, (n, x)
                    refused += 1
                e.set_test_limits(0)
                e.reset()
    assert 0 < refused < 79   # the last failures lie past the last allocation


@pytest.mark.parametrize("name", ["levels", "giants", "tables"])
def test_level_goes_on_after_a_failed_aggregation(lvb, name):
    """An aggregation that ran out of memory leaves its level as it was: swept
    again and aggregated, it gives what a handle gives whose aggregation never
    failed."""
    g, kw = _graph(lvb, name)

    def operators(fail):
        out, failed = [], 0
        with lvb.Louvain(g, **kw) as e:
            while e.optimise_modularity(GAIN):
                if fail:
                    e.set_test_limits(fail)
                    try:
                        e.aggregate_communities()
                        e.set_test_limits(0)
                        return None, 0   # past the level's last allocation
                    except lvb.LouvainError as x:
                        assert x.status == lvb.LV_ERR_NOMEM
                        failed += 1
                    e.set_test_limits(0)
                    fail = 0
                out.append((e.sweep(), e.calculate_modularity()))
                e.aggregate_communities()
                out.append(e.level_info())
            return out + [e.original_to_community()[0].tobytes()], failed

    want, _ = operators(0)
    for n in range(1, 60):
        got, failed = operators(n)
        if got is None:
            break
        assert failed == 1 and got == want, n
    assert 20 < n < 59


def test_threads_share_the_device_memory(lvb):
    """Engines, batches and CSR builds of several sizes in four threads, each
    from create to destroy, give what they give alone: blocks and streams pass
    from one owner to the next through the library's per-device lists."""
    import threading

    def engine(g, **kw):
        def f():
            with _engine(lvb, g, kw) as e:
                q, n, m = _result(e)
            return q, n, m.tobytes()
        return f

    def batch(graphs):
        def f():
            with lvb.Batch(graphs) as b:
                b.run(GAIN)
                r = b.results()
            return r["communities"].tobytes(), r["modularity"].tobytes()
        return f

    def entries(g):
        u, v, w = g.edges()

        def f():
            d = lvb.csr_from_entries_device(g.V, u, v, w)
            with lvb.Louvain(device_csr=(d.rowptr, d.col, d.w, d.V, d.E)) as e:
                q, n, m = _result(e)
            d.free()
            return q, n, m.tobytes()
        return f

    graphs = [lvb.gen_planted(300 + 900 * i, 8 + i, 12.0, 2.0, i, "uniform") for i in range(6)]
    jobs = [engine(graphs[2]), engine(lvb.gen_rmat(14, 16, 1)), engine(lvb.gen_rmat(15, 16, 2), giant_degree=1024),
            engine(lvb.gen_planted(10000, 24, 300.0, 15.0, 3, "uniform")),
            engine(lvb.gen_lfr(70000, 0.4, 5)[0], active_set=True, active_start=0.2, active_min_recall=0.5),
            batch(graphs), batch([lvb.gen_planted(20000, 40, 14.0, 3.0, 9, "uniform")] + graphs[:3]),
            entries(lvb.gen_rmat(13, 16, 4))]
    alone = [f() for f in jobs]
    bad = []

    def work(t):
        try:
            for i in np.random.default_rng(t).permutation(np.repeat(np.arange(len(jobs)), 3)):
                if jobs[i]() != alone[i]:
                    bad.append((t, int(i), "differs"))
        except Exception as x:   # noqa: BLE001 -- reported below
            bad.append((t, int(i), x))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
