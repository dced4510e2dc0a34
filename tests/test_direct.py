"""Small graphs scored without a grid barrier (csrc/gg_direct.cuh): every result field
against the oracle and against the level loop (GG_DIRECT=0), at the edges of the groups
(32, 64 and 128 sources), of the row tables (16-bit ids in shared memory or the table
itself), of the table's way to the device, and for ranges, caps and rejected tables."""
import numpy as np
import pytest

import graphgolf as G
import instances as I
import oracle as O

pytestmark = pytest.mark.gpu


def both(monkeypatch, make, call):
    monkeypatch.setenv("GG_DIRECT", "0")
    e = make()
    want = call(e)
    e.close()
    monkeypatch.delenv("GG_DIRECT")
    e = make()
    got = call(e)
    again = call(e)     # the counters of the first call were cleared
    e.close()
    return want, got, again


KEYS = ("total", "reached", "pairs", "levels", "capped", "connected", "n_sources")


@pytest.mark.parametrize("n,d", [(2, 1), (5, 2), (31, 4), (32, 3), (33, 4), (64, 5), (129, 6), (1000, 7), (1023, 8), (1025, 12),
                                 (700, 16), (600, 17), (3001, 4), (4740, 6), (5001, 8), (7001, 16), (9473, 4), (12001, 6)])
def test_direct_counts_equal_the_level_loop(n, d, monkeypatch):
    adj = G.random_regular(n if n * d % 2 == 0 else n + 1, d, 3) if n > 2 else np.array([[1], [0]], np.int32)
    n = len(adj)
    cap = 40
    want, got, again = both(monkeypatch, lambda: G.cudaASPLgraph(n, d),
                            lambda e: e.eval(adj, max_levels=cap, level_counts=True))
    for r in (got, again):
        assert all(r[k] == want[k] for k in KEYS)
        assert np.array_equal(r["level_counts"], want["level_counts"])
    o = O.bfs_pull(adj, np.arange(n))
    assert (got["total"], got["reached"], got["levels"]) == (o.total(), int(o.reached.sum()), o.levels)


@pytest.mark.parametrize("form", ["part", "part_m3", "piece", "box", "wvc", "wvc_bits"])
def test_direct_lifted_forms(form, monkeypatch):
    if form in ("part", "part_m3", "wvc", "wvc_bits"):
        N, M, T = G.cyclic_lift(*{"part": (150, 9, 5, 1), "part_m3": (64, 3, 4, 2), "wvc": (500, 12, 6, 3),
                                  "wvc_bits": (37, 40, 4, 4)}[form])
        make = lambda: G.cudaASPLconv(N, M, T.shape[1])
        call = (lambda e: e.WVCdiameterASPL(T)) if form.startswith("wvc") else (lambda e: e.diameterASPL(T))
    elif form == "piece":
        a = G.piece_lift(5, 7, 4, 3, 6, 1)
        make, call = (lambda: G.cudaASPLpiece(*a[:4], 6)), (lambda e: e.diameterASPL(a[4]))
    else:
        a = I.random_box(3, 2, 4, 2, 3, 2, 6, 1)
        make, call = (lambda: G.cudaASPLbox(*a[:6], 6)), (lambda e: e.diameterASPL(a[6]))
    want, got, again = both(monkeypatch, make, call)
    assert got == want and again == want


def test_direct_ranges_caps_disconnected_and_bad_tables(monkeypatch):
    adj = G.random_regular(1500, 4, 5)
    make = lambda: G.cudaASPLgraph(1500, 4)
    for call in (lambda e: e.eval(adj, src_range=(3, 700)), lambda e: e.eval(adj, max_levels=3),
                 lambda e: e.eval(adj, src_range=(1499, 1500), max_levels=2)):
        want, got, again = both(monkeypatch, make, call)
        assert all(got[k] == want[k] and again[k] == want[k] for k in KEYS)
    two = np.concatenate([I.cycle(40), I.cycle(40) + 40]).astype(np.int32)    # disconnected
    long = np.asarray(I.cycle(500), dtype=np.int32)                              # past calc's 199 levels
    for t in (two, long, I.path_graph(70)):
        want, got, again = both(monkeypatch, lambda: G.cudaASPLgraph(len(t), t.shape[1]), lambda e: e.calc(t))
        assert got == want and again == want
    wvc = np.array([[2, -2]] * 8, np.int32)                                      # two cycles, with masks
    o = lambda e: e.eval(wvc, max_levels=50, want_wvc=True)
    want, got, again = both(monkeypatch, lambda: G.cudaASPLconv(64, 8, 2), o)
    assert all(got[k] == want[k] and again[k] == want[k] for k in KEYS + ("wvc",))
    for n, d in ((100, 4), (9000, 16)):      # read over the bus; ids from the table itself
        e = G.cudaASPLgraph(n, d)
        good = G.random_regular(n, d, 6)
        first = e.calc(good)
        for v in (n, -1, 1 << 20):
            bad = good.copy()
            bad[n // 2, 1] = v
            with pytest.raises(G.GGError) as err:
                e.calc(bad)
            assert err.value.status == G.GG_BAD_ARG
            assert e.calc(good) == first
        e.close()


def test_direct_device_tables_of_any_alignment():
    import torch
    for n, d in ((200, 5), (3000, 8), (9000, 16)):
        adj = G.random_regular(n, d, 7)
        e = G.cudaASPLgraph(n, d)
        want = e.eval(adj)
        buf = torch.zeros(n * d + 8, dtype=torch.int32, device="cuda")
        for shift in (0, 1, 2, 3):
            buf[shift:shift + n * d] = torch.from_numpy(adj.ravel()).cuda()
            torch.cuda.synchronize()
            got = e.eval_device(buf.data_ptr() + 4 * shift)
            assert all(got[k] == want[k] for k in KEYS)
        e.close()


def one_way(n, d, seed, edits):
    """A table of n rows whose entries do not come back: an arbitrary one, or (edits > 0) a
    random regular graph's with a few entries replaced."""
    rng = np.random.default_rng(seed)
    if not edits:
        return rng.integers(0, n, (n, d)).astype(np.int32)
    adj = G.random_regular(n, d, seed).copy()
    for v in rng.choice(n, edits, replace=False):
        adj[v, rng.integers(d)] = (v + 1 + rng.integers(n - 1)) % n
    return adj


@pytest.mark.parametrize("n,d,edits", [(9, 2, 0), (31, 1, 0), (74, 4, 0), (552, 8, 1), (1236, 2, 0), (2667, 9, 0), (3001, 4, 3),
                                       (4096, 16, 1), (9000, 8, 2), (20000, 6, 1)])
def test_direct_tables_with_one_way_entries(n, d, edits):
    adj = one_way(n + n * d % 2 * bool(edits), d, 11, edits)
    n = len(adj)
    o = O.bfs_pull(adj, np.arange(n))
    e = G.cudaASPLgraph(n, d)
    good = G.random_regular(n, d, 5) if n * d % 2 == 0 and n > d + 1 else None
    for t in (adj, adj, good, adj):      # with walks and, after the first, without
        if t is None:
            continue
        w = o if t is adj else O.bfs_pull(t, np.arange(n))
        r = e.eval(t, level_counts=True, max_levels=w.levels + 3)
        assert (r["total"], r["reached"], r["levels"]) == (w.total(), int(w.reached.sum()), w.levels)
    part = O.bfs_pull(adj, np.arange(n // 3, n // 2 + 1))
    e.close()
    e = G.cudaASPLgraph(n, d)
    r = e.eval(adj, src_range=(n // 3, n // 2 + 1))
    assert (r["total"], r["reached"], r["levels"]) == (part.total(), int(part.reached.sum()), part.levels)
    e.close()


@pytest.mark.parametrize("form,args", [("part", (78, 2, 9)), ("part", (5, 1, 3)), ("part", (939, 6, 6)), ("part", (2, 39, 8)),
                                       ("ragged", (71, 296, 12)), ("ragged", (3, 64, 4)), ("piece", (3, 13, 4, 1, 5)),
                                       ("piece", (7, 17, 6, 3, 8)), ("box", (5, 5, 2, 4, 3, 2, 3)), ("one", (300, 11, 6))])
def test_direct_lifts_with_one_way_entries(form, args):
    rng = np.random.default_rng(5)
    if form in ("part", "ragged", "one"):
        M, g, d = args
        N = g if form == "ragged" else M * g
        T = rng.integers(-N, N, (M, d)).astype(np.int32)
        if form == "one":                # one entry of a symmetric lift, in the last orbit
            T = G.cyclic_lift(M, g, d, 3)[2].copy()
            T[M - 1, 0] += 1
        e, adj, src = G.cudaASPLconv(N, M, d), O.expand_part(N, M, T), np.arange(M)
    else:
        ax = 2 if form == "piece" else 3
        m, k, d = args[:ax], args[ax:2 * ax], args[-1]
        n = [x * y for x, y in zip(m, k)]
        T = rng.integers(-9, 9, (int(np.prod(m)), d, ax)).astype(np.int32)
        x = np.array(np.unravel_index(np.arange(int(np.prod(n))), n))
        o = np.ravel_multi_index([x[j] % m[j] for j in range(ax)], m)
        adj = np.ravel_multi_index([(x[j][:, None] + T[o][:, :, j]) % n[j] for j in range(ax)], n)
        src = np.ravel_multi_index(list(np.array(np.unravel_index(np.arange(int(np.prod(m))), m))), n)
        e = (G.cudaASPLpiece if ax == 2 else G.cudaASPLbox)(*n, *m, d)
    w = O.bfs_pull(np.ascontiguousarray(adj, dtype=np.int32), src)
    for wvc in (False, True, False):
        r = e.eval(T, want_wvc=wvc)
        assert (r["total"], r["reached"], r["levels"]) == (w.total(), int(w.reached.sum()), w.levels)
    e.close()


@pytest.mark.parametrize("rows", [1, 2, 33, 5000])
def test_degree_zero_takes_the_level_loop(rows):
    for make, table in ((lambda: G.cudaASPLgraph(rows, 0), np.zeros((rows, 0), np.int32)),
                        (lambda: G.cudaASPLconv(2 * rows, rows, 0), np.zeros((rows, 0), np.int32)),
                        (lambda: G.cudaASPLpiece(rows, 3, rows, 1, 0), np.zeros((rows, 0, 2), np.int32)),
                        (lambda: G.cudaASPLbox(rows, 2, 2, rows, 1, 1, 0), np.zeros((rows, 0, 3), np.int32))):
        e = make()
        for _ in range(2):
            r = e.eval(table)
            one = r["pairs"] == r["n_sources"]        # a single vertex reaches all there is
            assert (r["total"], r["reached"], r["levels"], r["connected"]) == (0, r["n_sources"], 0, int(one))
            assert r["n_sources"] == rows
        e.close()


def test_direct_while_the_default_stream_is_busy():
    """A new engine's counters are cleared in the order of its own work: other work that waits
    on the default stream neither delays nor follows it.  Also when a larger level cap makes
    them anew, and on a caller's stream."""
    import torch
    adj = G.random_regular(600, 4, 3)
    o = O.bfs_pull(adj, np.arange(600))
    table = torch.from_numpy(adj).cuda()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        torch.cuda._sleep(int(4e7))         # about 20 ms
        e = G.cudaASPLgraph(600, 4)
        torch.cuda._sleep(int(4e7))
        for cap in (0, 300, 40000, 0):      # (0: 600 levels)
            r = e.eval(adj, max_levels=cap)
            assert (r["total"], r["reached"], r["levels"]) == (o.total(), int(o.reached.sum()), o.levels)
            r = e.eval_device(table.data_ptr(), max_levels=2 * cap, stream=other.cuda_stream)
            assert (r["total"], r["reached"], r["levels"]) == (o.total(), int(o.reached.sum()), o.levels)
        e.close()
        torch.cuda.synchronize()


@pytest.mark.parametrize("n,d", [(5000, 6), (9000, 4), (12000, 8)])
def test_an_engine_takes_the_memory_of_what_it_runs(n, d):
    """Created and called once: the rows of all batches, the level loop's buffers and the
    level-2 lists only where the call needs them (bytes of the whole engine)."""
    import torch
    adj = G.random_regular(n, d, 1)
    G.cudaASPLgraph(n, d).calc(adj)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    e = G.cudaASPLgraph(n, d)
    e.calc(adj)
    used = before - torch.cuda.mem_get_info()[0]
    rows = n * ((n + 4095) // 4096) * 512                    # of every source, once
    assert used <= (3 * rows if n > 10000 else 0) + n * d * d * 4 + (8 << 20), used
    # and what it runs after that: a range of the sources, a graph with one-way entries
    half = [e.eval(adj, src_range=r) for r in ((0, 3000), (3000, n))]
    assert sum(r["total"] for r in half) == e.calc(adj)[1]
    odd = adj.copy()
    odd[7, 1] = (odd[7, 1] + 1) % n
    for t in (odd, adj):
        o = O.bfs_pull(t, np.arange(n))
        r = e.eval(t)
        assert (r["total"], r["reached"], r["levels"]) == (o.total(), int(o.reached.sum()), o.levels)
    e.close()


@pytest.mark.parametrize("n,d,oneway", [(3000, 40, 0), (9000, 24, 0), (1000, 64, 0), (20000, 10, 1), (14000, 13, 1)])
def test_calls_take_no_longer_than_the_level_loop(n, d, oneway, monkeypatch):
    """High degrees, and tables whose first levels no walk takes.  (Least of many, in turn.)"""
    import time
    q = -(-d // 12)
    t = np.ascontiguousarray(np.concatenate([G.random_regular(n, (d + k) // q, k) for k in range(q)], axis=1))
    if oneway:
        t[5, 0] = (t[5, 0] + 1) % n
    monkeypatch.setenv("GG_DIRECT", "0")
    monkeypatch.setenv("GG_SWEEP", "0")
    loop = G.cudaASPLgraph(n, d)
    monkeypatch.delenv("GG_DIRECT")
    monkeypatch.delenv("GG_SWEEP")
    e = G.cudaASPLgraph(n, d)
    best, seen = {loop: 1e9, e: 1e9}, set()
    for k in range(300):
        for h in (loop, e):
            t0 = time.perf_counter()
            seen.add(h.calc(t))
            best[h] = min(best[h], time.perf_counter() - t0)
        if k >= 29 and best[e] < 1.2 * best[loop]:    # (longer where the host was busy)
            break
    assert len(seen) == 1
    assert best[e] < 1.2 * best[loop], best
    loop.close()
    e.close()
