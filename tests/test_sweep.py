"""The levels after the walk of all batches in their plain case (csrc/gg_sweep.cuh) and the
walk itself at degrees 3, 4, 6 and 8 on batches of one or more 4096-source parts: every
result field against the oracle and against the general level loop (GG_SWEEP=0)."""
import numpy as np
import pytest

import graphgolf as G
import instances as I
import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("total", "reached", "pairs", "levels", "capped", "connected", "n_sources")


def both(monkeypatch, n, d, batch, calls):
    out = []
    for sweep in ("0", "1"):
        monkeypatch.setenv("GG_SWEEP", sweep)
        e = G.cudaASPLgraph(n, d)
        if batch:
            e.set_batch_sources(batch)
        out.append([c(e) for c in calls for _ in range(2)])
        e.close()
    for want, got in zip(*out):
        assert all(got[k] == want[k] for k in KEYS)
        assert not batch or got["level_steps"] == want["level_steps"]   # (the widths differ by default)
        assert np.array_equal(got["level_counts"], want["level_counts"])
    return out[1][0]


def full(adj, cap=40):
    return lambda e: e.eval(adj, max_levels=cap, level_counts=True)


def check_oracle(r, adj):
    o = O.bfs_pull(adj, np.arange(len(adj)))
    assert (r["total"], r["reached"], r["levels"]) == (o.total(), int(o.reached.sum()), o.levels)


@pytest.mark.parametrize("n,d,batch", [(5000, 3, 4096), (4098, 8, 4096), (8192, 8, 4096), (8193, 8, 8192), (12290, 4, 4096),
                                       (12289, 6, 8192), (4097, 5, 4096), (9001, 7, 8192), (10001, 9, 4096),
                                       (12001, 10, 4096), (9000, 11, 4096), (12300, 12, 12288), (8200, 13, 4096),
                                       (13001, 14, 0), (12290, 15, 0), (14001, 16, 0), (20002, 8, 8192), (20002, 6, 12288), (30011, 6, 0)])
def test_sweep_equals_the_level_loop(n, d, batch, monkeypatch):
    adj = G.random_regular(n if n * d % 2 == 0 else n + 1, d, 7)
    r = both(monkeypatch, len(adj), d, batch, [full(adj)])
    if n <= 13000:
        check_oracle(r, adj)


@pytest.mark.parametrize("cap", [1, 3, 4, 5, 6, 7])
def test_sweep_under_a_level_cap(cap, monkeypatch):
    adj = G.random_regular(9000, 8, 2)
    both(monkeypatch, 9000, 8, 4096, [full(adj, cap), full(adj)])


@pytest.mark.parametrize("what", ["padded", "tail", "ring", "halves", "one-way", "alone", "close"])
def test_sweep_gives_up_where_it_must(what, monkeypatch):
    n, d = 9000, 8
    adj = G.random_regular(n, d, 4)
    if what == "padded":          # self-loops in place of edges
        for v in range(0, n, 50):
            u = int(adj[v, 3])
            if u != v:
                adj[u, np.nonzero(adj[u] == v)[0][0]] = u
                adj[v, 3] = v
    elif what == "tail":          # a path of 5 vertices hanging off a random graph
        adj = np.concatenate([adj, np.arange(n, n + 5, dtype=np.int32)[:, None].repeat(d, 1)])
        u = int(adj[0, 0])
        adj[0, 0], adj[u, np.nonzero(adj[u] == 0)[0][0]] = n, u
        adj[n, 0] = 0
        for k in range(4):
            adj[n + k, 1], adj[n + k + 1, 0] = n + k + 1, n + k
        n += 5
    elif what == "ring":          # thin frontiers throughout
        adj = ((np.arange(n)[:, None] + np.array([-4, -3, -2, -1, 1, 2, 3, 4])) % n).astype(np.int32)
    elif what == "halves":
        half = G.random_regular(n // 2, d, 5)
        adj = np.concatenate([half, half + n // 2]).astype(np.int32)
    elif what == "one-way":
        adj[17, 2] = (int(adj[17, 2]) + 11) % n
    elif what == "alone":         # a vertex with no neighbour
        for u in set(adj[8999].tolist()):
            adj[u][adj[u] == 8999] = u
        adj[8999] = 8999
    else:                         # one level after the walk, then the last
        n, d = 4160, 8
        adj = G.random_regular(n, d, 4)
    adj = np.ascontiguousarray(adj, dtype=np.int32)
    r = both(monkeypatch, n, d, 4096, [full(adj, 1200)])
    if what != "ring":
        check_oracle(r, adj)


@pytest.mark.parametrize("form,args", [("part", (64, 40, 3)), ("part", (100, 30, 4)), ("part", (129, 17, 6)), ("part", (500, 12, 6)),
                                       ("part", (700, 9, 5)), ("part", (1024, 32, 12)), ("part", (1500, 11, 7)), ("part", (2500, 5, 8)),
                                       ("part", (4200, 3, 9)), ("part", (66, 500, 3)), ("piece", (16, 20, 4, 3, 8)),
                                       ("piece", (30, 33, 2, 5, 10)), ("box", (8, 4, 6, 2, 3, 2, 6)), ("halves", ()), ("one-way", ()),
                                       ("ring", ())])
def test_source_list_equals_the_level_loop(form, args, monkeypatch):
    if form == "piece":
        a = G.piece_lift(*args, 1)
        make, T = (lambda: G.cudaASPLpiece(*a[:4], args[-1])), a[4]
    elif form == "box":
        a = I.random_box(*args, 1)
        make, T = (lambda: G.cudaASPLbox(*a[:6], args[-1])), a[6]
    else:
        if form == "part":
            N, M, T = G.cyclic_lift(*args, 2)
        elif form == "halves":            # even steps only: the two residues never meet
            N, M, T = 8000, 8, np.array([[2, -2, 1000, -1000]] * 8, np.int32)
        elif form == "ring":
            N, M, T = 4000, 100, np.array([[1, -1, 2, -2]] * 100, np.int32)
        else:
            N, M, T = G.cyclic_lift(300, 11, 5, 3)
            T = T.copy()
            T[7, 2] += 1
        make = lambda: G.cudaASPLconv(N, M, T.shape[1])
    T = np.ascontiguousarray(T, dtype=np.int32)
    monkeypatch.setenv("GG_DIRECT", "0")
    out = []
    for sweep in ("0", "1"):
        monkeypatch.setenv("GG_SWEEP", sweep)
        e = make()
        out.append([e.eval(T, max_levels=cap, level_counts=True) for cap in (1100, 1100, 4)] + [e.diameterASPL(T)])
        e.close()
    for want, got in zip(*out):
        if isinstance(want, tuple):
            assert got == want
        else:
            assert all(got[k] == want[k] for k in KEYS)
            assert np.array_equal(got["level_counts"], want["level_counts"])


def test_engines_of_different_sizes_in_two_threads(monkeypatch):
    """Both engines launch the same kernels, each with shared memory for its own rows; a new
    level cap makes each call prepare its launches anew."""
    import threading
    monkeypatch.setenv("GG_DIRECT", "0")
    jobs, errors = [], []
    for n in (9000, 40000):
        adj = G.random_regular(n, 6, 1)
        jobs.append((lambda adj=adj: G.cudaASPLgraph(len(adj), 6), adj))
    for m, g in ((200, 12), (1024, 60)):
        N, M, T = G.cyclic_lift(m, g, 6, 1)
        jobs.append((lambda N=N, M=M: G.cudaASPLconv(N, M, 6), T))

    def work(make, t):
        try:
            e = make()
            seen = {(r["total"], r["reached"], r["levels"]) for r in (e.eval(t, max_levels=20 + k % 40) for k in range(120))}
            e.close()
            assert len(seen) == 1
        except Exception as x:
            errors.append(x)

    for _ in range(2):
        threads = [threading.Thread(target=work, args=j) for j in jobs]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
    assert not errors, errors


@pytest.mark.parametrize("fault", ["rows", "more_rows"])
@pytest.mark.parametrize("n,d,kind", [(10000, 4, "graph"), (17000, 6, "graph"), (20000, 8, "graph"), (12000, 8, "one-way"),
                                      (20000, 6, "list"), (20000, 6, "one-way list")])
def test_no_memory_for_the_rows_of_all_batches(n, d, kind, fault, monkeypatch):
    """The allocation that fails (on the host's side) is the sweep's own, or a larger one that
    only the general loop would need, when the sweep has its rows already."""
    monkeypatch.setenv("GG_DIRECT", "0")
    if kind.endswith("list"):
        N, M, T = G.cyclic_lift(n // 2, 2, d, 3)
        T = T.copy()
        adj, src, make = None, np.arange(M), lambda: G.cudaASPLconv(N, M, d)
    else:
        T = G.random_regular(n, d, 3)
        src, make = np.arange(n), lambda: G.cudaASPLgraph(n, d)
    if kind.startswith("one-way"):
        T[17, 2] += 1 if T[17, 2] + 1 < n else -1
    adj = O.expand_part(N, M, T) if kind.endswith("list") else T
    o = O.bfs_pull(adj, src)
    e = make()
    for inject in ("", fault, "", fault, fault):
        monkeypatch.setenv("GG_FAULT_INJECT", inject)
        r = e.eval(T)
        assert (r["total"], r["reached"], r["levels"]) == (o.total(), int(o.reached.sum()), o.levels)
    e.close()
    monkeypatch.setenv("GG_FAULT_INJECT", fault)
    e = make()
    r = e.eval(T)
    assert (r["total"], r["reached"], r["levels"]) == (o.total(), int(o.reached.sum()), o.levels)
    e.close()
