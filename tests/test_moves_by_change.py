"""Moves scored from what they change: lift moves (csrc/gg_delta.cuh, gg_lift.cu) and
single moves of a plain graph (csrc/gg_inc.cu).

CPU: the orbits followed and the weights, restated in numpy, give every edited lift's exact
counts.  GPU: forms (part, 2-D, 3-D torus), degrees with and without an unrolled row, one
copy and many, small and odd sizes, edits that do not keep the lift symmetric, level caps,
and a new base table, against the oracle; single moves at group edges, with repeated edges
and with few pairs at the diameter."""
import time

import numpy as np
import pytest

import graphgolf as G
import instances as I
import oracle as O


def rows_from(adj, srcs):
    """Distances [len(srcs), n] by the pull rule (99: not reached)."""
    D = np.full((len(srcs), len(adj)), 99, dtype=np.int64)
    D[np.arange(len(srcs)), srcs] = 0
    for L in range(1, len(adj) + 1):
        new = (D[:, adj] == L - 1).any(axis=2) & (D == 99)
        if not new.any():
            break
        D[new] = L
    return D


@pytest.mark.parametrize("m,g,d,seed", [(24, 5, 4, 1), (30, 1, 5, 2), (16, 8, 3, 3), (40, 2, 6, 4)])
def test_orbits_near_the_edit_see_every_change(m, g, d, seed):
    N, M, T = G.cyclic_lift(m, g, d, seed)
    reps = np.arange(M)
    D = rows_from(O.expand_part(N, M, T), reps)
    radius = (int(D.max()) - 1) // 2
    for e in G.gen_lift_moves(N, M, T, 40, seed):
        Dn = rows_from(O.expand_part(N, M, G.apply_lift_edit(T, e)), reps)
        P = np.zeros(M, dtype=bool)
        for o in e["row"][:e["count"]]:
            P[np.nonzero(D[o] <= radius)[0] % M] = True
        w = np.where(P[np.arange(N) % M], 1, 2)
        ok = Dn != 99
        hist = np.bincount(D.ravel(), minlength=100).astype(np.int64)
        for r in np.nonzero(P)[0]:
            np.add.at(hist, Dn[r], w)
            np.add.at(hist, D[r], -w)
        assert np.array_equal(hist, np.bincount(Dn.ravel(), minlength=100))
        assert ok.sum() == hist[:99].sum()


def expand(form, dims, t):
    if form == "part":
        return O.expand_part(dims[0], dims[1], t), np.arange(dims[1])
    ax = 2 if form == "piece" else 3
    n, m = dims[:ax], dims[ax:]
    N = int(np.prod(n))
    x = np.array(np.unravel_index(np.arange(N), n))
    o = np.ravel_multi_index([x[j] % m[j] for j in range(ax)], m)
    to = [(x[j][:, None] + t[o][:, :, j]) % n[j] for j in range(ax)]
    src = np.array(np.unravel_index(np.arange(int(np.prod(m))), m))
    return np.ravel_multi_index(to, n), np.ravel_multi_index(list(src), n)


def lifts():
    out = {}
    for name, (m, g, d, seed) in {"g8": (64, 8, 6, 1), "g1": (130, 1, 5, 2), "d3": (66, 7, 3, 3), "d12": (90, 6, 12, 4),
                                  "d17": (80, 3, 17, 5), "small": (8, 3, 3, 6), "m129": (130, 9, 4, 7),
                                  "d16": (200, 3, 16, 8)}.items():
        # (high degrees: two lifts of the same orbits together)
        parts = [G.cyclic_lift(m, g, k, seed + k) for k in ((d,) if d <= 12 else (d - 7, 7))]
        N, M, T = parts[0][0], parts[0][1], np.concatenate([p[2] for p in parts], axis=1)
        out[name] = ("part", (N, M), T, lambda n, s, N=N, M=M, T=T: G.gen_lift_moves(N, M, T, n, s))
    Nx, Ny, Mx, My, T = G.piece_lift(3, 4, 7, 6, 5, 2)
    out["piece"] = ("piece", (Nx, Ny, Mx, My), T,
                    lambda n, s, a=(Nx, Ny, Mx, My, T): G.gen_piece_moves(*a, n, s))
    Nx, Ny, Mx, My, T = G.piece_lift(4, 6, 3, 3, 15, 3)
    out["piece_d15"] = ("piece", (Nx, Ny, Mx, My), T,
                        lambda n, s, a=(Nx, Ny, Mx, My, T): G.gen_piece_moves(*a, n, s))
    for seed in range(20):   # a box without loops or repeated edges
        B = I.random_box(3, 2, 2, 2, 3, 2, 4, seed)
        nx, ny, nz, mx, my, mz, T = B
        adj, src = expand("box", (nx, ny, nz, mx, my, mz), T)
        if all(len(set(r)) == 4 and v not in r for v, r in enumerate(adj.tolist())) and \
                O.bfs_pull(adj, src).connected:
            out["box"] = ("box", (nx, ny, nz, mx, my, mz), T,
                          lambda n, s, a=B: G.gen_box_moves(*a, n, s))
            break
    return out


def handle(form, dims, deg):
    return G.Lift(*dims, deg) if form == "part" else (G.Lift.piece if form == "piece" else G.Lift.box)(*dims, deg)


def want(form, dims, t):
    adj, src = expand(form, dims, t)
    r = O.bfs_pull(adj, src)
    return r.total(), int(r.reached.sum()), r.levels, int(r.connected)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(lifts()))
def test_lift_moves_by_change_equal_the_oracle(name, monkeypatch):
    form, dims, T, gen = lifts()[name]
    deg, ax = T.shape[1], 1 if T.ndim == 2 else T.shape[2]
    L = handle(form, dims, deg)
    L.set_base(T)
    moves = gen(20, 3)
    odd = np.zeros(4, dtype=G.LIFT_EDIT_DTYPE)    # [0]: the base itself
    odd[1]["count"], odd[1]["row"][0], odd[1]["diff"][0][0] = 1, 1, 3           # one-way
    odd[2] = moves[0]
    odd[2]["diff"][0][:ax] += 1                                                 # one end moved
    odd[3]["count"], odd[3]["diff"][1][0] = 2, 5                                # one slot twice
    moves = np.concatenate([moves, odd])
    res = L.eval(moves)
    for e, got in zip(moves, res):
        assert (int(got["total"]), int(got["reached"]), int(got["levels"]), int(got["connected"])) == \
            want(form, dims, G.apply_lift_edit(T, e)), (name, e)
    # a level cap, a few candidates of a new base, and the search of every candidate
    for cap in (2, 5):
        monkeypatch.setenv("GG_LIFT_SEARCH", "1")
        S = handle(form, dims, deg)
        S.set_base(T)
        assert L.eval(moves, max_levels=cap).tobytes() == S.eval(moves, max_levels=cap).tobytes()
        assert S.eval(moves).tobytes() == res.tobytes()
        S.close()
        monkeypatch.delenv("GG_LIFT_SEARCH")
    T2 = G.apply_lift_edit(T, moves[1])
    L.set_base(T2)
    for part in (moves[4:6], moves[4:12]):
        for e, got in zip(part, L.eval(part)):
            w = want(form, dims, G.apply_lift_edit(T2, e))
            assert (int(got["total"]), int(got["reached"]), int(got["levels"]), int(got["connected"])) == w
    L.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(lifts()))
def test_every_population_by_change_equals_the_oracle(name, monkeypatch):
    """GG_LIFT_SEARCH=0: no population is too small, no change likely to outgrow the lists."""
    monkeypatch.setenv("GG_LIFT_SEARCH", "0")
    form, dims, T, gen = lifts()[name]
    L = handle(form, dims, T.shape[1])
    for k in range(2):
        L.set_base(T)
        for moves in (gen(1, k), gen(9, 5 + k)):
            for e, got in zip(moves, L.eval(moves)):
                assert (int(got["total"]), int(got["reached"]), int(got["levels"]), int(got["connected"])) == \
                    want(form, dims, G.apply_lift_edit(T, e))
        T = G.apply_lift_edit(T, moves[0])
    L.close()


@pytest.mark.gpu
@pytest.mark.parametrize("m,g,d,n", [(130, 5, 6, 128), (200, 15, 4, 200)])
def test_populations_before_and_after_the_base_is_followed_agree(m, g, d, n):
    """The first populations of a base are searched, the later ones go by change."""
    N, M, T = G.cyclic_lift(m, g, d, 2)
    moves = G.gen_lift_moves(N, M, T, n, 3)
    L = G.Lift(N, M, d)
    L.set_base(T)
    first = L.eval(moves)
    assert all(L.eval(moves).tobytes() == first.tobytes() for _ in range(4))
    for e, got in zip(moves[:6], first):
        assert (int(got["total"]), int(got["reached"]), int(got["levels"]), int(got["connected"])) == \
            want("part", (N, M), G.apply_lift_edit(T, e))
    L.close()


@pytest.mark.gpu
@pytest.mark.parametrize("m,g,d,n", [(500, 12, 6, 32), (418, 23, 4, 256), (64, 8, 4, 8)])
def test_population_on_a_new_base_takes_no_longer_than_its_search(m, g, d, n, monkeypatch):
    """An annealer's step: a new base, then a population.  (Least of many, both in turn.)"""
    N, M, T = G.cyclic_lift(m, g, d, 1)
    moves = G.gen_lift_moves(N, M, T, n, 3)
    monkeypatch.setenv("GG_LIFT_SEARCH", "1")
    S = G.Lift(N, M, d)
    monkeypatch.delenv("GG_LIFT_SEARCH")
    L = G.Lift(N, M, d)
    best = {S: 1e9, L: 1e9}
    for k in range(200):
        for h in (S, L):
            t = time.perf_counter()
            h.set_base(T)
            h.eval(moves)
            best[h] = min(best[h], time.perf_counter() - t)
        if k >= 39 and best[L] < 1.25 * best[S]:    # (longer where the host was busy)
            break
    assert best[L] < 1.25 * best[S], best
    S.close()
    L.close()


@pytest.mark.gpu
def test_lift_bases_outside_the_change_path():
    N, M = 200, 4                                   # a cycle: diameter 100
    T = np.array([[1, -1]] * M, np.int32)
    N2, M2 = 64, 8                                  # two cycles: disconnected
    T2 = np.array([[2, -2]] * M2, np.int32)
    N3, M3, T3 = G.cyclic_lift(40, 5, 4, 9)         # one-way entry
    T3 = T3.copy()
    T3[3, 1] += 7
    for n, m, t in ((N, M, T), (N2, M2, T2), (N3, M3, T3)):
        L = G.Lift(n, m, t.shape[1])
        L.set_base(t)
        ed = np.zeros(6, dtype=G.LIFT_EDIT_DTYPE)
        ed[1]["count"], ed[1]["diff"][0][0] = 1, 5
        for e, got in zip(ed, L.eval(ed)):
            w = want("part", (n, m), G.apply_lift_edit(t, e))
            assert (int(got["total"]), int(got["reached"]), int(got["levels"]), int(got["connected"])) == w
        L.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["n33", "n1023", "n1025", "n700_d7", "cycle28", "hypercube", "multi", "n4100"])
def test_single_moves_near_the_edit_equal_the_oracle(name):
    adj = {"n33": lambda: G.random_regular(33, 4, 1), "n1023": lambda: G.random_regular(1023, 4, 2),
           "n1025": lambda: G.random_regular(1025, 6, 3), "n700_d7": lambda: G.random_regular(700, 7, 4),
           "cycle28": lambda: I.cycle(28), "hypercube": lambda: I.hypercube(7),
           "multi": lambda: I.random_regular_np(120, 5, 5), "n4100": lambda: G.random_regular(4100, 8, 6)}[name]()
    adj = np.asarray(adj, dtype=np.int32)
    n, deg = adj.shape
    inc = G.Incremental(n, deg)
    inc.set_graph(adj)
    rng = np.random.default_rng(3)
    for k in range(24):
        while True:
            a, c = rng.integers(n, size=2)
            b, d = adj[a, rng.integers(deg)], adj[c, rng.integers(deg)]
            if len({int(a), int(b), int(c), int(d)}) == 4:
                break
        s = np.array([(0, a, b, c, d, k % 2)], dtype=G.SWAP_DTYPE)[0]
        got, _ = inc.eval(s)
        r = O.bfs_pull(G.apply_swap(adj, s), np.arange(n))
        assert (got["total"], got["reached"], got["levels"], bool(got["connected"])) == \
            (r.total(), int(r.reached.sum()), r.levels, bool(r.connected)), (name, s)
    inc.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["part", "piece"])
def test_lift_handles_of_different_sizes_take_turns(form, monkeypatch):
    """The second handle's rows are shorter than the first one's; both use one kernel."""
    monkeypatch.setenv("GG_LIFT_SEARCH", "0")
    if form == "part":
        lifts2 = [G.cyclic_lift(m, g, 12, 3) for m, g in ((512, 64), (250, 4))]
        lifts2 = [((N, M), T, G.gen_lift_moves(N, M, T, 6, 4)) for N, M, T in lifts2]
    else:
        lifts2 = [G.piece_lift(*a, 8, 3) for a in ((16, 16, 16, 8), (8, 8, 4, 4))]
        lifts2 = [(tuple(a[:4]), a[4], G.gen_piece_moves(*a, 6, 4)) for a in lifts2]
    handles = []
    for dims, T, _ in lifts2:
        handles.append(handle(form, dims, T.shape[1]))
        handles[-1].set_base(T)
    truth = [[want(form, dims, G.apply_lift_edit(T, e)) for e in moves] for dims, T, moves in lifts2]
    for _ in range(2):
        for L, (_, _, moves), w in zip(handles, lifts2, truth):
            got = L.eval(moves)
            assert [(int(x["total"]), int(x["reached"]), int(x["levels"]), int(x["connected"])) for x in got] == w
    for L in handles:
        L.close()


def twin_trees(b, depth):
    """Two b-ary trees of the given depth with their roots joined, padded with self-loops:
    b^(2 depth) pairs at the diameter 2 depth + 1 each way, all of them through one edge."""
    size = (b ** (depth + 1) - 1) // (b - 1)
    v = np.arange(size)
    kids = v[:, None] * b + 1 + np.arange(b)
    adj = np.concatenate([np.maximum((v - 1) // b, 0)[:, None], np.where(kids < size, kids, v[:, None])], axis=1)
    adj = np.concatenate([adj, adj + size]).astype(np.int32)
    adj[0, 0], adj[size, 0] = size, 0
    return adj, size


@pytest.mark.gpu
@pytest.mark.parametrize("b,depth", [(3, 4), (5, 7)])      # (5, 7): 1.2e10 pairs at the diameter
def test_single_move_that_takes_all_pairs_at_the_diameter_apart(b, depth):
    adj, size = twin_trees(b, depth)
    n = len(adj)
    inc = G.Incremental(n, b + 1)
    assert inc.set_graph(adj)["levels"] == 2 * depth + 1
    # the edge between the roots, and one between a child and a grandchild of the first
    s = np.array([(0, 0, size, 1, b + 1, 0)], dtype=G.SWAP_DTYPE)[0]
    got, _ = inc.eval(s)
    inc.close()
    left = size - (b ** (depth - 1) - 1) // (b - 1)             # less the grandchild's subtree
    right = n - left
    assert (got["levels"], got["connected"], got["reached"]) == (2 * depth, 0, left * left + right * right)
    if n < 1000:
        o = O.bfs_pull(G.apply_swap(adj, s), np.arange(n))
        assert (got["total"], got["reached"], got["levels"]) == (o.total(), int(o.reached.sum()), o.levels)
