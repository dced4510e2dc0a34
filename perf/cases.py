"""Cases that measure the engine through its public Python entry points.

What a search for low-ASPL graphs spends its time on: scoring one graph with a
calculator (plain, cyclic lift, 2-D torus lift), scoring a population of 2-opt
moves or of lift moves against one base, scoring one move of a large graph, and
one step of the surrogate ranker (predict a pool, train on the scored pairs).

    listed()             the cases, each a dict of plain values
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs and handles a search program holds before the call
    run(state)           one pass through the public entry points
    work(case)           bytes and operations the pass cannot do without
    exact(case, seed)    the same outputs from plain torch/numpy in 64 bits
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graphgolf-cuda_b200"))
import graphgolf as G  # noqa: E402


def listed():
    return [
        # The smallest calculator call: a hill climber on a contest-sized graph; launch latency.
        {"name": "graph_n256_d4", "kind": "graph", "n": 256, "d": 4, "ragged": False},
        # One graph that fits a single source batch.
        {"name": "graph_n4096_d16", "kind": "graph", "n": 4096, "d": 16, "ragged": False},
        # Odd size, irregular degrees (rows padded with self-loops), several source batches.
        {"name": "graph_n30011_d6_ragged", "kind": "graph", "n": 30011, "d": 6, "ragged": True},
        # The largest plain graph: the single-graph throughput workload.
        {"name": "graph_n65536_d8", "kind": "graph", "n": 65536, "d": 8, "ragged": False},
        # One symmetric (cyclic lift) graph, BFS from one vertex per orbit.
        {"name": "lift_m1024_g32_d12", "kind": "conv", "m": 1024, "g": 32, "d": 12, "wvc": False},
        # A smaller lift of odd sizes with the worst-vertex count, as the lift hill climbers call it.
        {"name": "lift_wvc_m500_g12_d6", "kind": "conv", "m": 500, "g": 12, "d": 6, "wvc": True},
        # One 2-D torus lift.
        {"name": "piece_32x32_x8x4_d8", "kind": "piece", "mx": 32, "my": 32, "kx": 8, "ky": 4, "d": 8},
        # One step of the batched annealer: a few 2-opt candidates of one graph.
        {"name": "moves32_n4096_d8", "kind": "moves", "n": 4096, "d": 8, "count": 32, "n2": 0, "d2": 0, "count2": 0},
        # A whole population over two bases of uneven size.
        {"name": "moves2048_n1024_d6_512_n3000_d4", "kind": "moves", "n": 1024, "d": 6, "count": 2048,
         "n2": 3000, "d2": 4, "count2": 512},
        # A population of lift moves.
        {"name": "liftmoves256_m1024_g32_d12", "kind": "liftmoves", "m": 1024, "g": 32, "d": 12, "count": 256},
        # One move of a large graph against its stored distances.
        {"name": "move1_n65536_d8", "kind": "move1", "n": 65536, "d": 8},
        # One surrogate step of the annealer: rank a pool of proposals, train on the scored pairs.
        {"name": "surrogate_n4096_d8_p4096_t64", "kind": "surrogate", "n": 4096, "d": 8, "pool": 4096, "train": 64},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _even(n, d):
    return n + 1 if (n * d) % 2 else n


def draw(rng):
    kind = rng.choice(["graph", "graph", "conv", "piece", "moves", "liftmoves", "move1", "surrogate"])
    if kind == "graph":
        d = rng.randint(3, 16)
        n = _log(rng, 64, 65536 if d <= 8 else 40000)
        return {"kind": kind, "n": min(_even(n, d), 65536), "d": d, "ragged": rng.random() < 0.25}
    if kind == "conv":
        g = rng.randint(2, 64)
        d = rng.randint(3, 12)
        return {"kind": kind, "m": _even(_log(rng, 64, 65536 // (g + 1)), d), "g": g, "d": d, "wvc": rng.random() < 0.4}
    if kind == "piece":
        return {"kind": kind, "mx": 2 * rng.randint(4, 20), "my": rng.randint(6, 40), "kx": rng.randint(2, 8),
                "ky": rng.randint(2, 6), "d": rng.randint(3, 10)}
    if kind == "moves":
        d = rng.randint(3, 8)
        n = _even(_log(rng, 200, 4096), d)
        count = _log(rng, 1, max(1, min(2048, 2 * 10 ** 9 // (n * n))))
        return {"kind": kind, "n": n, "d": d, "count": count, "n2": 0, "d2": 0, "count2": 0}
    if kind == "liftmoves":
        d = rng.randint(4, 12)
        g = rng.randint(4, 32)
        m = _even(_log(rng, 64, 1023), d)
        return {"kind": kind, "m": m, "g": g, "d": d, "count": rng.randint(8, 256)}
    if kind == "move1":
        return {"kind": kind, "n": 2 * _log(rng, 1000, 32768), "d": rng.randint(5, 8)}
    return {"kind": kind, "n": 2 * _log(rng, 256, 4096), "d": rng.randint(4, 8), "pool": _log(rng, 128, 4096),
            "train": rng.randint(16, 128)}


# ---- inputs --------------------------------------------------------------------

def _ragged(adj, seed):
    """About 1 % of the edges left out: both ends' slots become self-loops (padding)."""
    adj = adj.copy()
    n, d = adj.shape
    rng = np.random.default_rng(seed)
    for v in rng.choice(n, max(1, n * d // 200), replace=False):
        u = int(adj[v, rng.integers(d)])
        if u == v or (adj[v] != v).sum() <= 2 or (adj[u] != u).sum() <= 2:
            continue
        adj[v, np.nonzero(adj[v] == u)[0][0]] = v
        adj[u, np.nonzero(adj[u] == v)[0][0]] = u
    return adj


def _inputs(case, seed):
    k = case["kind"]
    if k == "graph":
        adj = G.random_regular(case["n"], case["d"], seed + 1)
        return {"adj": _ragged(adj, seed) if case["ragged"] else adj}
    if k == "conv":
        N, M, t = G.cyclic_lift(case["m"], case["g"], case["d"], seed + 1)
        return {"N": N, "M": M, "table": t}
    if k == "piece":
        nx, ny, mx, my, t = G.piece_lift(case["mx"], case["my"], case["kx"], case["ky"], case["d"], seed + 1)
        return {"dims": (nx, ny, mx, my), "table": t}
    if k == "moves":
        bases = [G.random_regular(case["n"], case["d"], seed + 1)]
        moves = [G.gen_swaps(bases[0], 0, case["count"], seed + 2)]
        if case["count2"]:
            bases.append(G.random_regular(case["n2"], case["d2"], seed + 3))
            moves.append(G.gen_swaps(bases[1], 1, case["count2"], seed + 4))
        return {"bases": bases, "moves": np.concatenate(moves)}
    if k == "liftmoves":
        N, M, t = G.cyclic_lift(case["m"], case["g"], case["d"], seed + 1)
        return {"N": N, "M": M, "table": t, "moves": G.gen_lift_moves(N, M, t, case["count"], seed + 2)}
    if k == "move1":
        adj = G.random_regular(case["n"], case["d"], seed + 1)
        return {"adj": adj, "move": G.gen_swaps(adj, 0, 1, seed + 2)[0]}
    adj = G.random_regular(case["n"], case["d"], seed + 1)
    rng = np.random.default_rng(seed)
    feats = np.concatenate([rng.standard_normal((case["n"], 4)), np.ones((case["n"], 1))], axis=1).astype(np.float32)
    params = []   # W_in, b_in, {Ws, Wn, b} x 3, Wr1, br1, wr2, br2: Glorot uniform, zero biases
    for fin, fout, bias in ([(5, 64, True)] + [(64, 64, False), (64, 64, True)] * 3 + [(192, 64, True), (64, 1, True)]):
        a = np.sqrt(6.0 / (fin + fout))
        params.append(rng.uniform(-a, a, fin * fout))
        if bias:
            params.append(np.zeros(fout))
    return {"adj": adj, "feats": feats, "params": np.concatenate(params).astype(np.float32),
            "pool": G.gen_swaps(adj, 0, case["pool"], seed + 2), "pairs": G.gen_swaps(adj, 0, case["train"], seed + 3),
            "target": rng.standard_normal(case["train"]).astype(np.float32)}


def prepare(case, seed):
    x, k = _inputs(case, seed), case["kind"]
    s = {"kind": k, "x": x}
    if k == "graph":
        s["calc"] = G.cudaASPLgraph(case["n"], case["d"])
    elif k == "conv":
        s["calc"] = G.cudaASPLconv(x["N"], x["M"], case["d"])
        s["wvc"] = case["wvc"]
    elif k == "piece":
        s["calc"] = G.cudaASPLpiece(*x["dims"], case["d"])
    elif k == "moves":
        s["batch"] = G.Batch()
        for adj in x["bases"]:
            s["batch"].add_base(adj)
    elif k == "liftmoves":
        s["lift"] = G.Lift(x["N"], x["M"], case["d"])
        s["lift"].set_base(x["table"])
    elif k == "move1":
        s["inc"] = G.Incremental(case["n"], case["d"])
        s["inc"].set_graph(x["adj"])
    else:
        s["net"] = G.Surrogate(case["n"], case["d"], 5)
        s["net"].set_params(x["params"])
        s["net"].set_graph(x["adj"], x["feats"])
    return s


def _fields(res):
    return {f: res[f].astype(np.int64) for f in ("total", "reached", "levels", "connected")}


def run(state):
    x, k = state["x"], state["kind"]
    if k == "graph":
        diam, total = state["calc"].calc(x["adj"])
        return {"diameter": diam, "total": total}
    if k == "conv":
        if state["wvc"]:
            wvc, diam, aspl = state["calc"].WVCdiameterASPL(x["table"])
            return {"wvc": wvc, "diameter": diam, "aspl": aspl}
        diam, aspl = state["calc"].diameterASPL(x["table"])
        return {"diameter": diam, "aspl": aspl}
    if k == "piece":
        diam, aspl = state["calc"].diameterASPL(x["table"])
        return {"diameter": diam, "aspl": aspl}
    if k == "moves":
        return _fields(state["batch"].eval(x["moves"]))
    if k == "liftmoves":
        res = state["lift"].eval(x["moves"])
        return dict(_fields(res), aspl=state["lift"].aspl(res))
    if k == "move1":
        res, searched = state["inc"].eval(x["move"])
        return dict(res, searched=searched)
    pred = state["net"].predict(x["pool"])
    loss = state["net"].train(x["pairs"], x["target"], lr=2e-3)
    return {"pred": pred, "loss": loss, "params": state["net"].get_params()}


# ---- work ----------------------------------------------------------------------

def work(case):
    """Each input read once and each output written once; operations: one per
    (source, edge) of a breadth-first search, 2 per multiply-add of the network."""
    k = case["kind"]
    if k == "graph":
        return {"bytes": 4.0 * case["n"] * case["d"] + 16, "flops": float(case["n"]) ** 2 * case["d"] / 32}
    if k == "conv":
        return {"bytes": 4.0 * case["m"] * case["d"] + 24, "flops": float(case["m"]) ** 2 * case["g"] * case["d"] / 32}
    if k == "piece":
        m = case["mx"] * case["my"]
        return {"bytes": 8.0 * m * case["d"] + 16, "flops": float(m) ** 2 * case["kx"] * case["ky"] * case["d"] / 32}
    if k == "moves":
        # the two distance rows of each move's four endpoints, and its result
        return {"bytes": sum(c * (4.0 * n + 48) + 4.0 * n * d for n, d, c in
                             ((case["n"], case["d"], case["count"]), (case["n2"], case["d2"], case["count2"]))),
                "flops": 0.0}
    if k == "liftmoves":
        return {"bytes": case["count"] * (4.0 * case["m"] * case["g"] + 92) + 4.0 * case["m"] * case["d"], "flops": 0.0}
    if k == "move1":
        return {"bytes": 4.0 * case["n"] + 4.0 * case["n"] * case["d"], "flops": 0.0}
    n, P, T = case["n"], case["pool"], case["train"]
    fwd = 2.0 * (n * 5 * 64 + 3 * n * 128 * 64 + P * 193 * 64)
    bwd = 4.0 * (n * 5 * 64 + 3 * n * 128 * 64 + T * 193 * 64)
    return {"bytes": 4.0 * n * (case["d"] + 5) + 28.0 * P + 4 * 37569.0 * 6, "flops": fwd + bwd}


# ---- the same outputs in 64 bits, from plain torch ---------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _popcount(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    return int(((x * 0x0101010101010101) >> 56).sum())


def _bfs(adj, sources):
    """Ordered pairs first reached at each level from `sources` over the rows of adj
    (a tensor [n, d]): 64 sources a word, at most 4096 at once."""
    n, d = adj.shape
    counts = [0]
    for lo in range(0, len(sources), 4096):
        src = sources[lo:lo + 4096]
        W = (len(src) + 63) // 64
        V = torch.zeros((n, W), dtype=torch.int64, device=adj.device)
        j = torch.arange(len(src), device=adj.device)
        V[src, j // 64] = torch.bitwise_left_shift(torch.ones_like(j), j % 64)   # sources are distinct vertices
        seen, L = len(src), 0
        counts[0] += seen
        while True:
            X = V.clone()
            for i in range(d):
                X |= V[adj[:, i]]
            now = _popcount(X)
            if now == seen:
                break
            L += 1
            if L == len(counts):
                counts.append(0)
            counts[L] += now - seen
            seen, V = now, X
    return counts


def _result(counts, pairs):
    reached = sum(counts)
    return {"total": sum(L * c for L, c in enumerate(counts)), "reached": reached, "levels": len(counts) - 1,
            "connected": int(reached == pairs)}


def _expand_conv(N, M, t, dev):
    v = torch.arange(N, device=dev)
    return (v[:, None] + torch.as_tensor(t, device=dev).long()[v % M]) % N


def _stack(rows):
    return {f: np.array([r[f] for r in rows], dtype=np.int64) for f in ("total", "reached", "levels", "connected")}


def exact(case, seed):
    x, k, dev = _inputs(case, seed), case["kind"], _dev()
    if k == "graph":
        adj = torch.as_tensor(x["adj"], device=dev).long()
        r = _result(_bfs(adj, torch.arange(len(adj), device=dev)), len(adj) ** 2)
        return {"diameter": r["levels"] if r["connected"] else -1, "total": r["total"] if r["connected"] else -1}
    if k in ("conv", "piece"):
        if k == "conv":
            N, M = x["N"], x["M"]
            adj, src = _expand_conv(N, M, x["table"], dev), torch.arange(M, device=dev)
        else:
            nx, ny, mx, my = x["dims"]
            N, M = nx * ny, mx * my
            v = torch.arange(N, device=dev)
            vx, vy = v // ny, v % ny
            t = torch.as_tensor(x["table"], device=dev).long()[(vx % mx) * my + vy % my]
            adj = (vx[:, None] + t[:, :, 0]) % nx * ny + (vy[:, None] + t[:, :, 1]) % ny
            m = torch.arange(M, device=dev)
            src = (m // my) * ny + m % my
        r = _result(_bfs(adj, src), M * N)
        aspl = float(r["total"] * (N // M)) / (N * (N - 1))
        out = {"diameter": r["levels"], "aspl": aspl}
        return {**out, "wvc": None} if case.get("wvc") else out
    if k == "moves":
        rows = []
        for s in x["moves"]:
            adj = torch.as_tensor(G.apply_swap(x["bases"][s["base"]], s), device=dev).long()
            rows.append(_result(_bfs(adj, torch.arange(len(adj), device=dev)), len(adj) ** 2))
        return _stack(rows)
    if k == "liftmoves":
        N, M, rows = x["N"], x["M"], []
        for e in x["moves"]:
            adj = _expand_conv(N, M, G.apply_lift_edit(x["table"], e), dev)
            rows.append(_result(_bfs(adj, torch.arange(M, device=dev)), M * N))
        out = _stack(rows)
        aspl = np.where(out["connected"] == 1, out["total"].astype(np.float64) * (N // M) / (N * (N - 1.0)), np.inf)
        return {**out, "aspl": aspl}
    if k == "move1":
        adj = torch.as_tensor(G.apply_swap(x["adj"], x["move"]), device=dev).long()
        return {**_result(_bfs(adj, torch.arange(len(adj), device=dev)), len(adj) ** 2), "searched": None}
    return _exact_surrogate(x, dev)


def _exact_surrogate(x, dev):
    p = torch.as_tensor(x["params"], device=dev).double().requires_grad_(True)
    adj, X = torch.as_tensor(x["adj"], device=dev).long(), torch.as_tensor(x["feats"], device=dev).double()
    at = [0]

    def take(*shape):
        n = int(np.prod(shape))
        at[0] += n
        return p[at[0] - n:at[0]].reshape(shape)

    H = torch.relu(X @ take(5, 64) + take(64))
    for _ in range(3):
        Ws, Wn, b = take(64, 64), take(64, 64), take(64)
        H = torch.relu(H @ Ws + H[adj].mean(1) @ Wn + b)
    Wr1, br1, wr2, br2 = take(192, 64), take(64), take(64, 1), take(1)

    def readout(sw):
        ix = {f: torch.as_tensor(np.ascontiguousarray(sw[f]), device=dev).long() for f in ("a", "b", "c", "d", "mode")}
        P = torch.where(ix["mode"] != 0, ix["d"], ix["c"])
        Q = torch.where(ix["mode"] != 0, ix["c"], ix["d"])
        a, b, c, d = (H[ix[f]] for f in ("a", "b", "c", "d"))
        z = torch.cat([a + b + c + d, a * b + c * d, a * H[P] + b * H[Q]], dim=1)
        return (torch.relu(z @ Wr1 + br1) @ wr2 + br2)[:, 0]

    with torch.no_grad():
        pred = readout(x["pool"])
    loss = ((readout(x["pairs"]) - torch.as_tensor(x["target"], device=dev).double()) ** 2).mean()
    g, = torch.autograd.grad(loss, p)
    # the first Adam step: m / (1 - beta1) = g, v / (1 - beta2) = g * g
    new = p.detach() - 2e-3 * g / (g.abs() + 1e-8)
    return {"pred": pred.cpu(), "loss": float(loss.detach()), "params": new.cpu()}
