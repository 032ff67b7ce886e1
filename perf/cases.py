"""What a user of the engine has it do, as cases to time and compare.

``listed()`` names fixed cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program has in hand before the call, ``run`` is one
pass through the public entry points with its whole results, ``work`` what the
pass cannot do without and ``exact`` the result of the differentiable case in
64 bits.  Inputs are seeded and synthetic; their shapes are the benchmark
configurations of ``bench.py`` and ``gen.py`` and the test sizes around them.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "strata-k_b200"))

import strata_b200 as S  # noqa: E402
from strata_b200.torch_bridge import prov_probability  # noqa: E402

def listed():
    return [
        # reachability in a network of a few hundred nodes, called with host columns: latency
        {"name": "closure_small", "kind": "closure_host", "n": 300, "m": 701},
        # one hop-by-hop routing query against a small network, device in, host out
        {"name": "mssp_small", "kind": "mssp", "nodes": 2048, "m": 12_345, "sources": 3, "wmax": 100},
        # the Bool closure configuration: ER 10k / 50k, the relation read back
        {"name": "closure_10k", "kind": "closure_dev", "n": 10_000, "m": 50_000},
        # the headline configuration: Trop MSSP, R-MAT-20, 64 sources, read back
        {"name": "mssp_rmat20", "kind": "mssp", "nodes": 1 << 20, "m": 8 << 20, "sources": 64, "wmax": 100},
        # all-pairs costs of an ordinary network whose weights need 64 bits
        {"name": "paths_wide", "kind": "paths", "n": 1501, "m": 6007, "wmax": 1 << 40},
        # costs through a large, shallow hierarchy (the index over all pairs would not fit)
        {"name": "paths_layers", "kind": "layers", "n": 200_003, "layers": 8, "deg": 2, "wmax": 100},
        # a batch of independent closures, sizes as in the batched configuration
        {"name": "closure_batch", "kind": "batch", "instances": 192, "n_max": 50_000},
        # the triangle configuration: R-MAT-22, 16 edges a node, device columns
        {"name": "triangles_rmat22", "kind": "tri_pattern", "nodes": 1 << 22, "m": 16 << 22},
        # triangles of an ordinary undirected graph from host columns
        {"name": "triangles_host", "kind": "tri_host", "nodes": 1 << 15, "m": 400_003},
        # `?grad` of a set of queries: capture, compilation and gradient rows
        {"name": "grad_queries", "kind": "prov", "n": 10_000, "m": 40_000, "queries": 96, "k": 8},
        # a training step through compiled circuits: forward and backward
        {"name": "circuit_step", "kind": "circuit", "leaves": 80_000, "queries": 1024, "proofs": 8},
        # one delta round of a rule over the operators: join, sort, reduce, merge
        {"name": "rule_round", "kind": "round", "nodes": 500_000, "rows": 2_000_003, "deg": 4, "trop": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closure_host", "closure_dev", "mssp", "paths", "layers", "batch", "tri_pattern", "tri_host",
                       "prov", "circuit", "round"])
    if kind == "closure_host":
        n = _log(rng, 20, 3000)
        return {"kind": kind, "n": n, "m": int(n * rng.uniform(1.2, 6))}
    if kind == "closure_dev":
        n = _log(rng, 500, 10_000)
        return {"kind": kind, "n": n, "m": int(n * rng.uniform(1.2, 8))}
    if kind == "mssp":
        nodes = 1 << rng.randint(9, 20)
        return {"kind": kind, "nodes": nodes, "m": int(nodes * rng.uniform(2, 8)), "sources": rng.randint(1, 64),
                "wmax": rng.choice([100, 10_000, 1 << 40])}
    if kind == "paths":
        n = _log(rng, 50, 3000)
        return {"kind": kind, "n": n, "m": int(n * rng.uniform(1.5, 5)), "wmax": rng.choice([100, 1 << 40])}
    if kind == "layers":
        return {"kind": kind, "n": _log(rng, 60_000, 400_000), "layers": rng.randint(4, 8), "deg": rng.randint(1, 2),
                "wmax": rng.choice([100, 1 << 40])}
    if kind == "batch":
        return {"kind": kind, "instances": _log(rng, 8, 256), "n_max": _log(rng, 1000, 40_000)}
    if kind == "tri_pattern":
        nodes = 1 << rng.randint(14, 22)
        return {"kind": kind, "nodes": nodes, "m": int(nodes * rng.uniform(4, 16))}
    if kind == "tri_host":
        nodes = 1 << rng.randint(8, 16)
        return {"kind": kind, "nodes": nodes, "m": int(nodes * rng.uniform(3, 16))}
    if kind == "prov":
        n = _log(rng, 500, 10_000)
        return {"kind": kind, "n": n, "m": int(n * rng.uniform(2, 4)), "queries": _log(rng, 4, 96),
                "k": rng.randint(1, 8)}
    if kind == "circuit":
        return {"kind": kind, "leaves": _log(rng, 500, 80_000), "queries": _log(rng, 16, 1500),
                "proofs": rng.randint(2, 8)}
    nodes = _log(rng, 1000, 500_000)
    return {"kind": "round", "nodes": nodes, "rows": int(nodes * rng.uniform(1, 4)), "deg": rng.randint(1, 4),
            "trop": rng.random() < 0.6}


_eng = []


def _engine():
    """The program's one engine on the device."""
    if not _eng:
        _eng.append(S.Engine(0))
    return _eng[0]


# ---- inputs, made on the device from the seed -------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ints(g, hi, n):
    return torch.randint(0, int(hi), (int(n),), generator=g, device="cuda")


def _er(g, n, m):
    """m directed edges over n nodes without self-loops (repeats possible, as in a file)."""
    u = _ints(g, n, m)
    return u, (u + 1 + _ints(g, n - 1, m)) % n


def _ring(g, n, m):
    """A strongly connected network: a ring through all n nodes and m - n further random edges, shuffled."""
    ring = torch.randperm(n, generator=g, device="cuda")
    u, v = _er(g, n, max(0, m - n))
    u, v = torch.cat([ring, u]), torch.cat([ring.roll(-1), v])
    o = torch.randperm(len(u), generator=g, device="cuda")
    return u[o], v[o]


def _distinct(g, n, make):
    """Exactly n distinct keys of those that make(count) draws, sorted."""
    k = torch.unique(make(n + n // 8 + 64))
    while len(k) < n:
        k = torch.unique(torch.cat([k, make(n)]))
    return k[torch.randperm(len(k), generator=g, device="cuda")[:n]].sort().values


def _rmat(g, nodes, m, undirected=False):
    """About m distinct R-MAT edges (0.57, 0.19, 0.19), in a random order."""
    scale = nodes.bit_length() - 1
    need = int(m * 1.05) + 16
    u = torch.zeros(need, dtype=torch.int64, device="cuda")
    v = torch.zeros(need, dtype=torch.int64, device="cuda")
    for level in range(scale):
        r = torch.rand(need, generator=g, device="cuda")
        bit = 1 << (scale - 1 - level)
        u += (r >= 0.76).long() * bit
        v += (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() * bit
    if undirected:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    k = torch.unique(((u << 32) | v)[u != v])
    k = k[torch.randperm(len(k), generator=g, device="cuda")[:m]]
    return k >> 32, k & 0xFFFFFFFF


def _first_seen(seed_ids, *cols):
    """Symbol ids in the order a file's cells are first seen, `seed_ids` before them."""
    flat = torch.cat([seed_ids, torch.stack(cols, 1).reshape(-1)])
    uniq, inv = torch.unique(flat, return_inverse=True)
    first = torch.full((len(uniq),), len(flat), dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inv, torch.arange(len(flat), device="cuda"), "amin")
    rank = torch.empty_like(first)
    rank[torch.argsort(first)] = torch.arange(len(uniq), device="cuda")
    ids = rank[inv].to(torch.int32)
    body = ids[len(seed_ids):].reshape(-1, len(cols))
    return ids[:len(seed_ids)].contiguous(), [body[:, i].contiguous() for i in range(len(cols))]


def _none():
    return torch.zeros(0, dtype=torch.int64, device="cuda")


def _pinned(n, trop):
    """Host columns a program keeps for the results (page-locked), as many rows as there can be."""
    t = [torch.zeros(n, dtype=torch.int32, pin_memory=True) for _ in range(2)]
    if trop:
        t += [torch.zeros(n, dtype=torch.int64, pin_memory=True), torch.zeros(n, dtype=torch.uint8, pin_memory=True)]
    a = [x.numpy() for x in t]
    return t, (a[0].view(np.uint32), a[1].view(np.uint32), a[2] if trop else None, a[3] if trop else None)


def _weights(g, wmax, m):
    return 1 + _ints(g, wmax, m)


def _proof_lists(rng, leaves, queries, proofs):
    """Per query up to `proofs` path-like proofs: a path of 2..9 edges and detours of it."""
    out = []
    for _ in range(queries):
        base = rng.integers(1, leaves + 1, int(rng.integers(2, 10))).tolist()
        sets = [sorted(set(base))]
        for _ in range(int(rng.integers(0, proofs))):
            p = list(base)
            a = int(rng.integers(0, len(p)))
            b = int(rng.integers(a, min(len(p), a + 4))) + 1
            p[a:b] = rng.integers(1, leaves + 1, int(rng.integers(1, 4))).tolist()
            sets.append(sorted(set(p)))
        out.append(sets)
    return out


def _circuit_inputs(case, seed):
    rng = np.random.default_rng(seed)
    lists = _proof_lists(rng, case["leaves"], case["queries"], case["proofs"])
    p = rng.beta(2.0, 5.0, case["leaves"]).astype(np.float32)
    y = rng.random(case["queries"], dtype=np.float32)
    return lists, p, y


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "circuit":
        lists, p, y = _circuit_inputs(case, seed)
        st["circ"] = _engine().compile_circuits(lists, case["leaves"])
        st["p"] = torch.from_numpy(p).cuda().requires_grad_()
        st["y"] = torch.from_numpy(y).cuda()
        return st
    g = _gen(seed)
    if kind in ("closure_host", "closure_dev"):
        u, v = (_ring if kind == "closure_host" else _er)(g, case["n"], case["m"])
        _, (s, d) = _first_seen(_none(), u, v)
        if kind == "closure_host":
            st["s"], st["d"] = (x.cpu().numpy().view(np.uint32) for x in (s, d))
        else:
            st["s"], st["d"] = s, d
            st["keep"], st["out"] = _pinned(case["n"] ** 2, False)
    elif kind == "mssp":
        u, v = _rmat(g, case["nodes"], case["m"])
        cand = torch.unique(u)
        src = cand[torch.randperm(len(cand), generator=g, device="cuda")[:case["sources"]]]
        st["src"], (st["s"], st["d"]) = _first_seen(src, u, v)
        st["sw"] = torch.zeros(len(src), dtype=torch.int64, device="cuda")
        st["w"] = _weights(g, case["wmax"], len(u))
        st["keep"], st["out"] = _pinned(case["nodes"] * case["sources"], True)
    elif kind == "paths":
        u, v = _er(g, case["n"], case["m"])
        _, (st["s"], st["d"]) = _first_seen(_none(), u, v)
        st["w"] = _weights(g, case["wmax"], case["m"])
        st["keep"], st["out"] = _pinned(case["n"] ** 2, True)
    elif kind == "layers":
        # nodes in `layers` equal layers, `deg` edges from each node to the next layer
        per = case["n"] // case["layers"]
        u = torch.arange(per * (case["layers"] - 1), device="cuda").repeat_interleave(case["deg"])
        v = (u // per + 1) * per + _ints(g, per, len(u))
        o = torch.randperm(len(u), generator=g, device="cuda")
        _, (st["s"], st["d"]) = _first_seen(_none(), u[o], v[o])
        st["w"] = _weights(g, case["wmax"], len(u))
        top = sum(per * min(case["deg"] ** k, per) for j in range(case["layers"]) for k in range(1, case["layers"] - j))
        st["keep"], st["out"] = _pinned(top, True)
    elif kind == "batch":
        c = case["instances"]
        # node counts log-uniform, spread evenly over the range, mean out-degree uniform in 2..8
        r = (torch.arange(c, device="cuda", dtype=torch.float64) +
             torch.rand(c, generator=g, device="cuda", dtype=torch.float64)) / c
        n = torch.exp(math.log(100) + r * math.log(case["n_max"] / 100)).round().long()
        m = (n * (2 + 6 * torch.rand(c, generator=g, device="cuda"))).long()
        o = torch.randperm(c, generator=g, device="cuda")
        n, m = n[o], m[o]
        nn = n.repeat_interleave(m)
        u = (torch.rand(len(nn), generator=g, device="cuda", dtype=torch.float64) * nn).long()
        step = (torch.rand(len(nn), generator=g, device="cuda", dtype=torch.float64) * (nn - 1)).long()
        st["s"], st["d"] = u.to(torch.int32), ((u + 1 + step) % nn).to(torch.int32)
        st["nodes"] = n.cpu().numpy().astype(np.uint32)
        st["off"] = np.concatenate([[0], np.cumsum(m.cpu().numpy())]).astype(np.uint64)
    elif kind in ("tri_pattern", "tri_host"):
        u, v = _rmat(g, case["nodes"], case["m"], undirected=True)
        if kind == "tri_host":
            st["s"], st["d"] = (x.to(torch.int32).cpu().numpy().view(np.uint32) for x in (u, v))
        else:  # oriented from the lower to the higher degree, as the count's rule wants it
            deg = torch.bincount(u, minlength=case["nodes"]) + torch.bincount(v, minlength=case["nodes"])
            lo = (deg[u] < deg[v]) | ((deg[u] == deg[v]) & (u < v))
            x, y = torch.where(lo, u, v), torch.where(lo, v, u)
            _, (st["s"], st["d"]) = _first_seen(_none(), x, y)
    elif kind == "prov":
        def edges(count):
            u, v = _er(g, case["n"], count)
            return (u << 32) | v
        k = _distinct(g, case["m"], edges)
        k = k[torch.randperm(len(k), generator=g, device="cuda")]
        rng = np.random.default_rng(seed)
        p = rng.beta(2.0, 5.0, len(k)).astype(np.float32)
        st["s"], st["d"] = (k >> 32).to(torch.int32), (k & 0xFFFFFFFF).to(torch.int32)
        st["p32"], st["p64"] = torch.from_numpy(p).cuda(), torch.from_numpy(p.astype(np.float64)).cuda()
        st["qs"], st["qt"] = (rng.integers(0, case["n"], case["queries"]).astype(np.uint32) for _ in range(2))
    elif kind == "round":
        # h and its delta over (X, Y), an edge relation over (Y, Z): sorted unique keys (c0 << 32) | c1
        nodes, rows, trop = case["nodes"], case["rows"], case["trop"]

        def pairs(count):
            return (_ints(g, nodes, count) << 32) | _ints(g, nodes, count)
        h = _distinct(g, rows, pairs)
        dh = h[torch.randperm(rows, generator=g, device="cuda")[:max(1, rows // 2)]].sort().values
        y = torch.arange(nodes, device="cuda").repeat_interleave(case["deg"])
        e = torch.unique((y << 32) | _ints(g, nodes, len(y)))
        for name, k in (("h", h), ("dh", dh), ("e", e)):
            st[name], st[name + "_w"] = k, _weights(g, 1000, len(k)) if trop else None
        # the buffers a program keeps from round to round
        top = len(dh) * case["deg"]
        for name, size in (("cand", top), ("sorted", top), ("red", top), ("h_next", rows + top), ("dh_next", top)):
            st[name] = torch.zeros(size, dtype=torch.int64, device="cuda")
            st[name + "_w"] = torch.zeros(size, dtype=torch.int64, device="cuda") if trop else None
        _engine()
    else:
        raise ValueError(kind)
    return st


# ---- one pass ------------------------------------------------------------------
def _read_back(rel, out):
    n = len(rel.to_host(out))
    rel.free()
    return [n] + [x.view(np.int32) if x.dtype == np.uint32 else x for x in out if x is not None]


def _p(t):
    return None if t is None else t.data_ptr()


def _rule_round(eng, st):
    """h(X,Z) :- h(X,Y), e(Y,Z) over the changed rows dh: the caller's sequence of operators."""
    lib, ctx, vb = eng.lib, eng.ctx, 8 if st["case"]["trop"] else 0
    t, nr, nh, nd = (C.c_uint64() for _ in range(4))
    arg = {k: (_p(st[k]), _p(st[k + "_w"])) for k in ("h", "dh", "e", "cand", "sorted", "red", "h_next", "dh_next")}
    left, right = (*arg["dh"], len(st["dh"]), 32), (*arg["e"], len(st["e"]), 32)
    eng._check(lib.strata_op_join(ctx, 8, *left, *right, 32, None, None, 0, C.byref(t)))
    eng._check(lib.strata_op_join(ctx, 8, *left, *right, 32, *arg["cand"], t.value, C.byref(t)))
    eng._check(lib.strata_op_sort(ctx, 8, vb, *arg["cand"], *arg["sorted"], t.value, 64))
    eng._check(lib.strata_op_reduce(ctx, 8, *arg["sorted"], t.value, *arg["red"], C.byref(nr)))
    eng._check(lib.strata_op_merge_diff(ctx, 8, *arg["h"], len(st["h"]), *arg["red"], nr.value, *arg["h_next"],
                                        *arg["dh_next"], C.byref(nh), C.byref(nd)))
    out = [t.value, nh.value, nd.value, st["h_next"], st["dh_next"]]
    return out + [st["h_next_w"], st["dh_next_w"]] if vb else out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "circuit":
        P = prov_probability(st["p"], st["circ"])
        loss = ((P - st["y"]) ** 2).mean()
        (grad,) = torch.autograd.grad(loss, st["p"])
        return P.detach(), grad
    eng = _engine()
    if kind == "round":
        return _rule_round(eng, st)
    if kind == "closure_host":
        r = eng.transitive_closure_bool((st["s"], st["d"]))
        return r.src.view(np.int32), r.dst.view(np.int32), r.stats["rounds"]
    if kind == "closure_dev":
        return _read_back(eng.tc_bool_dev(st["s"], st["d"]), st["out"])
    if kind == "mssp":
        return _read_back(eng.mssp_dev(st["src"], st["s"], st["d"], st["w"], source_weights=st["sw"]), st["out"])
    if kind in ("paths", "layers"):
        return _read_back(eng.trop_paths_dev(st["s"], st["d"], st["w"]), st["out"])
    if kind == "batch":
        r = eng.tc_bool_batch(st["nodes"], st["off"], st["s"], st["d"])
        return r.counts.view(np.int64), r.fps.view(np.int64), r.rounds.view(np.int32)
    if kind == "tri_pattern":
        return eng.count_triangle_pattern_dev(st["s"], st["d"])
    if kind == "tri_host":
        return eng.count_triangles((st["s"], st["d"]))
    if kind == "prov":
        P, G, circ, _ = eng.grad_queries(case["n"], st["s"], st["d"], st["p64"], st["p32"], st["qs"], st["qt"],
                                         k=case["k"])
        circ.free()
        return P, G
    raise ValueError(kind)


# ---- what a pass cannot do without ------------------------------------------------
def _giant(deg):
    """Share of an ER graph's nodes in the strongly connected core's reach (mean out-degree deg)."""
    x = 0.5
    for _ in range(60):
        x = 1 - math.exp(-deg * x)
    return x


def work(case):
    kind = case["kind"]
    if kind == "circuit":  # leaves and their gradients, labels and P; a node for about each literal and branch
        nodes = case["queries"] * case["proofs"] * 20
        return {"bytes": 8 * case["leaves"] + 12 * case["queries"] + 13 * nodes, "flops": 30 * nodes}
    if kind == "closure_host":  # every node reaches every node
        return {"bytes": 8 * case["m"] + 8 * case["n"] ** 2, "flops": 0}
    if kind == "closure_dev":
        return {"bytes": 8 * case["m"] + 8 * (_giant(case["m"] / case["n"]) * case["n"]) ** 2, "flops": 0}
    if kind == "mssp":
        reach = 0.5 * case["nodes"] * min(1.0, case["m"] / (8 * case["nodes"]))
        return {"bytes": 16 * case["m"] + 17 * case["sources"] * reach, "flops": 0}
    if kind == "paths":
        return {"bytes": 16 * case["m"] + 17 * (_giant(case["m"] / case["n"]) * case["n"]) ** 2, "flops": 0}
    if kind == "layers":
        per, d, L = case["n"] // case["layers"], case["deg"], case["layers"]
        rows = sum(per * d ** k for j in range(L) for k in range(1, L - j))
        return {"bytes": 16 * per * (L - 1) * d + 17 * rows, "flops": 0}
    if kind == "batch":  # the closures stay on the device: one bit each written, the edges read
        c, lr = case["instances"], math.log(case["n_max"] / 100)
        return {"bytes": c * (5 * 8 * (case["n_max"] - 100) / lr + (case["n_max"] ** 2 - 1e4) / (2 * lr) / 8 * 0.8),
                "flops": 0}
    if kind in ("tri_pattern", "tri_host"):
        return {"bytes": 8 * case["m"], "flops": 0}
    if kind == "prov":
        return {"bytes": 20 * case["m"] + 8.0 * case["queries"] * case["m"], "flops": 0}
    row = 16 if case["trop"] else 8
    t = case["rows"] // 2 * case["deg"] * 0.79
    return {"bytes": row * (case["rows"] * 1.5 + case["nodes"] * case["deg"] + case["rows"] + 2 * t), "flops": 0}


def exact(case, seed):
    """P and the loss gradient of the training step by inclusion-exclusion over each query's proofs, in FP64."""
    if case["kind"] != "circuit":
        return None
    lists, p32, y32 = _circuit_inputs(case, seed)
    p, y = p32.astype(np.float64), y32.astype(np.float64)
    P, grad = np.zeros(len(lists)), np.zeros(len(p))
    for q, sets in enumerate(lists):
        lits = sorted({x for s in sets for x in s})
        at = np.array(lits) - 1
        member = np.array([[x in s for x in lits] for s in map(set, sets)])
        pick = (np.arange(1, 1 << len(sets))[:, None] >> np.arange(len(sets))) & 1
        union = (pick @ member) > 0
        sign = np.where(pick.sum(1) % 2 == 1, 1.0, -1.0)
        P[q] = (sign * np.where(union, p[at], 1.0).prod(1)).sum()
        dP = np.empty(len(at))
        for j in range(len(at)):
            rest = union.copy()
            rest[:, j] = False
            dP[j] = (sign * union[:, j] * np.where(rest, p[at], 1.0).prod(1)).sum()
        np.add.at(grad, at, 2 * (P[q] - y[q]) / len(lists) * dP)
    return P, grad
