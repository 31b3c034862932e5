"""What the library is timed on: its own workloads, through its public entry points.

A case is a graph family with its size and the call that a program makes on it.
The families and the listed sizes are those of the benchmark and the tests:
R-MAT (0.57, 0.19, 0.19, 0.05), directed 2-D kNN with random vertex ids, and
the randomly oriented grid.  Graphs are generated on the GPU from the seed.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "parallel-strong-connectivity_gb300"))
import psc  # noqa: E402

LOW = 0xFFFFFFFF


def listed():
    return [
        # the smallest graphs that tests and smoke runs solve: launches and waits
        {"name": "scc_rmat12", "op": "scc", "graph": "rmat", "n": 1 << 12, "draws": 1 << 15},
        # one ordinary small graph (the benchmark's C1)
        {"name": "scc_rmat16", "op": "scc", "graph": "rmat", "n": 1 << 16, "draws": 1 << 20},
        # large-diameter graphs (the benchmark's C2): point sets and road-like grids
        {"name": "scc_knn7", "op": "scc", "graph": "knn", "n": 10_000_000},
        {"name": "scc_grid4096", "op": "scc", "graph": "grid", "rows": 4096, "cols": 4096},
        # the largest graph for one GPU (the benchmark's headline, C3)
        {"name": "scc_rmat26", "op": "scc", "graph": "rmat", "n": 1 << 26, "draws": 1 << 30},
        # a graph in host memory: upload, transpose on the device, solve, labels back
        {"name": "load_scc_rmat22", "op": "load_scc", "graph": "rmat", "n": 1 << 22, "draws": 1 << 26},
        # many independent graphs in one call (the benchmark's C4, fewer and smaller members)
        {"name": "batch_256", "op": "batch", "graph": "mix", "count": 256, "log2_max": 16},
        # connected components of a social-network-like and of a spatial graph
        {"name": "cc_rmat24", "op": "cc", "graph": "rmat", "n": 15_000_001, "draws": 1 << 28},
        {"name": "cc_knn6", "op": "cc", "graph": "knn", "n": 1_000_003},
        # LE-lists (distance sketches) of a symmetrised R-MAT graph
        {"name": "lelist_rmat20", "op": "lelist", "graph": "rmat", "n": 1 << 20, "draws": 1 << 24},
        # hop distances on a road-like graph
        {"name": "bfs_grid", "op": "bfs", "graph": "grid", "rows": 1021, "cols": 2043},
        # backward reachability on the caller's own device arrays, nothing allocated
        {"name": "reach_knn", "op": "reach", "graph": "knn", "n": 1_500_001, "dir": 1},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["scc", "scc", "scc", "load_scc", "load_cc", "batch", "cc", "lelist", "bfs", "reach"])
    if op == "batch":
        return {"op": op, "graph": "mix", "count": log_int(16, 256), "log2_max": rng.randint(12, 16)}
    family = rng.choice({"scc": ["rmat", "knn", "grid"], "bfs": ["rmat", "knn", "grid"],
                         "reach": ["rmat", "knn", "grid"], "lelist": ["rmat", "rmat", "knn"],
                         "cc": ["rmat", "knn", "grid"]}.get(op, ["rmat", "knn", "grid"]))
    case = {"op": op, "graph": family}
    top = {"scc": {"rmat": 1 << 24, "knn": 10_000_000, "grid": 1 << 24},
           "load_scc": {"rmat": 1 << 22, "knn": 1 << 22, "grid": 1 << 22},
           "load_cc": {"rmat": 1 << 22, "knn": 1 << 22, "grid": 1 << 22},
           "cc": {"rmat": 1 << 24, "knn": 1 << 23, "grid": 1 << 23},
           "lelist": {"rmat": 1 << 20, "knn": 1 << 15, "grid": 1 << 15},
           "bfs": {"rmat": 1 << 23, "knn": 1 << 21, "grid": 1 << 21},
           "reach": {"rmat": 2_000_000, "knn": 1_500_001, "grid": 2_000_000}}[op][family]
    n = log_int(4001, top)
    if family == "grid":
        case["rows"] = max(3, int(math.sqrt(n) * rng.uniform(0.4, 1.0)))
        case["cols"] = max(3, n // case["rows"])
    else:
        case["n"] = n
        if family == "rmat":
            case["draws"] = n * rng.choice([4, 8, 16])
    if op in ("scc", "load_scc") and rng.random() < 0.3:
        case["beta"] = rng.choice([1.2, 2.0, 3.0])
    if op == "reach":
        case["dir"] = rng.randint(0, 1)
    return case


# -- graphs -----------------------------------------------------------------
def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rmat_keys(n, draws, rng):
    bits = max(1, (n - 1).bit_length())
    out = []
    for start in range(0, draws, 1 << 26):
        c = min(1 << 26, draws - start)
        key = torch.zeros(c, dtype=torch.int64, device="cuda")
        r = torch.empty(c, dtype=torch.float32, device="cuda")
        for level in range(bits):
            r.uniform_(generator=rng)
            u = r >= 0.76
            v = (r >= 0.57) & ((r < 0.76) | (r >= 0.95))
            key |= (u.to(torch.int64) << (32 + bits - 1 - level)) | (v.to(torch.int64) << (bits - 1 - level))
        u, v = key >> 32, key & LOW
        out.append(key[(u != v) & (u < n) & (v < n)])
    return torch.cat(out) if len(out) > 1 else out[0]


def _knn_keys(n, rng, k=5):
    xy = torch.rand(n, 2, generator=rng, device="cuda")
    side = max(1, math.isqrt(n // 2))
    cell = (xy * side).long().clamp_(max=side - 1)
    cid = cell[:, 1] * side + cell[:, 0]
    cid, order = torch.sort(cid)
    start = torch.searchsorted(cid, torch.arange(side * side + 1, device="cuda"))
    xs, cell = xy[order], cell[order]
    width = torch.arange(20, device="cuda")
    out = []
    for a in range(0, n, 1 << 20):
        b = min(n, a + (1 << 20))
        cx, cy = cell[a:b, 0], cell[a:b, 1]
        cand, ok = [], []
        for dy in (-1, 0, 1):
            y = cy + dy
            row = y.clamp(0, side - 1) * side
            lo = start[row + (cx - 1).clamp(min=0)]
            hi = start[row + (cx + 1).clamp(max=side - 1) + 1]
            c = lo[:, None] + width
            ok.append((c < hi[:, None]) & ((y >= 0) & (y < side))[:, None])
            cand.append(c)
        cand, ok = torch.cat(cand, 1), torch.cat(ok, 1)
        ok &= cand != torch.arange(a, b, device="cuda")[:, None]
        cand.clamp_(max=n - 1)
        d = (xs[cand] - xs[a:b, None, :]).square_().sum(2)
        d[~ok] = math.inf
        d, pick = torch.topk(d, k, largest=False)
        dst = order[torch.gather(cand, 1, pick)]
        src = order[a:b, None].expand(-1, k)
        out.append(((src << 32) | dst)[d < math.inf])
    return torch.cat(out)


def _grid_keys(rows, cols, rng, both=0.3):
    v = torch.arange(rows * cols, device="cuda").view(rows, cols)
    a = torch.cat([v[:, :-1].reshape(-1), v[:-1].reshape(-1)])
    b = torch.cat([v[:, 1:].reshape(-1), v[1:].reshape(-1)])
    r = torch.rand(2, a.numel(), generator=rng, device="cuda")
    two, fwd = r[0] < both, r[1] < 0.5
    return torch.cat([((a << 32) | b)[two | fwd], ((b << 32) | a)[two | ~fwd]])


def _csr(keys, n):
    """(off int64[n+1], E int32[m]) of the sorted, distinct keys source << 32 | target."""
    ends = torch.arange(n + 1, device="cuda", dtype=torch.int64) << 32
    return torch.searchsorted(keys, ends), (keys & LOW).to(torch.int32)


def _both_csr(keys, n, transpose=True):
    keys = torch.unique_consecutive(torch.sort(keys)[0])
    off, E = _csr(keys, n)
    if not transpose:
        return n, off, E, None, None
    keys = torch.sort(((keys & LOW) << 32) | (keys >> 32))[0]
    return (n, off, E, *_csr(keys, n))


def _members(case):
    """(family, vertices) of a batch's graphs: half R-MAT, half kNN, sizes log-uniform from 2^8 up."""
    r = random.Random(case["count"] * 100 + case["log2_max"])
    return [("rmat", 1 << r.randint(8, case["log2_max"])) if k % 2 else
            ("knn", int(2 ** r.uniform(8, case["log2_max"]))) for k in range(case["count"])]


def _size(case):
    return case["rows"] * case["cols"] if case["graph"] == "grid" else case["n"]


def _graph(case, seed, transpose=True):
    """The directed graph of a case on the GPU: n, off, E, in_off, in_E."""
    n, rng = _size(case), _rng(seed)
    if case["graph"] == "rmat":
        keys = _rmat_keys(n, case["draws"], rng)
    elif case["graph"] == "knn":
        keys = _knn_keys(n, rng)
    else:
        keys = _grid_keys(case["rows"], case["cols"], rng)
    return _both_csr(keys, n, transpose)


def _upload(n, off, E, in_off=None, in_E=None, symmetrize=False):
    lib, h = psc.cuda(), ctypes.c_void_p()
    torch.cuda.synchronize()
    if symmetrize:
        status = lib.psc_graph_upload_symmetrize(off.data_ptr(), E.data_ptr(), n, E.numel(), ctypes.byref(h))
    else:
        status = lib.psc_graph_upload_device(off.data_ptr(), E.data_ptr(), in_off.data_ptr(), in_E.data_ptr(),
                                             n, E.numel(), ctypes.byref(h))
    if status:
        raise psc.PscError(status, "upload")
    return psc.DeviceGraph(handle=h.value)


def _pinned(count, dtype):
    return torch.empty(count, dtype=dtype, pin_memory=True)


# -- the calls --------------------------------------------------------------
def prepare(case, seed):
    op, dev = case["op"], "cuda"
    s = {"op": op}
    if op == "batch":
        sizes, rng = [n for _, n in _members(case)], _rng(seed)
        base = np.concatenate([[0], np.cumsum(sizes)])
        keys = [(_rmat_keys(n, 16 * n, rng) if kind == "rmat" else _knn_keys(n, rng)) + int(b) * ((1 << 32) + 1)
                for (kind, n), b in zip(_members(case), base)]
        s["dg"] = _upload(*_both_csr(torch.cat(keys), int(base[-1])))
        s["dg"].set_batch(base.astype(np.uint64))
        s["seeds"] = np.arange(case["count"], dtype=np.uint64) + np.uint64(seed)
        s["out"] = torch.empty(int(base[-1]), dtype=torch.int64, device=dev)
        s["params"] = psc.default_params()
        return s
    sym = op in ("cc", "lelist")
    n, off, E, in_off, in_E = _graph(case, seed, transpose=not (sym or op.startswith("load")))
    if op == "scc":
        s["dg"] = _upload(n, off, E, in_off, in_E)
        s["out"] = torch.empty(n, dtype=torch.int64, device=dev)
    elif op in ("load_scc", "load_cc"):
        for name, t, as_np in (("off", off, np.uint64), ("E", E, np.uint32)):
            h = _pinned(t.numel(), t.dtype)
            h.copy_(t)
            s[name] = h.numpy().view(as_np)
        s["out"] = _pinned(n, torch.int64 if op == "load_scc" else torch.int32)
    elif sym:
        s["dg"] = _upload(n, off, E, symmetrize=True)
        if op == "cc":
            s["out"] = _pinned(n, torch.int32)
        else:
            s["perm"] = psc.random_permutation(n, seed)
            # zeros, so that what lies behind the list is the same for everybody
            s["out"] = torch.zeros(3 * 16 * n, dtype=torch.int32, pin_memory=True)
    elif op == "bfs":
        s["dg"] = _upload(n, off, E, in_off, in_E)
        s["out"] = _pinned(n, torch.int32)
    elif op == "reach":
        s["arrays"] = (off, E, in_off, in_E)
        s["dir"] = case["dir"]
        s["out"] = torch.empty(n, dtype=torch.uint8, device=dev)
    if op in ("scc", "load_scc"):
        s["params"] = psc.default_params(seed=seed & 0x7FFFFFFF, beta=case.get("beta", 1.5))
    if op in ("bfs", "reach"):  # a source with edges: the tail or head of some edge
        e = int(torch.randint(E.numel(), (1,), generator=_rng(seed + 1), device=dev))
        if case.get("dir"):
            s["src"] = int(E[e])
        else:
            s["src"] = int(torch.searchsorted(off, torch.tensor([e], device=dev), right=True)) - 1
    s["n"] = n
    torch.cuda.synchronize()
    if _size(case) > 1 << 25:
        torch.cuda.empty_cache()
    return s


def _components(labels):
    """Each vertex's component as the component's smallest vertex: the roots are not fixed by the
    call, so a program that keeps or compares components renames them."""
    lab = labels.cuda(non_blocking=True)
    v = torch.arange(lab.numel(), device=lab.device, dtype=lab.dtype)
    # most vertices share one root: theirs is found by itself, the others scatter
    big = torch.mode(lab[:: max(1, lab.numel() // 4096)])[0]
    giant = lab == big
    least = v.clone().scatter_reduce_(0, torch.where(giant, v, lab).long(), v, "amin", include_self=False)
    least[big.long()] = giant.to(torch.uint8).argmax().to(lab.dtype)
    return least[lab.long()]


def run(s):
    op, out = s["op"], s["out"]
    lib = psc.cuda()
    if op == "scc":
        s["dg"].scc_device(out.data_ptr(), s["params"])
        return out
    if op == "batch":
        s["dg"].scc_batch_device(out.data_ptr(), s["params"], s["seeds"])
        return out
    if op == "load_scc":
        with psc.DeviceGraph.directed(s["off"], s["E"]) as dg:
            dg.scc(s["params"], out=out.numpy().view(np.uint64))
        return out
    if op == "load_cc":
        with psc.DeviceGraph.symmetrized(s["off"], s["E"]) as dg:
            dg.cc(out=out.numpy().view(np.uint32))
        return _components(out)
    if op == "cc":
        s["dg"].cc(out=out.numpy().view(np.uint32))
        return _components(out)
    if op == "lelist":
        s["dg"].lelist(s["perm"], out=out.numpy().view(np.uint32))
        return out
    if op == "bfs":
        status = lib.psc_bfs(s["dg"].h, s["src"], out.data_ptr(), None)
    else:
        off, E, in_off, in_E = s["arrays"]
        status = lib.psc_reach_noalloc(off.data_ptr(), E.data_ptr(), in_off.data_ptr(), in_E.data_ptr(),
                                       s["n"], E.numel(), s["src"], s["dir"], out.data_ptr(), None, None)
    if status:
        raise psc.PscError(status, op)
    return out


def work(case):
    op = case["op"]
    if op == "batch":
        members = _members(case)
        n = sum(size for _, size in members)
        m = sum(size * (16 if kind == "rmat" else 5) for kind, size in members)
    else:
        n = _size(case)
        m = {"rmat": case.get("draws", 0), "knn": 5 * n, "grid": 2.6 * n}[case["graph"]]
    one, ids = 8 * n + 4 * m, 4 * n  # one direction's offsets and targets; one number a vertex
    two = 8 * n + 8 * m  # a symmetrised graph
    b = {"scc": 2 * one + 2 * ids, "batch": 2 * one + 2 * ids, "load_scc": one + 2 * ids, "load_cc": one + ids,
         "cc": two + ids, "lelist": two + 4 * ids, "bfs": one + ids, "reach": one + n}[op]
    return {"bytes": b, "flops": 0}


def exact(case, seed):
    """Every output is whole numbers, which are compared as they are."""
    return None
