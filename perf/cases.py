"""Performance cases: the calls that a program using wetric makes, with the
inputs and handles it has in hand beforehand.

Every case is a dict of plain values with a ``kind``, the public call it
times:

* ``count``      -- ``wetric.count`` on a device CSR with u32 offsets, or
                    ``OrientedGraph.count`` on the u64 offsets that
                    ``orient_edges`` leaves (``offsets``)
* ``orient``     -- ``wetric.orient_edges`` on raw device pairs
* ``symmetric``  -- ``wetric.count(..., oriented=False)`` on a symmetric
                    device CSR: orientation and count in one call
* ``tc_gpu``     -- ``wetric.tc_GPU`` on a host CSR in ordinary (pageable)
                    numpy arrays, the call a program of the reference makes
* ``create``     -- ``wetric.Batch`` from raw pairs and its first count: many
                    graphs seen once
* ``batch``      -- ``Batch.count`` of a resident batch, again and again
* ``serve``      -- requests submitted to a running ``wetric.Server`` and
                    waited for

and the graphs it is made on: R-MAT (a, b, c, d = 0.57, 0.19, 0.19, 0.05),
Erdos-Renyi and Chung-Lu graphs of the sizes and degrees that the package's
own workloads have (``wetric.workloads``), and for ``create``, ``batch`` and
``serve`` an uneven mixture of the last two.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "wedge-parallel-triangle-counting_b200"))

import wetric  # noqa: E402
from wetric.workloads import chung_lu_for  # noqa: E402

DEV = "cuda:0"


# ------------------------------------------------------------------- cases


def listed():
    return [
        # a small graph counted on its own, as in a loop over many small
        # inputs: launches and host work
        {"name": "count-er-2k", "kind": "count", "graph": "er", "n": 2000, "pairs": 16000,
         "offsets": 32, "s": 5, "a": 8192},
        # the package's plain single-graph workload, a co-purchase sized
        # power-law graph
        {"name": "count-chunglu-262k", "kind": "count", "graph": "chunglu", "n": 262111,
         "pairs": 899990, "gamma": 2.6, "offsets": 32, "s": 5, "a": 8192},
        # a graph without hubs: nearly all rows are short
        {"name": "count-er-700k", "kind": "count", "graph": "er", "n": 700001,
         "pairs": 13300019, "offsets": 32, "s": 2, "a": 4096},
        # the headline workload, on the CSR that orient_edges made
        {"name": "count-rmat-s22", "kind": "count", "graph": "rmat", "n": 1 << 22,
         "pairs": 16 << 22, "offsets": 64, "s": 5, "a": 8192},
        # a large graph
        {"name": "count-rmat-s24", "kind": "count", "graph": "rmat", "n": 1 << 24,
         "pairs": 16 << 24, "offsets": 64, "s": 10, "a": 16384},
        # preprocessing of a small edge list
        {"name": "orient-er-9k", "kind": "orient", "graph": "er", "n": 9001, "pairs": 70003},
        # preprocessing of the headline workload
        {"name": "orient-rmat-s22", "kind": "orient", "graph": "rmat", "n": 1 << 22,
         "pairs": 16 << 22},
        # a symmetric adjacency as other graph packages keep it
        {"name": "symmetric-chunglu-500k", "kind": "symmetric", "graph": "chunglu",
         "n": 500009, "pairs": 6000011, "gamma": 2.4, "offsets": 32, "s": 5, "a": 8192},
        # the reference's own call, host CSR in and count out
        {"name": "tc_gpu-rmat-s20", "kind": "tc_gpu", "graph": "rmat", "n": 1 << 20,
         "pairs": 16 << 20, "s": 5, "a": 8192},
        # a set of graphs that arrives, is counted once and goes
        {"name": "create-mixture-64", "kind": "create", "graphs": 64, "mix": 11, "n": 100000,
         "s": 5, "a": 8192},
        # a resident set of graphs
        {"name": "batch-mixture-96", "kind": "batch", "graphs": 96, "mix": 12, "n": 1000000,
         "s": 5, "a": 8192},
        # a burst of requests at a counting service
        {"name": "serve-mixture-48", "kind": "serve", "graphs": 48, "mix": 13, "n": 1000000,
         "s": 5, "a": 8192},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count", "count", "orient", "symmetric", "tc_gpu", "create", "batch",
                       "serve"])
    case = {"kind": kind}
    if kind in ("create", "batch", "serve"):
        case["graphs"] = _log_uniform(rng, 8, 96)
        case["mix"] = rng.randrange(1 << 20)
        case["n"] = _log_uniform(rng, 20000, 100000 if kind == "create" else 1000000)
        case["s"], case["a"] = 5, 8192
        return case
    case["graph"] = rng.choice(["rmat", "er", "chunglu"])
    if case["graph"] == "rmat":
        top = {"count": 23, "orient": 22, "symmetric": 20, "tc_gpu": 21}[kind]
        case["n"] = 1 << rng.randint(12, top)
        case["pairs"] = case["n"] * rng.randint(8, 16) + rng.randrange(1000)
    else:
        case["n"] = _log_uniform(rng, 1000, 1000000)
        case["pairs"] = int(case["n"] * rng.uniform(4, 64) / 2)
        if case["graph"] == "chunglu":
            case["gamma"] = round(rng.uniform(2.2, 3.0), 3)
    if kind != "orient":
        case["s"] = rng.choice([1, 2, 5, 10])
        case["a"] = rng.choice([0, 4096, 8192, 16384])
    if kind in ("count", "symmetric"):
        case["offsets"] = rng.choice([32, 64])
    return case


# ------------------------------------------------------------------ graphs


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _pairs(graph, n, pairs, gamma, gen):
    """Raw 0-based endpoint draws (loops and repeats included), int32."""
    src = torch.empty(pairs, dtype=torch.int32, device=DEV)
    dst = torch.empty(pairs, dtype=torch.int32, device=DEV)
    step = 1 << 25
    if graph == "chunglu":
        i0 = chung_lu_for(n, 2.0 * pairs / n, gamma, 0).i0
        w = (1.0 + torch.arange(n, dtype=torch.float64, device=DEV) / i0) ** (-1.0 / (gamma - 1.0))
        cdf = torch.cumsum(w, 0)
    for lo in range(0, pairs, step):
        k = min(step, pairs - lo)
        if graph == "rmat":
            s = torch.zeros(k, dtype=torch.int32, device=DEV)
            d = torch.zeros(k, dtype=torch.int32, device=DEV)
            for _ in range(n.bit_length() - 1):
                r = torch.rand(k, device=DEV, generator=gen)
                s = s * 2 + (r >= 0.76)
                d = d * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        elif graph == "chunglu":
            s, d = (torch.searchsorted(
                cdf, torch.rand(k, dtype=torch.float64, device=DEV, generator=gen) * cdf[-1])
                .clamp_(max=n - 1) for _ in range(2))
        else:
            s, d = (torch.randint(0, n, (k,), device=DEV, generator=gen) for _ in range(2))
        src[lo:lo + k] = s
        dst[lo:lo + k] = d
    return src, dst


def _edge_list(case, gen):
    """An edge list of the case's length with one row in twenty a repeat (in
    the other direction) or a loop: the first distinct edges that the draws
    give, so that lists of every seed make CSRs of one size."""
    n, pairs = case["n"], case["pairs"]
    extra = pairs // 20
    draws = pairs
    while True:
        src, dst = _pairs(case["graph"], n, draws, case.get("gamma", 0.0), gen)
        keep = src != dst
        src, dst = src[keep], dst[keep]
        key = torch.minimum(src, dst).long() * n + torch.maximum(src, dst)
        key, at = torch.sort(key, stable=True)
        first = torch.ones_like(key, dtype=torch.bool)
        first[1:] = key[1:] != key[:-1]
        at = torch.sort(at[first]).values[:pairs - extra]
        if at.numel() == pairs - extra:
            break
        draws += draws // 2
    src, dst = src[at], dst[at]
    loops = torch.arange(extra, dtype=torch.int32, device=DEV) % 2 * dst[:extra]
    return (torch.cat([src, dst[:extra]]),
            torch.cat([dst, torch.where(loops > 0, loops, src[:extra])]))


def _case_pairs(case, seed):
    gen = _generator(seed)
    if case["kind"] == "orient":
        return _edge_list(case, gen)
    return _pairs(case["graph"], case["n"], case["pairs"], case.get("gamma", 0.0), gen)


def _mixture(case):
    """(graph, n, pairs, gamma) of each graph of a mixture: half Erdos-Renyi,
    half Chung-Lu, n log-uniform up to the case's, mean degree 4 to 64."""
    rng = random.Random(case["mix"])
    out = []
    for i in range(case["graphs"]):
        n = _log_uniform(rng, 1000, case["n"])
        pairs = int(n * rng.uniform(4, 64) / 2)
        gamma = rng.uniform(2.2, 3.0)
        out.append(("er" if i % 2 == 0 else "chunglu", n, pairs, gamma))
    return out


class _View:
    """A device array of a handle as torch sees it; it keeps the handle."""

    def __init__(self, handle, ptr, count, typestr):
        self.handle = handle
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr,
                                         "data": (ptr, False), "version": 3}


def _arrays(og):
    """(row_ptr int64, col_ind int32) of an OrientedGraph, where it lies."""
    return (torch.as_tensor(_View(og, og.row_ptr_ptr, og.n + 1, "<i8"), device=DEV),
            torch.as_tensor(_View(og, og.col_ind_ptr, og.m, "<i4"), device=DEV))


def _symmetric_csr(src, dst, n):
    """Sorted symmetric adjacency without loops and repeats."""
    s, d = src.long(), dst.long()
    keep = s != d
    s, d = s[keep], d[keep]
    key = torch.unique(torch.cat([s * n + d, d * n + s]))
    deg = torch.bincount(torch.div(key, n, rounding_mode="floor"), minlength=n)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=src.device)
    rp[1:] = torch.cumsum(deg, 0)
    return rp, (key % n).int()


# ------------------------------------------------------- what a user has, does


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("create", "batch", "serve"):
        gen = _generator(seed)
        specs = _mixture(case)
        parts = [_pairs(*sp, gen) for sp in specs]
        n = np.array([sp[1] for sp in specs], np.uint64)
        if kind == "serve":
            state = {"server": wetric.Server(device=0, spread=case["s"], a=case["a"]),
                     "requests": [(s, d, sp[1]) for (s, d), sp in zip(parts, specs)]}
        else:
            off = np.zeros(len(specs) + 1, np.uint64)
            off[1:] = np.cumsum([sp[2] for sp in specs])
            state = {"src": torch.cat([p[0] for p in parts]),
                     "dst": torch.cat([p[1] for p in parts]), "off": off, "n": n,
                     "s": case["s"], "a": case["a"]}
            torch.cuda.synchronize()
            if kind == "batch":
                state = {"batch": wetric.Batch(state["src"], state["dst"], off, n,
                                               spread=case["s"], a=case["a"])}
    else:
        src, dst = _case_pairs(case, seed)
        torch.cuda.synchronize()
        if kind == "orient":
            state = {"src": src, "dst": dst, "n": case["n"]}
        elif kind == "symmetric":
            rp, ci = _symmetric_csr(src, dst, case["n"])
            state = {"rp": rp.int() if case["offsets"] == 32 else rp, "ci": ci}
        else:
            og = wetric.orient_edges(src, dst, case["n"])
            if kind == "tc_gpu":
                state = {"graph": og.download()}
            elif case["offsets"] == 32:
                rp, ci = _arrays(og)
                state = {"rp": rp.int(), "ci": ci.clone()}
            else:
                state = {"og": og}
        state["s"], state["a"] = case.get("s"), case.get("a")
    state["kind"] = kind
    torch.cuda.synchronize()
    return state


def _counted(count, st):
    return {"triangles": count, "wedges": st.wedges, "max_out_degree": st.max_out_degree}


def run(state):
    kind = state["kind"]
    if kind == "count":
        if "og" in state:
            return _counted(*state["og"].count(state["s"], state["a"]))
        return _counted(*wetric.count(state["rp"], state["ci"], state["s"], state["a"]))
    if kind == "symmetric":
        return _counted(*wetric.count(state["rp"], state["ci"], state["s"], state["a"],
                                      oriented=False))
    if kind == "orient":
        rp, ci = _arrays(wetric.orient_edges(state["src"], state["dst"], state["n"]))
        return {"row_ptr": rp, "col_ind": ci}
    if kind == "tc_gpu":
        return {"triangles": wetric.tc_GPU(state["graph"], state["s"], state["a"])}
    if kind == "create":
        b = wetric.Batch(state["src"], state["dst"], state["off"], state["n"],
                         spread=state["s"], a=state["a"])
        counts, _ = b.count()
        b.free()
        return {"triangles": counts}
    if kind == "batch":
        return {"triangles": state["batch"].count()[0]}
    server = state["server"]
    tickets = [server.submit(s, d, n) for s, d, n in state["requests"]]
    return {"triangles": np.array([server.wait(t)[0] for t in tickets], np.uint64)}


def work(case):
    """Bytes read and written once: pairs (8 each) or the CSR's columns (4,
    about one per pair) and offsets in, the CSR or the counts out."""
    kind = case["kind"]
    specs = _mixture(case) if "mix" in case else [(None, case["n"], case["pairs"], None)]
    n, pairs = sum(sp[1] for sp in specs), sum(sp[2] for sp in specs)
    if kind == "orient":
        return {"bytes": 8 * pairs + 8 * (n + 1) + 4 * pairs, "flops": 0}
    if kind in ("create", "serve"):
        return {"bytes": 8 * pairs + 8 * len(specs), "flops": 0}
    if kind == "symmetric":
        return {"bytes": 8 * pairs + case["offsets"] // 8 * (n + 1) + 8, "flops": 0}
    return {"bytes": 4 * pairs + case.get("offsets", 64) // 8 * (n + 1) + 8 * len(specs),
            "flops": 0}


# ------------------------------------------------------------------- oracle


def _oriented(src, dst, n):
    """The oriented CSR by its definition: vertices relabelled by ascending
    (degree, id), each edge kept once toward the higher label, rows sorted."""
    s, d = src.long(), dst.long()
    keep = s != d
    lo, hi = torch.minimum(s, d)[keep], torch.maximum(s, d)[keep]
    key = torch.unique(lo * n + hi)
    lo, hi = torch.div(key, n, rounding_mode="floor"), key % n
    deg = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
    rank = torch.empty(n, dtype=torch.int64, device=src.device)
    rank[torch.argsort(deg, stable=True)] = torch.arange(n, device=src.device)
    a, b = rank[lo], rank[hi]
    key = torch.sort(torch.minimum(a, b) * n + torch.maximum(a, b)).values
    rp = torch.zeros(n + 1, dtype=torch.int64, device=src.device)
    rp[1:] = torch.cumsum(torch.bincount(torch.div(key, n, rounding_mode="floor"), minlength=n), 0)
    return rp, (key % n).int(), key


def _triangles(rp, ci, key, n, most):
    """(triangles, wedges, max out-degree), wedge by wedge; no triangles
    where there are more than `most` wedges."""
    deg = rp[1:] - rp[:-1]
    wedges = int((deg * (deg - 1) // 2).sum())
    if wedges > most:
        return None, wedges, int(deg.max())
    row = torch.div(key, n, rounding_mode="floor")
    tail = rp[1:][row] - torch.arange(key.numel(), device=key.device) - 1  # later columns of the row
    total, start = 0, torch.cumsum(tail, 0)
    lo, step = 0, 1 << 26
    while lo < key.numel():
        base = int(start[lo - 1]) if lo else 0
        hi = max(lo + 1, int(torch.searchsorted(start, base + step, right=True)))
        t = tail[lo:hi]
        e = torch.repeat_interleave(torch.arange(lo, hi, device=key.device), t)
        j = torch.arange(e.numel(), device=key.device) - (start[e] - tail[e] - base)
        if e.numel():
            want = ci[e].long() * n + ci[e + 1 + j].long()
            at = torch.searchsorted(key, want).clamp_(max=key.numel() - 1)
            total += int((key[at] == want).sum())
        lo = hi
    return total, wedges, int(deg.max())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("create", "batch", "serve"):
        specs = _mixture(case)
        if sum(sp[2] for sp in specs) > 40_000_000:
            return None
        gen = _generator(seed)
        counts = []
        for sp in specs:
            src, dst = _pairs(*sp, gen)
            counts.append(_triangles(*_oriented(src, dst, sp[1]), sp[1], 1 << 31)[0])
        return None if None in counts else {"triangles": np.array(counts, np.uint64)}
    if case["pairs"] > 70_000_000:
        return None
    src, dst = _case_pairs(case, seed)
    rp, ci, key = _oriented(src, dst, case["n"])
    if kind == "orient":
        return {"row_ptr": rp, "col_ind": ci}
    tri, wedges, most = _triangles(rp, ci, key, case["n"], 1 << 32)
    if kind == "tc_gpu":
        return {"triangles": tri}
    return {"triangles": tri, "wedges": wedges, "max_out_degree": most}
