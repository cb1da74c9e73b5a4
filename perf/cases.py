"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values; ``listed()`` gives the fixed ones, ``draw(rng)``
one more of the same ranges, ``prepare`` what a program has in hand before the
call, ``run`` one pass through the public entry points, ``work`` the bytes and
operations a pass cannot do without and ``exact`` the same outputs in 64 bits.

Kinds:

* ``fit``   -- a progressive build through ``GPUMAP``: a model over host rows,
  ``run_with_n_ops(chunk, upd, emb)`` until every row is in, then the views.
* ``embed`` -- ``run_with_n_ops(0, 0, emb)`` on a model that a program keeps: the
  layout step of an interactive session.
* ``fuzzy`` -- the operator ``gm_op_fuzzy_schedule`` on a published k-NN table.

Learning rate: the layout's SGD is Hogwild parallel, and at the default rate
(1.0) two runs on the same inputs give layouts as different as two seeds do.
Cases that return a layout use a small ``alpha`` instead, as for fine tuning: the
edges, samples and epochs are the same, and the layouts can be compared.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

DEV = "cuda"
ALPHA = 1e-4


def listed():
    return [
        # a first look at a small table, default engine (FP32 NN-Descent), all
        # three phases, short schedule: launches and latency count
        {"name": "fit_small_600x24", "kind": "fit", "data": "mixture", "n": 600, "d": 24, "k": 15, "metric": "euclidean",
         "precision": 0, "overlap": 0, "chunk": 200, "upd": 400, "emb": 200, "epochs": 20},
        # the whole of a 10,000 x 64 table in one call, all phases, 200 epochs
        {"name": "fit_one_call_10kx64", "kind": "fit", "data": "mixture", "n": 10_000, "d": 64, "k": 15, "metric": "euclidean",
         "precision": 0, "overlap": 0, "chunk": 10_000, "upd": 20_000, "emb": 50_000, "epochs": 200},
        # the default engine on image rows, 500 a cycle with 2,000 update ops
        {"name": "nnd_image_20kx784", "kind": "fit", "data": "image", "n": 20_000, "d": 784, "k": 15, "metric": "euclidean",
         "precision": 0, "overlap": 0, "chunk": 500, "upd": 2000, "emb": 0, "epochs": 200},
        # the default engine on cosine embeddings, the wide list, large cycles
        {"name": "nnd_cosine_100kx128_k30", "kind": "fit", "data": "cosine", "n": 100_000, "d": 128, "k": 30, "metric": "cosine",
         "precision": 0, "overlap": 0, "chunk": 10_000, "upd": 10_000, "emb": 0, "epochs": 200},
        # exact engine, odd sizes: ragged cycles, feature count past two chunks
        {"name": "exact_odd_4999x131_k10", "kind": "fit", "data": "mixture", "n": 4999, "d": 131, "k": 10, "metric": "cosine",
         "precision": 1, "overlap": 0, "chunk": 333, "upd": 0, "emb": 0, "epochs": 200},
        # exact engine on the full image table, 500 rows a cycle, graph only
        {"name": "exact_image_70kx784", "kind": "fit", "data": "image", "n": 70_000, "d": 784, "k": 15, "metric": "euclidean",
         "precision": 1, "overlap": 0, "chunk": 500, "upd": 0, "emb": 0, "epochs": 200},
        # the same with every cycle's layout step beside the next cycle's
        # distance work (overlap)
        {"name": "full_image_70kx784", "kind": "fit", "data": "image", "n": 70_000, "d": 784, "k": 15, "metric": "euclidean",
         "precision": 1, "overlap": 1, "chunk": 500, "upd": 0, "emb": 1000, "epochs": 200},
        # exact engine on cosine embeddings, the wide list, large cycles
        {"name": "exact_cosine_160kx128_k30", "kind": "fit", "data": "cosine", "n": 160_000, "d": 128, "k": 30, "metric": "cosine",
         "precision": 1, "overlap": 0, "chunk": 10_000, "upd": 0, "emb": 0, "epochs": 200},
        # the layout step of an interactive session: 1,000 rows, 200 epochs
        {"name": "embed_1k_of_20k", "kind": "embed", "data": "mixture", "n": 20_000, "d": 64, "k": 15, "metric": "euclidean", "emb": 1000,
         "epochs": 200},
        # the layout step over every row: throughput counts
        {"name": "embed_all_20k", "kind": "embed", "data": "mixture", "n": 20_000, "d": 64, "k": 15, "metric": "euclidean", "emb": 20_000,
         "epochs": 200},
        # the fuzzy set and edge schedule alone: a cycle's batch of a large
        # table, and every row of one with the wide list
        {"name": "fuzzy_1k_of_70k", "kind": "fuzzy", "data": "mixture", "n": 70_000, "d": 64, "k": 15, "metric": "euclidean", "nb": 1000,
         "epochs": 200},
        {"name": "fuzzy_all_100k_k30", "kind": "fuzzy", "data": "cosine", "n": 100_000, "d": 64, "k": 30, "metric": "cosine",
         "nb": 100_000, "epochs": 200},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.choice([5, 10, 15, 15, 30, 32])
    data, metric = rng.choice([("mixture", "euclidean"), ("image", "euclidean"), ("cosine", "cosine"), ("mixture", "cosine")])
    pick = rng.random()
    if pick < 0.6:
        d = _log(rng, 10, 784)
        n = _log(rng, 500, 60_000 if d <= 200 else 20_000)
        precision = rng.choice([0, 1])
        chunk = min(n, _log(rng, max(n // 30, 100), n))
        upd = 0 if precision else rng.choice([0, chunk, 4 * chunk])
        emb = rng.choice([0, 0, min(n, 2 * chunk)])
        return {"kind": "fit", "data": data, "n": n, "d": d, "k": k, "metric": metric, "precision": precision,
                "overlap": rng.choice([0, 1]) if emb else 0, "chunk": chunk, "upd": upd, "emb": emb,
                "epochs": rng.choice([20, 50, 200])}
    n = _log(rng, 1000, 60_000)
    if pick < 0.8:
        return {"kind": "embed", "data": data, "n": n, "d": 64, "k": k, "metric": metric, "emb": min(n, _log(rng, 200, 20_000)),
                "epochs": rng.choice([50, 200])}
    return {"kind": "fuzzy", "data": data, "n": n, "d": 64, "k": k, "metric": metric, "nb": _log(rng, 200, n), "epochs": 200}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rows(case, seed):
    """Rows of the case's distribution, on the GPU (the shapes of gpumap_gb300.datasets)."""
    n, d, kind = case["n"], case["d"], case["data"]
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)

    def normal(*shape):
        return torch.randn(*shape, device=DEV, generator=g)

    def uniform(*shape):
        return torch.rand(*shape, device=DEV, generator=g)

    if kind == "image":  # sparse nonnegative centres plus noise, clipped to [0, 1]
        c = torch.where(uniform(10, d) < 0.2, uniform(10, d), torch.zeros((), device=DEV))
        z = torch.randint(0, 10, (n,), device=DEV, generator=g)
        return (c[z] + 0.1 * normal(n, d)).clamp_(0.0, 1.0)
    if kind == "cosine":  # centres on the sphere, weights ~ j^-1.1, small angles
        c = torch.nn.functional.normalize(normal(100, d), dim=1)
        w = torch.arange(1, 101, device=DEV, dtype=torch.float32) ** -1.1
        z = torch.multinomial(w, n, replacement=True, generator=g)
        return torch.nn.functional.normalize(c[z] + 0.15 / math.sqrt(d) * normal(n, d), dim=1)
    c = 4.0 * normal(10, d)  # isotropic mixture
    z = torch.randint(0, 10, (n,), device=DEV, generator=g)
    return c[z] + normal(n, d)


def _model(case, x, precision, overlap=0):
    import gpumap_gb300 as gm
    from gpumap_gb300.data_loader import ArrayDataLoader

    p = gm.GPUMAPParams()
    p.n_instances, p.n_features = case["n"], case["d"]
    p.n_neighbors, p.metric = case["k"], case["metric"]
    p.max_epoch, p.alpha = case["epochs"], ALPHA
    p.precision, p.overlap = precision, overlap
    return gm.GPUMAP(ArrayDataLoader(x), p)


def prepare(case, seed):
    x = _rows(case, seed).cpu().numpy()
    if case["kind"] == "fit":
        return {"case": case, "x": x}
    # a model whose rows are all in, with exact neighbours
    m = _model(case, x, 1)
    m.run_with_n_ops(case["n"], 0, 0)
    if case["kind"] == "embed":
        return {"case": case, "model": m}
    # its published table, and the newest rows as the batch
    n, k, nb = case["n"], case["k"], case["nb"]
    wide = {}
    for name, view in (("idx", m._impl.get_neighbor_indices()), ("dist", m._impl.get_neighbor_dists())):
        t = torch.from_dlpack(view)
        wide[name] = (t.view(torch.int32) if name == "idx" else t).clone()
    torch.cuda.synchronize()
    m.close()
    return {"case": case, "idx": wide["idx"], "dist": wide["dist"],
            "batch": torch.arange(n - nb, n, device=DEV, dtype=torch.int32)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "fit":
        m = _model(case, state["x"], case["precision"], case["overlap"])
        for _ in range(0, case["n"], case["chunk"]):
            m.run_with_n_ops(case["chunk"], case["upd"], case["emb"])
        out = {"indices": m.get_neighbor_indices().view(torch.int32), "dists": m.get_neighbor_dists()}
        if case["emb"]:
            out["embedding"] = m.get_embedding()
        return out
    if case["kind"] == "embed":
        m = state["model"]
        m.run_with_n_ops(0, 0, case["emb"])
        return {"embedding": m.get_embedding()}
    return _fuzzy(state)


def _fuzzy(state):
    from gpumap_gb300 import _native

    case = state["case"]
    n, k, nb = case["n"], case["k"], case["nb"]
    cap = 2 * nb * k
    ints = torch.zeros(4, cap, device=DEV, dtype=torch.int32)
    vals = torch.zeros(2, cap, device=DEV)
    rows = torch.empty(2, n, device=DEV)
    counts, scalars = (C.c_int64 * 4)(), (C.c_float * 3)()
    _native.check(_native.load().gm_op_fuzzy_schedule(
        state["idx"].data_ptr(), state["dist"].data_ptr(), n, k, int(case["metric"] == "euclidean"),
        state["batch"].data_ptr(), nb, case["epochs"], 1.0, ints[0].data_ptr(), ints[1].data_ptr(), vals[0].data_ptr(),
        ints[2].data_ptr(), ints[3].data_ptr(), vals[1].data_ptr(), rows[0].data_ptr(), rows[1].data_ptr(), counts, scalars,
        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    # the set and the schedule, each with zeros past its last edge
    ints[2:, int(counts[2]):] = 0
    vals[1, int(counts[2]):] = 0
    return {"coo_row": ints[0], "coo_col": ints[1], "coo_val": vals[0],
            "edge_head": ints[2], "edge_tail": ints[3], "edge_period": vals[1],
            "sigma": rows[0], "rho": rows[1], "counts": [int(c) for c in counts], "scalars": [float(s) for s in scalars]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n, d, k = case["n"], case["d"], case["k"]
    table = n * k * 8.0
    if case["kind"] == "fit":
        cycles = -(-n // case["chunk"])
        nbytes = n * d * 4.0 + table + (n * 8.0 if case["emb"] else 0.0)
        if case["precision"]:
            flops = float(n) * n * d  # every pair once
        else:
            # ten rounds of up to 256 two-hop candidates a row; joins of about
            # 2k new with 6k others
            flops = 10.0 * n * min(k * k, 256, n) * 2 * d
            flops += float(cycles) * min(case["upd"], 2 * n) * min(2 * k, 64) * min(6 * k, 128) * 2 * d
        flops += cycles * _sgd_flops(case, min(case["emb"], n))
        return {"bytes": nbytes, "flops": flops}
    if case["kind"] == "embed":
        return {"bytes": table + n * 16.0, "flops": _sgd_flops(case, case["emb"])}
    # edges: about 1.6 nb k, 12 bytes each in the set and in the schedule
    return {"bytes": table + 1.6 * case["nb"] * k * 24.0 + n * 8.0, "flops": n * k * 20.0 * 10.0}


def _sgd_flops(case, rows):
    # about 1.6 k edges a row, a third of them active in an epoch, an
    # attraction and five repulsions of about 30 operations each
    return rows * 1.6 * case["k"] * case["epochs"] / 3.0 * 6 * 30.0


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "fit":
        # every pair's distance: lists of the exact engine
        if not case["precision"] or float(case["n"]) ** 2 * case["d"] > 5e12 or case["n"] <= case["k"]:
            return None
        out = {"indices": None, "dists": _exact_dists(case, seed)}
        if case["emb"]:
            out["embedding"] = None
        return out
    return _exact_fuzzy(case, seed) if case["kind"] == "fuzzy" else None


def _exact_dists(case, seed):
    x = _rows(case, seed).double()
    n, k = case["n"], case["k"]
    if case["metric"] == "cosine":
        x = torch.nn.functional.normalize(x, dim=1)
    sq = (x * x).sum(1)
    out = torch.empty(n, k, device=DEV, dtype=torch.float64)
    step = max(1, (1 << 28) // n)
    for s in range(0, n, step):
        e = min(n, s + step)
        dist = torch.addmm(sq[s:e, None] + sq[None, :], x[s:e], x.T, alpha=-2.0)
        dist[torch.arange(e - s, device=DEV), torch.arange(s, e, device=DEV)] = math.inf
        out[s:e] = torch.topk(dist, k, dim=1, largest=False, sorted=True).values.clamp_(min=0.0)
    return out


def _exact_fuzzy(case, seed):
    state = prepare(case, seed)
    n, k, epochs = case["n"], case["k"], case["epochs"]
    me = torch.arange(n, device=DEV)
    # the row itself at distance 0, then its first k - 1 neighbours
    col = torch.cat([me[:, None], state["idx"][:, : k - 1].long()], 1)
    raw = torch.cat([torch.zeros(n, 1, device=DEV, dtype=torch.float64), state["dist"][:, : k - 1].double()], 1)
    raw = raw.clamp(min=0.0).sqrt() if case["metric"] == "euclidean" else raw
    mean = raw.mean()
    nz = raw > 0
    has = nz.any(1)
    rho = torch.where(has, raw.gather(1, nz.to(torch.int8).argmax(1, keepdim=True))[:, 0], torch.zeros((), device=DEV, dtype=torch.float64))
    off = raw - rho[:, None]
    target = math.log2(k - 1)
    lo, hi, mid = torch.zeros_like(rho), torch.full_like(rho, math.inf), torch.ones_like(rho)
    done = torch.zeros_like(has)
    for _ in range(64):
        term = torch.where(off > 0, torch.exp(-off / mid[:, None]), torch.ones_like(off))[:, 2:].sum(1)
        done = done | ((term - target).abs() < 1e-5)
        big = term > target
        nhi, nlo = torch.where(big, mid, hi), torch.where(big, lo, mid)
        nmid = torch.where(big | nhi.isfinite(), (nlo + nhi) / 2, mid * 2)
        hi, lo, mid = torch.where(done, hi, nhi), torch.where(done, lo, nlo), torch.where(done, mid, nmid)
    floor = 1e-3 * torch.where(rho > 0, raw.mean(1), mean)
    sigma = torch.where(has, torch.maximum(mid, floor), 1e-3 * mean)

    def member(dist, r, s):
        return torch.where((dist - r <= 0) | (s == 0), torch.ones_like(dist), torch.exp(-(dist - r) / s).clamp(min=2.0 ** -126))

    b = state["batch"].long()
    cb = col[b]
    pij = member(raw[b], rho[b, None], sigma[b, None])
    pij = torch.where(cb == b[:, None], torch.zeros_like(pij), pij)
    pji = torch.zeros_like(pij)
    for c in range(k - 1, -1, -1):  # the first listing of the batch row counts
        hit = col[:, c][cb] == b[:, None]
        pji = torch.where(hit, member(raw[:, c][cb], rho[cb], sigma[cb]), pji)
    w = pij + pji - pij * pji
    extra = w[pji == 0]
    val = torch.cat([w.reshape(-1), extra])
    top = val.max()
    left = val[val >= top / epochs]
    pad = torch.zeros(2, 2 * case["nb"] * k, device=DEV, dtype=torch.float64)
    pad[0, : val.numel()], pad[1, : left.numel()] = val, top / left
    return {"coo_row": None, "coo_col": None, "coo_val": pad[0], "edge_head": None, "edge_tail": None, "edge_period": pad[1],
            "sigma": sigma, "rho": rho, "counts": [None] * 4, "scalars": [float(mean), float(top), None]}
