"""The workloads by which the speed of the device backend is measured.

Every case is one model of the suite driven the way a training script drives it: ``prepare`` builds
the model on one GPU, loads synthetic seeded data into it and initialises its parameters; ``run``
makes one pass through the model's public calls (an epoch, a round, a solve) and returns what the
script would keep.  ``listed`` names the cases, ``draw`` makes more of them over the same ranges,
``work`` states the bytes and floating-point operations a pass cannot do without and ``tolerance``
how far two correct fp32 implementations may differ.
"""
from __future__ import annotations

import math
from typing import Any, Dict

import numpy as np
import torch

from paracel_b200.models.als_gpu import AlsGpu
from paracel_b200.models.kmeans_gpu import KMeansGpu
from paracel_b200.models.lda_gpu import LdaGibbsGpu
from paracel_b200.models.linear_gpu import DenseLinearGpu, SparseLinearGpu, remap_by_frequency
from paracel_b200.models.mf_gpu import MfSgdGpu
from paracel_b200.models.pagerank_gpu import PageRankGpu
from paracel_b200.models.similarity_gpu import SimDenseGpu
from paracel_b200.models.svd_gpu import SvdGpu
from paracel_b200.utils import synth

DEV = "cuda"
MANY = 1 << 30          # rounds of a training run that is stopped from outside


def listed():
    return [
        # Matrix factorisation by SGD.  The small one is a film-rating sample on a workstation: a
        # round is a handful of short kernels, so launches and host calls count.
        {"name": "mf_small", "kind": "mf", "users": 6040, "items": 3706, "ratings": 1_000_209, "rank": 32},
        # The framework's headline configuration: 1 M users x 200 k items, 200 M Zipf(1.1) ratings.
        {"name": "mf_large", "kind": "mf", "users": 1_000_000, "items": 200_000, "ratings": 200_000_000,
         "rank": 128},
        # Logistic regression on a small dense table (the 20,000 x 100 plumbing configuration):
        # ten rounds, bound by latency.
        {"name": "dense_lr_small", "kind": "dense_lr", "rows": 20_000, "dim": 100, "rounds": 10, "logistic": True},
        # The same on a table far larger than the caches: bound by reading the rows.
        {"name": "dense_lr_large", "kind": "dense_lr", "rows": 2_000_000, "dim": 512, "rounds": 2, "logistic": True},
        # Click-through style L1 logistic regression on hashed features, 40 per row, Zipf(1.05), one
        # epoch of four minibatches with the proximal update.
        {"name": "sparse_l1_lr", "kind": "sparse_lr", "rows": 8_000_000, "features": 1 << 24, "per_row": 40,
         "batches": 4, "valued": False, "logistic": True},
        # PageRank, 20 iterations: a web-crawl sample that fits the caches ...
        {"name": "pagerank_small", "kind": "pagerank", "scale": 17, "edge_factor": 16, "iters": 20},
        # ... and a power-law graph of 16.8 M vertices and 268 M edges.
        {"name": "pagerank_large", "kind": "pagerank", "scale": 24, "edge_factor": 16, "iters": 20},
        # One half-iteration of alternating least squares: every user's normal equations at rank 128,
        # heavy-tailed numbers of ratings per user.
        {"name": "als", "kind": "als", "users": 100_000, "items": 50_000, "ratings": 10_000_000, "rank": 128},
        # k-means, three rounds on a million points.
        {"name": "kmeans", "kind": "kmeans", "points": 1_000_000, "dim": 128, "clusters": 1024, "rounds": 3},
        # Truncated SVD of a sparse rating matrix (20 factors, ten oversampled columns).
        {"name": "svd", "kind": "svd", "rows": 400_000, "cols": 100_000, "entries": 16_000_000, "factors": 20,
         "iters": 5},
        # Top-k neighbours of an odd number of rows among all of them.
        {"name": "similarity", "kind": "sim", "rows": 12_007, "dim": 100, "top": 20},
        # One sweep of the LDA sampler over a small corpus, four minibatches.
        {"name": "lda_sweep", "kind": "lda", "docs": 6_000, "vocab": 100_000, "mean_len": 200, "topics": 1024,
         "batches": 4},
    ]


def _log(rng, lo, hi):
    """An integer spread over [lo, hi] by its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mf", "dense_lr", "sparse_lr", "pagerank", "als", "kmeans", "svd", "sim", "lda"])
    if kind == "mf":
        nnz = _log(rng, 200_000, 100_000_000)
        return {"kind": kind, "users": max(1000, nnz // rng.randint(80, 250)),
                "items": max(500, nnz // rng.randint(250, 1000)), "ratings": nnz,
                "rank": rng.choice([16, 32, 50, 64, 100, 128])}
    if kind == "dense_lr":
        dim = _log(rng, 8, 1500)
        return {"kind": kind, "rows": max(1000, min(3_000_000, _log(rng, 1_000_000, 1_000_000_000) // dim)), "dim": dim,
                "rounds": rng.choice([2, 5, 10]), "logistic": rng.random() < 0.7}
    if kind == "sparse_lr":
        per_row = _log(rng, 8, 90)
        return {"kind": kind, "rows": max(2000, _log(rng, 400_000, 300_000_000) // per_row),
                "features": _log(rng, 1 << 14, 1 << 24), "per_row": per_row, "batches": rng.choice([1, 2, 4]),
                "valued": rng.random() < 0.5, "logistic": rng.random() < 0.7}
    if kind == "pagerank":
        return {"kind": kind, "scale": rng.randint(14, 23), "edge_factor": rng.randint(6, 24),
                "iters": rng.choice([10, 20])}
    if kind == "als":
        users = _log(rng, 1000, 90_000)
        return {"kind": kind, "users": users, "items": _log(rng, 1000, 50_000),
                "ratings": users * rng.randint(15, 110), "rank": rng.choice([10, 20, 32, 50, 64, 100, 128])}
    if kind == "kmeans":
        return {"kind": kind, "points": _log(rng, 10_000, 900_000), "dim": _log(rng, 8, 128),
                "clusters": _log(rng, 10, 1024), "rounds": rng.choice([1, 3])}
    if kind == "svd":
        rows = _log(rng, 20_000, 350_000)
        return {"kind": kind, "rows": rows, "cols": _log(rng, 5_000, 90_000), "entries": rows * rng.randint(15, 40),
                "factors": rng.choice([6, 10, 20, 40]), "iters": rng.choice([3, 5])}
    if kind == "sim":
        return {"kind": kind, "rows": _log(rng, 1000, 12_000), "dim": rng.randint(16, 256), "top": rng.choice([5, 10, 20])}
    topics = rng.choice([128, 256, 512, 1024])
    # the corpus is small beside the word-topic table (see tolerance)
    return {"kind": kind, "docs": _log(rng, 500, 6000), "vocab": rng.randint(80_000, 100_000) * 1024 // topics,
            "mean_len": rng.randint(50, 200), "topics": topics, "batches": rng.choice([2, 4])}


class Program:
    """What the training script holds: the case and its model.  The tables live in memory of their
    own, so they are given back when the script lets go of the model."""

    def __init__(self, case: Dict[str, Any], model):
        self.case, self.model = case, model

    def __del__(self):
        self.model.free()


def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _zipf(n, s, m, g):
    """m ids in [0, n), p(id) ~ (id + 1)^-s: inverse distribution function in closed form, so that a
    seed always gives the same ids."""
    x = torch.rand(m, device=DEV, generator=g, dtype=torch.float64)
    x = torch.pow(1.0 - x * (1.0 - float(n + 1) ** (1.0 - s)), 1.0 / (1.0 - s))
    return (x.to(torch.int64) - 1).clamp_(0, n - 1)


def _ratings(users, items, nnz, seed):
    """Ratings 1..5 of a rank-16 taste model plus noise, users and items drawn Zipf(1.1)."""
    g = _gen(seed)
    P = 0.5 * torch.randn(users, 16, device=DEV, generator=g)
    Q = 0.5 * torch.randn(items, 16, device=DEV, generator=g)
    u, i = _zipf(users, 1.1, nnz, g), _zipf(items, 1.1, nnz, g)
    # ids are those that occur in a rating file: every user and every item has a rating
    u[:users], i[users:users + items] = torch.arange(users, device=DEV), torch.arange(items, device=DEV)
    r = 0.5 * torch.randn(nnz, device=DEV, generator=g)
    for a in range(0, nnz, 1 << 24):
        b = min(nnz, a + (1 << 24))
        r[a:b] += (P[u[a:b]] * Q[i[a:b]]).sum(1)
    return u, i, torch.round(r.clamp_(1.0, 5.0))


def prepare(case, seed):
    c, seed = dict(case), int(seed)
    kind = c["kind"]
    if kind == "mf":
        u, i, r = _ratings(c["users"], c["items"], c["ratings"], seed)
        m = MfSgdGpu(c["users"], c["items"], k=c["rank"], alpha=0.0005, rounds=MANY, staleness=2, device=DEV,
                     seed=seed % 1000)
        m.load_ratings(u, i, r)
        m.init_parameters()
        return Program(c, m)
    if kind == "dense_lr":
        g = _gen(seed)
        n, d = c["rows"], c["dim"]
        X = torch.randn(n, d, device=DEV, generator=g)
        w = torch.randn(d, device=DEV, generator=g)
        z = X @ w
        if c["logistic"]:
            y = (torch.rand(n, device=DEV, generator=g) < torch.sigmoid(z)).float()
        else:
            y = z + 0.5 * torch.randn(n, device=DEV, generator=g)
        m = DenseLinearGpu(d, eta=0.1, beta=0.0 if c["logistic"] else 1e-4, logistic=c["logistic"], device=DEV)
        m.load(X, y)
        return Program(c, m)
    if kind == "sparse_lr":
        g = _gen(seed)
        cols = _zipf(c["features"], 1.05, c["rows"] * c["per_row"], g)
        # true weights: one feature in a hundred, N(0, 1)
        w = torch.randn(c["features"], device=DEV, generator=g)
        w *= torch.rand(c["features"], device=DEV, generator=g) < 0.01
        z = w[cols].view(c["rows"], c["per_row"]).sum(1)
        y = (torch.rand(c["rows"], device=DEV, generator=g) < torch.sigmoid(z)).float()
        # the loader renumbers features by frequency; rows are ragged: a quarter lose some entries
        keep = torch.ones(c["rows"], c["per_row"], dtype=torch.bool, device=DEV)
        short = torch.rand(c["rows"], device=DEV, generator=g) < 0.25
        cut = torch.randint(1, c["per_row"] + 1, (c["rows"],), device=DEV, generator=g)
        keep &= ~(short[:, None] & (torch.arange(c["per_row"], device=DEV)[None, :] >= cut[:, None]))
        lens = keep.sum(1)
        row_ptr = torch.zeros(c["rows"] + 1, dtype=torch.int64, device=DEV)
        row_ptr[1:] = torch.cumsum(lens, 0)
        cols = cols[keep.view(-1)]
        cols, _ = remap_by_frequency(cols, c["features"])
        vals = None
        if c["valued"]:
            vals = 0.5 + torch.rand(cols.numel(), device=DEV, generator=g)
        m = SparseLinearGpu(c["features"], eta=0.5 if c["logistic"] else 0.02, lam=1e-6, logistic=c["logistic"],
                            nbatch=c["batches"], device=DEV)
        m.load(row_ptr, cols, y, vals)
        return Program(c, m)
    if kind == "pagerank":
        n, left, chunk = 1 << c["scale"], c["edge_factor"] << c["scale"], 1 << 26
        src, dst, j = [], [], 0
        while left > 0:
            s, t = synth.rmat_edges_chunk(c["scale"], min(chunk, left), 0.57, 0.19, 0.19, seed * 131 + j, DEV)
            src.append(synth.scramble_vertex_blocks(s, c["scale"]))
            dst.append(synth.scramble_vertex_blocks(t, c["scale"]))
            left -= chunk
            j += 1
        m = PageRankGpu(n, 0.85, device=DEV)
        m.load_edges(torch.cat(src), torch.cat(dst))
        return Program(c, m)
    if kind == "als":
        u, i, r = _ratings(c["users"], c["items"], c["ratings"], seed)
        m = AlsGpu(c["users"], c["items"], c["rank"], lam=0.1, device=DEV)
        H = torch.randn(c["items"], c["rank"], device=DEV, generator=_gen(seed)) / math.sqrt(c["rank"])
        m.load(u, i, r, torch.arange(c["items"], device=DEV), H)
        return Program(c, m)
    if kind == "kmeans":
        g = _gen(seed)
        n, d, k = c["points"], c["dim"], c["clusters"]
        centres = torch.randn(k, d, device=DEV, generator=g)
        X = centres[torch.randint(0, k, (n,), device=DEV, generator=g)]
        X = X + 0.5 * torch.randn(n, d, device=DEV, generator=g)
        m = KMeansGpu(k, d, device=DEV)
        m.load(X)
        return Program(c, m)
    if kind == "svd":
        u, i, r = _ratings(c["rows"], c["cols"], c["entries"], seed)
        key = torch.unique(u * c["cols"] + i, return_inverse=True)
        # one value per cell: the best of a user's ratings of an item
        vals = torch.zeros(key[0].numel(), device=DEV).scatter_reduce_(0, key[1], r, "amax")
        row = key[0] // c["cols"]
        ptr = torch.zeros(c["rows"] + 1, dtype=torch.int64, device=DEV)
        ptr[1:] = torch.cumsum(torch.bincount(row, minlength=c["rows"]), 0)
        m = SvdGpu(c["cols"], c["factors"], iters=c["iters"], seed=3, device=DEV)
        m.load(ptr, (key[0] % c["cols"]).to(torch.int32), vals)
        return Program(c, m)
    if kind == "sim":
        X = torch.randn(c["rows"], c["dim"], device=DEV, generator=_gen(seed))
        m = SimDenseGpu(c["dim"], ktop=c["top"], simbar=-1.0, device=DEV)
        m.load(torch.arange(c["rows"], device=DEV), X)
        return Program(c, m)
    g = _gen(seed)
    lens = torch.poisson(torch.full((c["docs"],), float(c["mean_len"]), device=DEV), generator=g).long().clamp(min=1)
    ptr = torch.zeros(c["docs"] + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(lens, 0)
    words = _zipf(c["vocab"], 1.07, int(ptr[-1]), g)
    m = LdaGibbsGpu(c["vocab"], c["topics"], beta=0.01, iters=1 << 20, nbatch=c["batches"], device=DEV, seed=seed % 1000)
    m.load_docs(ptr, words)
    return Program(c, m)


def run(state):
    c, m = state.case, state.model
    kind = c["kind"]
    if kind == "mf":
        m.round()
        return {"W": m.Wl, "H": m.Hl, "bu": m.bul, "bi": m.bil}
    if kind == "dense_lr":
        for _ in range(c["rounds"]):
            m.step()
        return {"weights": m.weights(), "loss": m.grad.loss}
    if kind == "sparse_lr":
        m.epoch()
        return {"weights": m.weights(), "loss": m.loss}
    if kind == "pagerank":
        m.run(c["iters"])
        return m.ranks()
    if kind == "als":
        m.solve()
        return m.W
    if kind == "kmeans":
        m.fit(c["rounds"])
        return {"centres": m.cluster_centres(), "assign": m.assign}
    if kind == "svd":
        m.solve()
        return {"U": m.U, "sigma": m.sigma, "V": m.V}
    if kind == "sim":
        m.solve()
        got = np.array(list(m.result.values()))        # rows x top x (neighbour, similarity)
        return {"neighbour": got[:, :, 0].astype(np.int64), "similarity": got[:, :, 1]}
    loglik = m.iteration(with_loglik=True)
    return {"loglik": loglik, "word_topic": m.topic_word_counts().clone()}


def work(case):
    c = case
    kind = c["kind"]
    if kind == "mf":
        # a rating needs its two ids and its value; every row of W and H is read and written once
        rows = (c["users"] + c["items"]) * (c["rank"] + 1) * 4.0
        return {"bytes": 2 * rows + 12.0 * c["ratings"], "flops": 10.0 * c["ratings"] * c["rank"]}
    if kind == "dense_lr":
        x = 4.0 * c["rows"] * c["dim"]
        return {"bytes": c["rounds"] * (x + 4.0 * c["rows"]), "flops": c["rounds"] * x}
    if kind == "sparse_lr":
        nnz = 0.875 * c["rows"] * c["per_row"]
        one = nnz * (8.0 if c["valued"] else 4.0) + 12.0 * c["rows"]
        return {"bytes": one + c["batches"] * 8.0 * c["features"], "flops": 4.0 * nnz}
    if kind == "pagerank":
        n, e = float(1 << c["scale"]), float(c["edge_factor"] << c["scale"])
        return {"bytes": c["iters"] * (4 * e + 20 * n), "flops": c["iters"] * (e + 3 * n)}
    if kind == "als":
        k, n = c["rank"], c["users"]
        return {"bytes": 8.0 * c["ratings"] + 4.0 * k * (c["items"] + n),
                "flops": c["ratings"] * (k * k + 2.0 * k) + n * (k ** 3 / 3.0 + 2.0 * k * k)}
    if kind == "kmeans":
        x = float(c["points"]) * c["dim"]
        return {"bytes": c["rounds"] * (8 * x + 8.0 * c["points"]), "flops": c["rounds"] * (2 * x * c["clusters"] + x)}
    if kind == "svd":
        K = min((c["factors"] + 10 + 3) // 4 * 4, 112)
        it, e, mn = c["iters"], float(c["entries"]), float(c["rows"] + c["cols"])
        return {"bytes": (2 * it + 1) * (8 * e + 4 * K * mn) + 4 * K * mn,
                "flops": (2 * it + 1) * 2 * e * K + (2 * it + 2) * 4 * mn * K * K}
    if kind == "sim":
        n, d = float(c["rows"]), c["dim"]
        return {"bytes": 4 * n * d + 12 * n * c["top"], "flops": 2 * n * n * d}
    tok = float(c["docs"]) * c["mean_len"]
    # a token needs its word, its topic and the counts of both; the table is read and written once
    return {"bytes": 12 * tok + 8.0 * c["topics"] * (c["docs"] + c["vocab"]), "flops": 8.0 * tok * c["topics"]}


def tolerance(case):
    """About four times the largest difference seen between a pass and the same pass in 64 bits, or
    between two passes on the same inputs where the order of the updates is not fixed."""
    kind = case["kind"]
    if kind == "mf":
        # thousands of ratings are in flight and meet rows of different age in every run; the biases
        # of the hottest rows show it most (rel 0.011, max 0.5)
        return {"rel": 3e-2, "max": 0.99}
    if kind == "dense_lr":
        return {"rel": 1e-6, "max": 4e-6}
    if kind == "sparse_lr":
        return {"rel": 1e-4, "max": 4e-4}
    if kind == "pagerank":
        return {"rel": 4e-7, "max": 1e-6}
    if kind == "als":
        return {"rel": 4e-5, "max": 2e-3}
    if kind == "kmeans":
        # a point between two centres may go to either and moves both
        return {"rel": 2e-3, "max": 0.1, "differ": 1.5e-4}
    if kind == "svd":
        # columns of U and V with neighbouring singular values turn into one another
        return {"rel": 4e-4, "max": 0.15}
    if kind == "sim":
        return {"rel": 8e-6, "max": 1.5e-5, "differ": 3e-4}
    # Two runs of the sampler order their count updates differently and so draw other topics; the
    # likelihood is stable, and 0.55 % of the table's cells are touched by one run only.
    return {"rel": 4e-4, "max": 4e-4, "differ": 1e-2}
