"""The calls whose speed matters to a user of this package, from one vector to ten million.

Every case names one public entry point (``op``) and its sizes; ``draw`` gives further cases of the same ranges:

* rows: 1 .. 1,000,000 for ``quantize`` (10,000,000 for the element-wise quantizers), 2,000 .. 1,000,000 for training;
* product quantizers: 4 .. 32 sub-spaces, 4, 8 or 16 values wide; full-width quantizers: 24 .. 128 values per row;
* 16 .. 256 centroids, any number between, most often 256; 10 iterations;
* Euclidean distance for the most part; cosine and Manhattan distance where ``quantize`` looks at it;
* rows on the GPU, and for small batches in host memory too (a service that encodes what it has just received).

The values follow the benchmark's configurations: uniform rows for the product and element-wise quantizers, a mixture of 64
Gaussians for the residual and tree quantizers, correlated normal rows for the rotated product quantizer.
"""
import math

import numpy as np
import torch

import vq_b200 as vq

DISTANCES = {
    "euclidean": vq.Distance.Euclidean,
    "squared": vq.Distance.SquaredEuclidean,
    "cosine": vq.Distance.CosineDistance,
    "manhattan": vq.Distance.Manhattan,
}
ORDERED_ROWS = 65536  # up to here training adds up rows in their order: the codebooks are the same bits every time


def listed():
    pq = {"dim": 128, "m": 16, "k": 256, "distance": "euclidean"}
    return [
        # one vector at a time, as the reference's own API is called in a loop: latency and launches only
        {"name": "bq_row", "op": "bq", "n": 1, "dim": 128},
        {"name": "pq_encode_row", "op": "pq_encode", "n": 1, "where": "gpu", **pq},
        # a request of a service: rows in host memory, codes and reconstruction back to it
        {"name": "pq_encode_host", "op": "pq_encode", "n": 1000, "where": "host", **pq},
        # encoding a whole collection; element-wise at the size where only memory bandwidth counts
        {"name": "pq_encode_1m", "op": "pq_encode", "n": 1_000_000, "where": "gpu", **pq},
        {"name": "sq_10m", "op": "sq", "n": 10_000_000, "dim": 128, "levels": 256},
        # another metric, and sizes that are no powers of two
        {"name": "pq_encode_cosine", "op": "pq_encode", "n": 60_001, "where": "gpu", "dim": 96, "m": 12, "k": 200, "distance": "cosine"},
        # residual encode of a batch: eight dependent stages
        {"name": "rvq_encode_batch", "op": "rvq_encode", "n": 4_999, "where": "gpu", "dim": 128, "stages": 8, "k": 256, "distance": "euclidean"},
        # training: on a sample, on the whole collection, and the other quantizers at the benchmark's size
        {"name": "pq_fit_10k", "op": "pq_fit", "n": 10_000, "iters": 10, **pq},
        {"name": "pq_fit_1m", "op": "pq_fit", "n": 1_000_000, "iters": 10, **pq},
        {"name": "rvq_fit_1m", "op": "rvq_fit", "n": 1_000_000, "dim": 128, "stages": 4, "k": 256, "iters": 10, "distance": "euclidean"},
        {"name": "opq_fit_1m", "op": "opq_fit", "n": 1_000_000, "iters": 5, "outer": 10, **pq},
        {"name": "tsvq_fit_100k", "op": "tsvq_fit", "n": 100_000, "dim": 128, "depth": 10, "distance": "euclidean"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["sq", "bq", "pq_encode", "pq_encode", "rvq_encode", "opq_encode", "tsvq_encode", "pq_fit", "rvq_fit", "opq_fit", "tsvq_fit"])
    if op in ("sq", "bq"):
        dim = rng.choice([128, rng.randint(16, 256)])
        c = {"op": op, "n": _log(rng, 1, 1_280_000_000 // max(dim, 128)), "dim": dim}
        if op == "sq":
            c["levels"] = rng.choice([256, rng.randint(2, 256)])
        return c
    fit = op.endswith("_fit")
    c = {"op": op, "n": _log(rng, 2_000, 1_000_000) if fit else _log(rng, 1, 1_000_000), "k": rng.choice([256, _log(rng, 16, 256)])}
    c["distance"] = rng.choice(["euclidean", "euclidean", "euclidean", "squared"] + ([] if fit else ["cosine", "manhattan"]))
    if op.startswith(("pq", "opq")):
        # rotations of wider rows depend on the last bits of the sums when they are trained on few rows
        c["m"] = rng.choice([16, rng.randint(4, 16 if op == "opq_fit" else 32)])
        c["dim"] = c["m"] * rng.choice([8, 8, 8, 4] + ([] if op == "opq_fit" else [16]))
    else:
        c["dim"] = rng.choice([32, 64, 96, 128, rng.randint(24, 128), rng.randint(24, 128)])
    if op.startswith("rvq"):
        c["stages"] = rng.randint(2, 8)
    if op.startswith("tsvq"):
        del c["k"]
        c["depth"] = rng.randint(4, 10)
        return c
    if fit:
        c["iters"] = 5 if op == "opq_fit" else 10
        if op == "opq_fit":
            c["outer"] = 2
        elif op == "rvq_fit" and c["n"] > ORDERED_ROWS:
            c["stages"] = 2  # see tolerance()
        # no more distance computations than the product quantizer's training on a million rows
        per_row = c["k"] * c["dim"] * c["iters"] * c.get("stages", 1) * c.get("outer", 1)
        c["n"] = max(2_000, min(c["n"], 256 * 128 * 10 * 1_000_000 // per_row))
    elif c["n"] <= 4096 and op == "pq_encode":
        c["where"] = rng.choice(["gpu", "host"])
    return c


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rows(case, g, n):
    """n rows with the distribution that this quantizer is benchmarked on."""
    dim, op = case["dim"], case["op"]
    if op in ("sq", "bq"):
        return torch.rand(n, dim, generator=g, device="cuda").mul_(2.0).sub_(1.0)
    if op.startswith("pq"):
        return torch.rand(n, dim, generator=g, device="cuda")
    if op.startswith("opq"):
        a = torch.randn(dim, dim, generator=g, device="cuda") / math.sqrt(dim)
        return torch.randn(n, dim, generator=g, device="cuda") @ a
    means = torch.rand(64, dim, generator=g, device="cuda")
    which = torch.randint(64, (n,), generator=g, device="cuda")
    return torch.randn(n, dim, generator=g, device="cuda").mul_(0.05).add_(means[which])


def _nearest(sample, centroids):
    return torch.cdist(sample, centroids).argmin(dim=1)


def _trained(sample, k, g):
    """k centroids as training leaves them: rows of the sample, moved to their clusters' means twice."""
    c = sample[torch.randperm(sample.shape[0], generator=g, device="cuda")[:k]].clone()
    for _ in range(2):
        member = torch.nn.functional.one_hot(_nearest(sample, c), k).to(sample.dtype)
        count = member.sum(dim=0).unsqueeze(1)
        c = torch.where(count > 0, (member.T @ sample) / count.clamp(min=1), c)
    return c


def prepare(case, seed):
    op, g, n = case["op"], _generator(seed), case["n"]
    if op == "tsvq_encode":
        rows = _rows(case, g, n + 8192)
    elif op.endswith("_encode"):
        rows = _rows(case, g, n + 4096)
    else:
        rows = _rows(case, g, n)
    state = {"op": op, "x": rows[:n]}
    if op == "sq":
        state["quantizer"] = vq.ScalarQuantizer.fit(0.0, 1.0, case["levels"])
        return state
    if op == "bq":
        state["quantizer"] = vq.BinaryQuantizer.fit(0.0, 0, 1)
        return state
    distance = DISTANCES[case["distance"]]
    if op.endswith("_fit"):
        state.update(case=dict(case), distance=distance, seed=int(seed))
        return state
    # quantize: the quantizer a program keeps, with codebooks of a sample of the same distribution
    state["x"], sample = rows[:n].clone(), rows[n:]
    if n == 1:
        state["x"] = state["x"][0]
    if case.get("where") == "host":
        state["x"] = state["x"].cpu().numpy()
    if op == "tsvq_encode":
        state["quantizer"] = vq.TSVQ(sample, case["depth"], distance)
        return state
    k = case["k"]
    if op == "rvq_encode":
        books = []
        for _ in range(case["stages"]):
            books.append(_trained(sample, k, g))
            sample = sample - books[-1][_nearest(sample, books[-1])]
        state["quantizer"] = vq.ResidualQuantizer.from_codebooks(torch.stack(books).cpu().numpy(), 0.01, distance)
        return state
    m, dim = case["m"], case["dim"]
    if op == "opq_encode":
        rotation = torch.linalg.qr(torch.randn(dim, dim, generator=g, device="cuda"))[0].contiguous()
        sample = sample @ rotation.T
    books = torch.stack([_trained(s.contiguous(), k, g) for s in sample.view(-1, m, dim // m).unbind(dim=1)]).cpu().numpy()
    if op == "opq_encode":
        state["quantizer"] = vq.OptimizedProductQuantizer.from_parts(rotation.cpu().numpy(), books, distance)
    else:
        state["quantizer"] = vq.ProductQuantizer.from_codebooks(books, distance)
    return state


def run(state):
    op, x = state["op"], state["x"]
    if op in ("sq", "bq"):
        return state["quantizer"].quantize(x)
    if op == "tsvq_encode":
        return state["quantizer"].quantize(x, return_leaf=True)
    if op.endswith("_encode"):
        return state["quantizer"].quantize(x, return_codes=True)
    c, distance, seed = state["case"], state["distance"], state["seed"]
    if op == "pq_fit":
        return vq.ProductQuantizer.fit(x, c["m"], c["k"], c["iters"], distance, seed).codebooks
    if op == "rvq_fit":
        return vq.ResidualQuantizer.fit(x, c["stages"], c["k"], c["iters"], 0.01, distance, seed).codebooks
    if op == "opq_fit":
        q = vq.OptimizedProductQuantizer.fit(x, c["m"], c["k"], c["iters"], c["outer"], distance, seed)
        return q.rotation, q.codebooks
    centroids, left, right = vq.TSVQ(x, c["depth"], distance).tree()
    return centroids, left, right


def work(case):
    op, n, dim = case["op"], case["n"], case["dim"]
    if op in ("sq", "bq"):
        return {"bytes": 5 * n * dim, "flops": 3 * n * dim}
    if op == "tsvq_fit":  # every level: a mean and a spread of every row, and one comparison
        nodes = 2 ** (case["depth"] + 1)
        return {"bytes": 4 * n * dim + 4 * min(nodes, 2 * n) * dim, "flops": 4 * n * dim * case["depth"]}
    if op == "tsvq_encode":
        return {"bytes": 6 * n * dim + 4 * n + 4 * 2 ** (case["depth"] + 1) * dim, "flops": 6 * n * dim * case["depth"]}
    scores = 2 * n * case["k"] * dim
    if op == "rvq_encode":
        s = case["stages"]
        return {"bytes": 6 * n * dim + 4 * n * s + 4 * s * case["k"] * dim, "flops": scores * s}
    books = 4 * case["k"] * dim
    if op in ("pq_encode", "opq_encode"):
        turn = dim * dim if op == "opq_encode" else 0
        return {"bytes": 6 * n * dim + 4 * n * case["m"] + books + 4 * turn, "flops": scores + 2 * n * turn}
    if op == "pq_fit":
        return {"bytes": 4 * n * dim + books, "flops": scores * case["iters"]}
    if op == "rvq_fit":
        return {"bytes": 4 * n * dim + case["stages"] * books, "flops": scores * case["iters"] * case["stages"]}
    return {"bytes": 4 * n * dim + books + 4 * dim * dim, "flops": (scores * (case["iters"] + 1) + 4 * n * dim * dim) * case["outer"]}


def tolerance(case):
    op = case["op"]
    if op == "opq_encode":
        # the rotated rows are 32-bit sums in any order: a row between two centroids may take either one's values and code
        return {"rel": 1e-3, "max": 1 - 1e-9, "differ": 1e-4}
    # Training on more than ORDERED_ROWS rows adds them up in any order: centroids start 1e-7 apart, a row between two of them
    # then goes to either, and every iteration multiplies that (two runs of one program differ by a third of these figures).
    if op == "pq_fit" and case["n"] > ORDERED_ROWS:
        return {"rel": 3e-3, "max": 0.1}
    # Later residual stages train on what the earlier ones left, and the rotation is the polar factor of an ill-conditioned matrix.
    if op == "opq_fit" or (op == "rvq_fit" and case["n"] > ORDERED_ROWS):
        return {"rel": 0.03, "max": 0.9}
    return "exact"
