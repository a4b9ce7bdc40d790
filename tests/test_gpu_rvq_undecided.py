"""Residual encode of rows that the tensor cores' scores leave undecided: the exact evaluation against the oracle, and what it costs."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS
from vq_b200 import synth

pytestmark = pytest.mark.gpu


def make(kind, n, dim, k, stages):
    x = synth.gaussian_mixture(n, dim, 5)
    books = 0.2 * synth.normal(stages * k, dim, 3).reshape(stages, k, dim)
    books[0] = x[np.arange(k) % n] + 0.01 * books[0]
    books = books.astype(np.float32)
    if kind == "pairs":  # every second centroid a rounding behind the first
        books[:, 1::2] = np.nextafter(books[:, 0:2 * (k // 2):2], np.float32(9))
    elif kind == "families":  # eight families of centroids next to each other
        for j in range(8, k):
            books[:, j] = books[:, j % 8] * np.float32(1 + 1.2e-7 * (j // 8))
    elif kind == "far":
        x = x + np.float32(1e4)
    elif kind == "few far":
        x[::67] += np.float32(1e5)
    elif kind == "overflow":
        x = x * np.float32(1e20)
    elif kind == "not finite":
        x[::5, dim // 2], x[1::5, 0], x[2::5, dim - 1] = np.nan, np.inf, -np.inf
        books[0, k - 1, 1], books[1, 0, 2] = np.inf, np.nan
    return x, books


@pytest.mark.parametrize("kind", ["pairs", "families", "far", "few far", "overflow", "not finite"])
@pytest.mark.parametrize("n,dim,k,stages", [(1_301, 128, 256, 3), (9_537, 128, 256, 2), (2_003, 96, 256, 3), (9_601, 96, 130, 2), (1_200, 80, 70, 3), (9_500, 80, 256, 2),
                                            (1_111, 61, 100, 2), (9_990, 33, 256, 2), (3_001, 24, 17, 3), (9_473, 112, 128, 2), (2_222, 64, 9, 2)])
@pytest.mark.parametrize("name", ["Euclidean", "SquaredEuclidean"])
def test_against_the_oracle(oracle, n, dim, k, stages, kind, name):
    x, books = make(kind, n, dim, k, stages)
    distance = getattr(vq.Distance, name)
    out_o, codes_o, _ = oracle.rvq_quantize(books, 0.01, x, METRICS[name])
    out, codes = vq.ResidualQuantizer.from_codebooks(books, 0.01, distance).quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(out, out_o.view(np.float16), equal_nan=True)


@pytest.mark.parametrize("kind,most", [("pairs", 4), ("far", 14), ("not finite", 4)])
@pytest.mark.parametrize("n", [1_500, 5_000])
def test_cost_against_rows_that_are_decided(n, kind, most):
    """Times an ordinary encode of the same shape.  A kernel that examines every centroid takes 3 (5,000 rows: 6) times as long as one on the tensor
    cores; where a warp examined its own rows far ones and those with values that are not finite took 50 and 60 times."""
    import torch

    def seconds(kind):
        x, books = make(kind, n, 128, 256, 8)
        x = torch.from_numpy(x).cuda()
        q = vq.ResidualQuantizer.from_codebooks(books, 1e-9, vq.Distance.Euclidean)
        for _ in range(3):
            q.quantize(x, return_codes=True)
        times = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            q.quantize(x, return_codes=True)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return sorted(times)[4]

    plain, this = seconds("plain"), seconds(kind)
    print(f"{kind}, {n} rows: {1e3 * this:.0f} us, plain {1e3 * plain:.0f}")
    assert this < most * plain
