"""The product quantizer's chain of two steps (training passes, encodes of many rows): its fixed-point scores against f64, and its codes where they
are close."""
import ctypes as C

import numpy as np
import pytest

import vq_b200 as vq
from tests.golden import reference_known_answers as ka
from vq_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["euclid", "cosine"])
@pytest.mark.parametrize("case", ["uniform", "normal", "offset", "far", "tight", "signs"])
@pytest.mark.parametrize("m,k", [(5, 256), (4, 100)])
def test_scores_against_f64(ctx, m, k, case, metric):
    """T = sigma S + K0 cut to a whole number: eleven addends with fractions beside 2^23 and the result's unit, (-3.75, 2.25), and 0.17 for the
    parts that are dropped or rounded before (FEW in the header of pq_tc.cu)."""
    rng = np.random.default_rng(m * k + len(case))
    n, sd = 6_001, 8
    x = rng.normal(size=(n, m * sd)).astype(np.float32)
    cb = rng.normal(size=(m, k, sd)).astype(np.float32)
    if case == "uniform":
        x, cb = rng.random(x.shape, dtype=np.float32), rng.random(cb.shape, dtype=np.float32)
    elif case == "offset":
        x, cb = x + np.float32(100), cb + np.float32(100)
    elif case == "far":
        cb[:, 7] *= 100
        x[::3] *= 50
    elif case == "tight":
        where = rng.normal(size=(8, m, sd)).astype(np.float32) * 10
        cb = (where[rng.integers(8, size=k)] + rng.normal(size=(k, m, sd)) * 1e-2).astype(np.float32).transpose(1, 0, 2).copy()
        x = (where[rng.integers(8, size=n)] + rng.normal(size=(n, m, sd)) * 1e-2).astype(np.float32).reshape(n, m * sd)
    elif case == "signs":  # the products of the last step with one sign each
        x, cb = np.abs(x), np.abs(cb) * np.where(np.arange(k) % 2, 1, -1).astype(np.float32)[None, :, None]
    t, frames, consts = np.zeros((n, m, 256), np.float32), np.zeros((n, m, 2), np.float32), np.zeros((m, 32), np.float32)
    rc = _lib.load().vqb_pq_tensor_fixed_point(ctx.handle, x.ctypes.data, n, m, sd, cb.ctypes.data, k, 2 if metric == "cosine" else 0, t.ctypes.data,
                                               frames.ctypes.data, consts.ctypes.data)
    assert rc == 0, _lib.load().vqb_last_error(ctx.handle).decode()
    sigma, k0 = frames[:, :, :1].astype(np.float64), frames[:, :, 1:].astype(np.float64)
    far = np.unpackbits(consts[:, 24:].copy().view(np.uint8), axis=1, bitorder="little")[:, :k].astype(bool)
    mu = -consts[:, :sd].astype(np.float64)
    y, c = x.astype(np.float64).reshape(n, m, sd) - mu, cb.astype(np.float64) - mu[:, None]
    if metric == "cosine":
        half, c = np.zeros((m, k)), c / np.linalg.norm(c, axis=-1, keepdims=True)
    else:
        half = 0.5 * (c * c).sum(-1)
    exact = sigma * (half[None] - np.einsum("nmd,mkd->nmk", y, c)) + k0
    use = (sigma > 0) & ~far[None]
    error = np.where(use, t[:, :, :k] - exact, 0.0)
    print(f"T - sigma S - K0: {error.min():.3f} .. {error.max():.3f}; T {t[:, :, :k][use].min()} .. {t[:, :, :k][use].max()}")
    assert (t == np.floor(t)).all() and t[:, :, :k][use].min() >= 1
    assert -3.75 - 0.17 < error.min() and error.max() < 2.25 + 0.17
    assert (np.abs(t[:, :, k:] - 57344)[np.broadcast_to(sigma > 0, (n, m, 256 - k))] <= 1).all()


@pytest.mark.parametrize("n", [5_999, 6_000])
@pytest.mark.parametrize("gap", [1e-5, 3e-5, 1e-4, 3e-4])
def test_pairs_of_close_centroids(oracle, n, gap):
    """Second centroids 1 to 20 units of T behind the first, on both sides of the line between the chains."""
    rng = np.random.default_rng(int(gap * 1e6))
    m, k = 4, 256
    cb = rng.random((m, k, 8), dtype=np.float32)
    cb[:, 1::2] = cb[:, ::2] + (gap * rng.normal(size=(m, k // 2, 8))).astype(np.float32)
    x = rng.random((n, m * 8), dtype=np.float32)
    for distance, metric in ((vq.Distance.Euclidean, ka.EUCLID), (vq.Distance.SquaredEuclidean, ka.SQ), (vq.Distance.CosineDistance, ka.COSINE)):
        _, codes = vq.ProductQuantizer.from_codebooks(cb, distance).quantize(x, return_codes=True)
        assert np.array_equal(codes, oracle.pq_quantize(cb, x, metric)[1])
