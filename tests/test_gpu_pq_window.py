"""Many rows are scored as exactly as few: the window of the product quantizer's fixed-point scores does not widen with the number of rows."""
import numpy as np
import pytest

from vq_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("n", [1_000, 6_001, 20_000])
def test_scores_of_clustered_rows_against_f64(ctx, n, metric):
    """Clusters, whose rows lie within a few units of T of several centroids.  T = sigma S + K0 cut to a whole number, one addend with a fraction
    beside 2^23 and the result's unit: (-1.25, 0.25), and 0.17 for the parts that are dropped or rounded before (header of pq_tc.cu)."""
    rng = np.random.default_rng(n + metric)
    m, k, sd = 4, 256, 8
    where = rng.normal(size=(64, m, sd))
    cb = (where[rng.integers(64, size=k)] + 0.05 * rng.normal(size=(k, m, sd))).astype(np.float32).transpose(1, 0, 2).copy()
    x = (where[rng.integers(64, size=n)] + 0.05 * rng.normal(size=(n, m, sd))).astype(np.float32).reshape(n, m * sd)
    t, frames, consts = np.zeros((n, m, 256), np.float32), np.zeros((n, m, 2), np.float32), np.zeros((m, 32), np.float32)
    rc = _lib.load().vqb_pq_tensor_fixed_point(ctx.handle, x.ctypes.data, n, m, sd, cb.ctypes.data, k, metric, t.ctypes.data, frames.ctypes.data,
                                               consts.ctypes.data)
    assert rc == 0, _lib.load().vqb_last_error(ctx.handle).decode()
    sigma, k0 = frames[:, :, :1].astype(np.float64), frames[:, :, 1:].astype(np.float64)
    mu = -consts[:, :sd].astype(np.float64)
    far = np.unpackbits(consts[:, 24:].copy().view(np.uint8), axis=1, bitorder="little")[:, :k].astype(bool)
    y, c = x.astype(np.float64).reshape(n, m, sd) - mu, cb.astype(np.float64) - mu[:, None]
    half = 0.5 * (c * c).sum(-1)
    if metric == 2:
        half, c = np.zeros((m, k)), c / np.linalg.norm(c, axis=-1, keepdims=True)
    exact = sigma * (half[None] - np.einsum("nmd,mkd->nmk", y, c)) + k0
    error = np.where((sigma > 0) & ~far[None], t - exact, 0.0)
    print(f"T - sigma S - K0: {error.min():.3f} .. {error.max():.3f}")
    assert -1.25 - 0.17 < error.min() and error.max() < 0.25 + 0.17
