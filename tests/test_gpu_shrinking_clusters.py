"""Unordered sums: the mean of a cluster that used to be large is as exact as that of any other of its size."""
import numpy as np
import pytest

import vq_b200 as vq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [33, 61, 127])
def test_mean_of_a_cluster_that_has_shrunk(dim):
    """Blobs along the first dimension.  The first centroid starts in the small one at 0 and gets the large ones at -10 and 10 too; the others start
    at -30 and 30, move to -16 and 16 and take the large ones over.  110,120 rows are more than are added up in order; 100 remain, whose sum of f32
    is at most 100 2^-24 of the sum of their magnitudes away from the exact one, in any order; the division rounds once more."""
    rng = np.random.default_rng(dim)
    blobs = [(0, 100), (-10, 50_000), (10, 50_000), (-16, 5_000), (16, 5_000), (-30, 10), (30, 10)]
    at = np.concatenate([np.full(rows, where, np.float64) for where, rows in blobs])
    x = 0.3 * rng.normal(size=(len(at), dim)) + 100.0
    x[:, 0] += at - 100.0
    x = x.astype(np.float32)
    first = [0, len(at) - 15, len(at) - 5]
    order = rng.permutation(len(at))
    place = np.empty(len(at), np.int64)
    place[order] = np.arange(len(at))
    got = vq.ResidualQuantizer.fit(x[order], 1, 3, 6, 1e-6, vq.Distance.SquaredEuclidean, 5, init=lambda stage, n, k: place[first],
                                   accumulate=vq.ACCUM_FAST).codebooks[0]
    rows = x[:100].astype(np.float64)
    want = rows.mean(axis=0)
    bound = 2.0 ** -24 * (np.abs(rows).sum(axis=0) + np.abs(want))
    print(f"largest error {np.abs(got[0] - want).max():.2e}, bound {bound.max():.2e}")
    assert (np.abs(got[0] - want) <= bound).all()
