"""Ordered cluster sums: lists of every length around the stages of ordered_sums_long_kernel, and lists made in one launch, bit for bit."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS, RecordingSeeder
from vq_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [17, 32, 61, 64, 100, 128])
def test_lists_around_whole_stages(oracle, dim):
    sizes = [1, 19, 20, 127, 128, 129, 139, 140, 141, 255, 256, 257, 383, 384, 385, 511, 512, 513, 640, 1025]
    rng = np.random.default_rng(dim)
    member = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    centers = 50.0 * synth.normal(len(sizes), dim, 3).reshape(len(sizes), dim)
    x = (centers[member] + 0.1 * rng.normal(size=(len(member), dim))).astype(np.float32)
    first = np.array([np.flatnonzero(member == j)[0] for j in range(len(sizes))], np.uint64)
    init = lambda stage, n, k: first  # noqa: E731
    want, _res, _norms = oracle.rvq_fit(x, 1, len(sizes), 3, 1e-6, METRICS["Euclidean"], init, RecordingSeeder(1).draw)
    got = vq.ResidualQuantizer.fit(x, 1, len(sizes), 3, 1e-6, vq.Distance.Euclidean, 1, init=init, accumulate=vq.ACCUM_ORDERED).codebooks
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n,m,k", [(5, 2, 2), (33, 1, 3), (4096, 3, 5), (4097, 3, 5), (4129, 2, 300), (65_536, 2, 5), (65_537, 2, 5), (5000, 1, 1024), (5000, 1, 1025)])
def test_lists_of_one_launch_and_of_two(oracle, n, m, k):
    """Rows of a warp in whole and in broken groups of 32, the last rows and clusters of the one-launch kernel and the first beyond."""
    x = synth.uniform(n, 4 * m, n, -1.0, 1.0)
    so, sg = RecordingSeeder(3), RecordingSeeder(3)
    init = so.init_pq(n, m, k)
    sg.init_pq(n, m, k)
    want, _iters = oracle.pq_fit(x, m, k, 2, init, so.draw)
    got = vq.ProductQuantizer.fit(x, m, k, 2, vq.Distance.Euclidean, 3, init_idx=init, draw=sg.draw, accumulate=vq.ACCUM_ORDERED).codebooks
    assert np.array_equal(got, want)
