"""Ordered cluster sums of wide rows (ordered_sums_long_kernel): lists of every length around its stages, bit for bit."""
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
