"""Unordered sums of wide rows in no whole 16-byte pieces, of which only the moved rows are added up: whole numbers, exact in any order."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS, RecordingSeeder
from vq_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k", [(80_000, 33, 5), (79_999, 61, 20), (80_031, 61, 20), (81_000, 127, 3)])
def test_codebooks_of_whole_numbers_equal_the_oracle(oracle, n, dim, k):
    x = np.round(4 * synth.gaussian_mixture(n, dim, 3, components=9)).astype(np.float32)
    so, sg = RecordingSeeder(5), RecordingSeeder(5)
    want, _res, _norms = oracle.rvq_fit(x, 1, k, 4, 1e-6, METRICS["SquaredEuclidean"], so.init_stage, so.draw)
    got = vq.ResidualQuantizer.fit(x, 1, k, 4, 1e-6, vq.Distance.SquaredEuclidean, 5, init=sg.init_stage, draw=sg.draw, accumulate=vq.ACCUM_FAST).codebooks
    assert np.array_equal(got, want)
