"""Kernels at the sizes where a split, tile or list can go wrong, against the CPU oracle."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import RecordingSeeder, by_stream
from vq_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,sd,k", [(1023, 2, 3, 2), (1025, 3, 5, 7), (4097, 1, 12, 300), (5000, 1, 40, 33), (70_001, 2, 8, 5), (9000, 1, 2, 4096),
                                      (9000, 1, 2, 4097)])
def test_ordered_sums_bit_exact(oracle, n, m, sd, k):
    """Chunk edges of the row lists, every lane split of the sums (4, 8, 16, 32 lanes and wider rows), codes of one and two
    bytes, a cluster of thousands of rows beside clusters of one, and one cluster more than the lists take."""
    x = synth.uniform01(n, m * sd, 5 + n)
    x[n // 3: n // 3 + n // 2] = x[0]  # half of the rows in one cluster
    so, sg = RecordingSeeder(3), RecordingSeeder(3)
    init = so.init_pq(n, m, k)
    sg.init_pq(n, m, k)
    cb_o, it_o = oracle.pq_fit(x, m, k, 3, init, so.draw)
    pq = vq.ProductQuantizer.fit(x, m, k, 3, vq.Distance.Euclidean, 3, init_idx=init, draw=sg.draw, accumulate=vq.ACCUM_ORDERED)
    assert np.array_equal(pq.iterations, it_o) and by_stream(so.draws) == by_stream(sg.draws)
    assert np.array_equal(pq.codebooks, cb_o)
