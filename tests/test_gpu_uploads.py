"""Small uploads through the ring in pinned memory: its wrap, and sizes on both sides of what goes through it."""
import numpy as np
import pytest
import torch

import vq_b200 as vq
from vq_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(16, 256), (7, 100), (64, 256), (65, 256)])  # 64, 11, 256 and 260 KiB of row numbers
def test_initial_rows_of_many_fits(m, k):
    x = synth.uniform01(3000, 4 * m, 5)
    xd = torch.from_numpy(x).cuda()
    rng = np.random.default_rng(m)
    fits = []
    for _ in range(40):
        idx = np.stack([rng.permutation(3000)[:k] for _ in range(m)]).astype(np.uint64)
        fits.append((idx, vq.ProductQuantizer.fit(xd, m, k, 0, vq.Distance.Euclidean, 1, init_idx=idx)))
    for idx, q in fits:
        want = np.stack([x[idx[s].astype(np.int64), 4 * s:4 * s + 4] for s in range(m)])
        assert np.array_equal(q.codebooks, want)
