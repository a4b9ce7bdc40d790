"""Encodes of few rows whose shared memory is just below 48 KiB without the kernel's own arrays and above it with them."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS
from vq_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sd", [111, 112, 113, 127, 128])
def test_wide_subspaces_of_few_centroids(oracle, sd):
    x = synth.uniform(4000, sd, 3, -1.0, 1.0)
    books = synth.uniform(64, sd, 5, -1.0, 1.0).reshape(1, 64, sd)
    for n in (9, 2000, 4000):  # (one, some and eight rows a thread group)
        want, codes_o = oracle.pq_quantize(books, x[:n], METRICS["Euclidean"])
        got, codes = vq.ProductQuantizer.from_codebooks(books, vq.Distance.Euclidean).quantize(x[:n], return_codes=True)
        assert np.array_equal(codes, codes_o) and np.array_equal(got.view(np.uint16), want)
