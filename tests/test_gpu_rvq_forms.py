"""Residual encodes in forms that the tensor-core kernel takes beside the usual ones."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS
from vq_b200 import synth

pytestmark = pytest.mark.gpu


def check(oracle, x, books, eps, quantized, codes):
    out_o, codes_o, _ = oracle.rvq_quantize(books, eps, x, METRICS["Euclidean"])
    assert np.array_equal(codes, codes_o.view(codes.dtype))
    assert np.array_equal(quantized, out_o.view(np.float16), equal_nan=True)


@pytest.mark.parametrize("n,dim,k,stages", [(2_100, 128, 256, 2), (13_000, 96, 100, 3), (1_500, 32, 256, 4)])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_rows_off_16_bytes_beside_codebooks_that_are_not(oracle, n, dim, k, stages, shift):
    import torch

    x = synth.gaussian_mixture(n, dim, 5).astype(np.float32)
    books = (0.2 * synth.normal(stages * k, dim, 3)).astype(np.float32).reshape(stages, k, dim)
    room = torch.empty(n * dim + shift, device="cuda")
    rows = room[shift:].view(n, dim)
    rows.copy_(torch.from_numpy(x))
    assert rows.data_ptr() % 16 == 4 * shift
    out, codes = vq.ResidualQuantizer.from_codebooks(books, 0.01, vq.Distance.Euclidean).quantize(rows, return_codes=True)
    check(oracle, x, books, 0.01, out.cpu().numpy(), codes.cpu().numpy())


@pytest.mark.parametrize("stages", [254, 255, 256, 300])
@pytest.mark.parametrize("n,dim,k", [(1_400, 24, 4), (9_600, 64, 17)])
def test_many_stages(oracle, n, dim, k, stages):
    x = synth.gaussian_mixture(n, dim, 5).astype(np.float32)
    books = (synth.normal(stages * k, dim, 3).reshape(stages, k, dim) * (0.5 ** (np.arange(stages) / 30.0))[:, None, None]).astype(np.float32)
    out, codes = vq.ResidualQuantizer.from_codebooks(books, 1e-6, vq.Distance.Euclidean).quantize(x, return_codes=True)
    check(oracle, x, books, 1e-6, out, codes)
