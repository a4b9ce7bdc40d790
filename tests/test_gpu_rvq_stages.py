"""The residual encoder with all stages in one launch (rvq_tc.cu) against the CPU oracle, bit for bit."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS
from vq_b200 import synth

pytestmark = pytest.mark.gpu


# widths of one, two and four rows to an instruction, and those that fill no whole K step or 16-byte piece; 128 and 256 columns; the last row
# of a tile and the first of the next; half tiles up to 64 rows per SM (9,472 rows on 148 SMs), whole ones above; codebook images made in the same launch, and (19,073 rows) before
@pytest.mark.parametrize("n,dim,k,stages,eps,name", [
    (1_280, 17, 2, 3, 0.01, "Euclidean"), (2_049, 32, 256, 2, 0.01, "SquaredEuclidean"), (1_217, 33, 129, 3, 0.3, "Euclidean"),
    (1_409, 48, 128, 4, 0.01, "Euclidean"), (300, 61, 100, 8, 1.0, "Euclidean"), (9_472, 64, 60, 2, 0.01, "Euclidean"),
    (9_473, 80, 256, 2, 3.0, "SquaredEuclidean"), (1_089, 96, 200, 3, 0.01, "Euclidean"), (2_176, 112, 31, 1, 0.01, "Euclidean"),
    (19_073, 128, 256, 2, 0.01, "Euclidean"), (1_100, 128, 256, 5, 0.01, "SquaredEuclidean")])
@pytest.mark.parametrize("special", [False, True])
def test_codes_and_rows_equal_the_oracle(oracle, n, dim, k, stages, eps, name, special):
    x = synth.gaussian_mixture(n, dim, 9)
    books = (0.3 * synth.normal(stages * k, dim, 3)).reshape(stages, k, dim)
    books[0, :min(k, n)] = x[:min(k, n)]  # rows on centroids: residuals of zero
    if k > 20:
        books[-1, 9:20] = books[-1, 5]                      # equal centroids: the lowest number wins
        books[0, 7] = np.nextafter(books[0, 3], np.inf)     # and all but equal ones
    if special:
        x[n - 1, dim - 1], x[3, 0] = np.nan, np.inf
        x[4], x[5], x[6] = 0.0, 1e20, 1e-30
        x[7] *= 1e4
        x[8] *= 1e-6
        books[-1, k - 1, 0] = np.nan
        books[0, 1] = -0.0
    want, codes_o, _ = oracle.rvq_quantize(books, eps, x, METRICS[name])
    q = vq.ResidualQuantizer.from_codebooks(books, eps, getattr(vq.Distance, name))
    got, codes = q.quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(got, want.view(np.float16), equal_nan=True)


def test_norms_next_to_epsilon_are_added_up_in_order(oracle):
    """The early end of a row (src/rvq.rs:204-207) with norms within the rounding of a sum of epsilon, on both sides of it."""
    rng = np.random.default_rng(5)
    x = rng.normal(size=(2_000, 128)).astype(np.float32)
    books = rng.normal(size=(3, 40, 128)).astype(np.float32)
    books[0] = 0.0
    eps = 3.0
    norms = np.sqrt((x.astype(np.float64) ** 2).sum(axis=1))
    x = (x * (eps * (1 + 1e-7 * rng.integers(-6, 7, size=2_000)) / norms)[:, None]).astype(np.float32)
    want, codes_o, _ = oracle.rvq_quantize(books, eps, x, METRICS["Euclidean"])
    assert 100 < (codes_o[:, 1] == 0xFFFFFFFF).sum() < 1_900  # the case is on both sides
    got, codes = vq.ResidualQuantizer.from_codebooks(books, eps, vq.Distance.Euclidean).quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o) and np.array_equal(got.view(np.uint16), want)


@pytest.mark.parametrize("n", [2_000, 20_000])
def test_captured_encode_follows_its_rows(n):
    """One launch and two, replayed: the counters that the CTAs of the first wait on are left as they were found."""
    import torch

    x = torch.from_numpy(synth.gaussian_mixture(n, 128, 7)).cuda()
    books = (0.3 * synth.normal(3 * 256, 128, 3)).reshape(3, 256, 128)
    q = vq.ResidualQuantizer.from_codebooks(books, 0.01, vq.Distance.Euclidean)
    q.quantize(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, codes = q.quantize(x, return_codes=True)
    for seed in (7, 8):
        x.copy_(torch.from_numpy(synth.gaussian_mixture(n, 128, seed)))
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        got, got_codes = out.clone(), codes.clone()
        want, want_codes = q.quantize(x, return_codes=True)
        assert torch.equal(got_codes, want_codes) and torch.equal(got, want)
