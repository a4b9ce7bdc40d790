"""The product quantizer's tensor-core kernel where its fixed-point scores could go wrong: edges of the column tiles, centroids and rows
far from the rest, offsets, sub-spaces and rows that only the full scan can decide, queues that fill up.  Codes and codebooks are
the oracle's bit for bit."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.golden import reference_known_answers as ka
from tests.util import RecordingSeeder

pytestmark = pytest.mark.gpu


def _check(oracle, cb, x, metric=(vq.Distance.Euclidean, ka.EUCLID)):
    q = vq.ProductQuantizer.from_codebooks(cb, metric[0])
    out, codes = q.quantize(x, return_codes=True)
    out_o, codes_o = oracle.pq_quantize(cb, x, metric[1])
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(out, out_o.view(np.float16), equal_nan=True)


@pytest.mark.parametrize("k", [2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 192, 255, 256])
@pytest.mark.parametrize("m,sd", [(4, 8), (20, 8), (7, 8), (9, 4)])
def test_edges_of_the_column_tiles(oracle, k, m, sd):
    rng = np.random.default_rng(k * 100 + m)
    n = 90_000 // m + 1  # past the one-launch path, a ragged last tile
    x = rng.random((n, m * sd), dtype=np.float32)
    cb = rng.random((m, k, sd), dtype=np.float32)
    cb[1, k - 1] = cb[1, 0]                 # a tie between the first and the last column
    x[n - 3:, sd:2 * sd] = cb[1, 0]
    _check(oracle, cb, x)


@pytest.mark.parametrize("m,sd", [(4, 4), (5, 8), (6, 4), (13, 8), (31, 4), (63, 8), (64, 4)])
def test_groups_that_are_not_full(oracle, m, sd):
    """Numbers of sub-spaces that leave the last group of a launch with one to three, both widths, against the oracle: encode with each
    metric of the path (rows and outputs in host memory and on the GPU) and training."""
    import torch

    rng = np.random.default_rng(m * sd)
    n, k = 90_000 // m + 77, 100
    x = rng.normal(size=(n, m * sd)).astype(np.float32)
    cb = rng.normal(size=(m, k, sd)).astype(np.float32)
    for metric in ((vq.Distance.Euclidean, ka.EUCLID), (vq.Distance.SquaredEuclidean, ka.SQ), (vq.Distance.CosineDistance, ka.COSINE)):
        _check(oracle, cb, x, metric)
    q = vq.ProductQuantizer.from_codebooks(cb, vq.Distance.Euclidean)
    out, codes = q.quantize(torch.from_numpy(x).cuda(), return_codes=True)
    out_o, codes_o = oracle.pq_quantize(cb, x, ka.EUCLID)
    assert np.array_equal(codes.cpu().numpy(), codes_o) and np.array_equal(out.cpu().numpy(), out_o.view(np.float16))
    rows, iters = min(n, 3000), 5
    so, sg = RecordingSeeder(7), RecordingSeeder(7)
    init = so.init_pq(rows, m, k)
    sg.init_pq(rows, m, k)
    cb_o, _ = oracle.pq_fit(x[:rows], m, k, iters, init, so.draw)
    pq = vq.ProductQuantizer.fit(x[:rows], m, k, iters, vq.Distance.Euclidean, 7, init_idx=init, draw=sg.draw, accumulate=vq.ACCUM_ORDERED)
    assert np.array_equal(pq.codebooks, cb_o)


@pytest.mark.parametrize("k", [2, 16, 17, 33])
@pytest.mark.parametrize("m,sd", [(7, 8), (5, 4)])
def test_training_with_few_centroids_in_groups_that_are_not_full(oracle, m, sd, k):
    """Encodes of these shapes leave few centroids to the CUDA-core kernels; training does not."""
    rng = np.random.default_rng(k)
    n, iters = 2_500, 5
    x = rng.normal(size=(n, m * sd)).astype(np.float32)
    so, sg = RecordingSeeder(7), RecordingSeeder(7)
    init = so.init_pq(n, m, k)
    sg.init_pq(n, m, k)
    cb_o, _ = oracle.pq_fit(x, m, k, iters, init, so.draw)
    pq = vq.ProductQuantizer.fit(x, m, k, iters, vq.Distance.Euclidean, 7, init_idx=init, draw=sg.draw, accumulate=vq.ACCUM_ORDERED)
    assert np.array_equal(pq.codebooks, cb_o)


@pytest.mark.parametrize("m,sd,n,euclid,cosine", [(7, 8, 30_000, 36, 20), (5, 4, 60_000, 40, 24), (4, 4, 60_000, 40, 24), (4, 4, 150_000, 2, 2), (9, 4, 20_000, 40, 24),
                                                  (9, 4, 30_000, 2, 2), (8, 8, 30_000, 2, 2)])
def test_encodes_take_the_kernels_that_are_faster(m, sd, n, euclid, cosine):
    """One launch on the CUDA cores up to the line, three on the tensor cores from there on."""
    import torch

    ctx = vq.Context(0)
    x = torch.rand(n, m * sd, device="cuda")
    for distance, line in ((vq.Distance.Euclidean, euclid), (vq.Distance.SquaredEuclidean, euclid), (vq.Distance.CosineDistance, cosine)):
        for k in (line - 1, line):
            if k < 2:
                continue
            q = vq.ProductQuantizer.from_codebooks(np.random.default_rng(k).random((m, k, sd), dtype=np.float32), distance, ctx=ctx)
            before = ctx.launch_count()
            q.quantize(x)
            assert ctx.launch_count() - before == (3 if k >= line else 1), (distance, k)


@pytest.mark.parametrize("metric", ["euclid", "cosine"])
@pytest.mark.parametrize("case", ["uniform", "normal", "offset", "far", "tight", "small", "large"])
@pytest.mark.parametrize("m,sd,k", [(6, 8, 256), (5, 4, 200), (4, 8, 100)])
def test_fixed_point_scores_against_f64(ctx, m, sd, k, case, metric):
    """What the decision rests on: T = sigma S + K0 cut to a whole number lies within (-1.25, 0.25) of its value, and within 0.17 of that for
    the parts that are dropped or rounded before (the header of pq_tc.cu).  The cut is the tensor core's own, so it is measured here."""
    import ctypes as C

    from vq_b200 import _lib

    rng = np.random.default_rng(m * k + len(case))
    n = 3000
    x = rng.normal(size=(n, m * sd)).astype(np.float32)
    cb = rng.normal(size=(m, k, sd)).astype(np.float32)
    if case == "uniform":
        x, cb = rng.random(x.shape, dtype=np.float32), rng.random(cb.shape, dtype=np.float32)
    elif case == "offset":
        x, cb = x + np.float32(100), cb + np.float32(100)
    elif case == "far":
        cb[:, 7] *= 100
        x[::3] *= 50
    elif case == "tight":
        where = rng.normal(size=(8, m, sd)).astype(np.float32) * 10
        cb = (where[rng.integers(8, size=k)] + rng.normal(size=(k, m, sd)) * 1e-2).astype(np.float32).transpose(1, 0, 2).copy()
        x = (where[rng.integers(8, size=n)] + rng.normal(size=(n, m, sd)) * 1e-2).astype(np.float32).reshape(n, m * sd)
    elif case in ("small", "large"):
        scale = np.float32(1e-6 if case == "small" else 1e6)
        x, cb = x * scale, cb * scale
    t, frames, consts = np.zeros((n, m, 256), np.float32), np.zeros((n, m, 2), np.float32), np.zeros((m, 32), np.float32)
    rc = _lib.load().vqb_pq_tensor_fixed_point(ctx.handle, x.ctypes.data, n, m, sd, cb.ctypes.data, k, 2 if metric == "cosine" else 0, t.ctypes.data,
                                               frames.ctypes.data, consts.ctypes.data)
    assert rc == 0, _lib.load().vqb_last_error(ctx.handle).decode()
    sigma, k0 = frames[:, :, :1].astype(np.float64), frames[:, :, 1:].astype(np.float64)
    far = np.unpackbits(consts[:, 24:].copy().view(np.uint8), axis=1, bitorder="little")[:, :k].astype(bool)
    assert (frames[:, :, 0] > 0).mean() > 0.99 and far.sum() <= (m if case == "far" else 0)
    mu = -consts[:, :sd].astype(np.float64)
    y, c = x.astype(np.float64).reshape(n, m, sd) - mu, cb.astype(np.float64) - mu[:, None]
    if metric == "cosine":
        assert not mu.any()
        half, c = np.zeros((m, k)), c / np.linalg.norm(c, axis=-1, keepdims=True)
    else:
        half = 0.5 * (c * c).sum(-1)
    exact = sigma * (half[None] - np.einsum("nmd,mkd->nmk", y, c)) + k0
    use = (sigma > 0) & ~far[None]
    error = np.where(use, t[:, :, :k] - exact, 0.0)
    print(f"T - sigma S - K0: {error.min():.3f} .. {error.max():.3f}; T {t[:, :, :k][use].min()} .. {t[:, :, :k][use].max()}")
    assert (t == np.floor(t)).all()
    assert -1.25 - 0.17 < error.min() and error.max() < 0.25 + 0.17
    assert (exact[use] > 8 - 1).all() and (exact[use] < 65400 + 1).all()
    beyond = np.broadcast_to(sigma > 0, (n, m, 256)).copy()  # columns without a centroid, and those left out: above all others
    beyond[:, :, :k] &= far[None]
    assert (np.abs(t[beyond] - 57344) <= 1).all()


CASES = ["far", "very_far", "many_far", "offset", "tight", "equal", "nan", "tiny", "huge", "far_rows"]


def _crafted(case, rng, n, m, k):
    x = rng.normal(size=(n, m * 8)).astype(np.float32)
    cb = rng.normal(size=(m, k, 8)).astype(np.float32)
    if case == "far":                       # one centroid far away; rows near it, on the way to it and beyond
        cb[:, 7] *= 100
        x[: n // 4] = cb[:, 7].reshape(-1) * rng.random((n // 4, 1), dtype=np.float32) * 1.5
    elif case == "very_far":
        cb[:, 7] *= 1e6
        x[: n // 4] = cb[:, 7].reshape(-1) * rng.random((n // 4, 1), dtype=np.float32)
    elif case == "many_far":
        cb[:, ::5] *= 30
        x[::3] *= 30
    elif case == "offset":                  # far from the origin: only the distances to the centroids' mean count
        x += 1000
        cb += 1000
    elif case == "tight":                   # tight clusters far apart: most rows have several centroids within reach
        where = rng.normal(size=(8, m * 8)).astype(np.float32) * 10
        x = (where[rng.integers(8, size=n)] + rng.normal(size=(n, m * 8)) * 1e-3).astype(np.float32)
        cb = np.ascontiguousarray(x[rng.permutation(n)[:k]].reshape(k, m, 8).transpose(1, 0, 2))
    elif case == "equal":                   # every row ties with every centroid
        x[:] = 0.25
        cb[:] = 0.25
    elif case == "nan":
        cb[1, 3, 2] = np.nan
        cb[2, 0, 0] = np.nan
        cb[3, 5] = np.inf
        x[5, 3], x[6, 9] = np.nan, -np.inf
    elif case == "tiny":
        x *= np.float32(1e-16)
        cb *= np.float32(1e-16)
    elif case == "huge":
        x *= np.float32(1e16)
        cb *= np.float32(1e16)
    elif case == "far_rows":
        x[::2] *= np.float32(1e4)
        x[1::4] *= np.float32(1e19)
    return x, cb


@pytest.mark.parametrize("case", CASES)
def test_values_that_strain_the_fixed_point(oracle, case):
    n, m, k = 22_500, 4, 200
    x, cb = _crafted(case, np.random.default_rng(len(case)), n, m, k)
    with np.errstate(all="ignore"):
        _check(oracle, cb, x)
        _check(oracle, cb, x, (vq.Distance.SquaredEuclidean, ka.SQ))
        _check(oracle, cb, x, (vq.Distance.CosineDistance, ka.COSINE))


@pytest.mark.parametrize("case", ["far", "many_far", "offset", "tight", "equal", "far_rows"])
def test_training_on_values_that_strain_the_fixed_point(oracle, case):
    n, m, k, iters = 12_000, 4, 150, 4
    x, _ = _crafted(case, np.random.default_rng(len(case) + 1), n, m, k)
    if case == "far_rows":
        x = np.minimum(np.abs(x), np.float32(1e12))
    so, sg = RecordingSeeder(3), RecordingSeeder(3)
    init = so.init_pq(n, m, k)
    sg.init_pq(n, m, k)
    cb_o, _ = oracle.pq_fit(x, m, k, iters, init, so.draw)
    pq = vq.ProductQuantizer.fit(x, m, k, iters, vq.Distance.Euclidean, 3, init_idx=init, draw=sg.draw, accumulate=vq.ACCUM_ORDERED)
    assert np.array_equal(pq.codebooks, cb_o, equal_nan=True)


@pytest.mark.parametrize("k", [2, 3, 4, 5, 7, 9])
@pytest.mark.parametrize("case", ["equal", "equal_but_last", "wild_rows", "void"])
def test_scans_of_all_centroids(oracle, case, k):
    """Rows that look at every centroid, around the number of distances that are worked out at a time."""
    rng = np.random.default_rng(k)
    n, m = 9_000, 4
    x = rng.normal(size=(n, m * 8)).astype(np.float32)
    cb = rng.normal(size=(m, k, 8)).astype(np.float32)
    if case.startswith("equal"):
        cb[:] = cb[:, :1]
        if case == "equal_but_last":
            cb[:, -1] = np.nextafter(cb[:, -1], np.float32(100))
    elif case == "wild_rows":
        x[::3, ::5] = np.nan
        x[1::3] *= np.float32(1e19)
        x[5::7, 3] = np.inf
    else:  # a radius that leaves f32: the whole sub-space is scanned
        cb *= np.float32(1e-20)
    with np.errstate(all="ignore"):
        for metric in ((vq.Distance.Euclidean, ka.EUCLID), (vq.Distance.SquaredEuclidean, ka.SQ), (vq.Distance.CosineDistance, ka.COSINE)):
            _check(oracle, cb, x, metric)
