"""Kernels at the sizes where a split, tile or list can go wrong, against the CPU oracle."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.util import METRICS, RecordingSeeder, by_stream
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


@pytest.mark.parametrize("name", ["SquaredEuclidean", "Euclidean", "CosineDistance", "Manhattan", "Chebyshev", "Hamming"])
@pytest.mark.parametrize("n,m,sd,k", [(1, 3, 1, 1), (1, 16, 8, 256), (63, 2, 5, 64), (65, 2, 16, 65), (9, 1, 17, 129), (1200, 4, 8, 40)])
def test_direct_encode_bit_exact(oracle, name, n, m, sd, k):
    """Few rows in one launch: every number of threads per row group (32, 64, 128) and of rows per thread, chunks of the codebook
    that are not whole, ties (duplicate centroids), a zero centroid, NaN and infinity in rows and centroids."""
    x, cb = synth.uniform(n, m * sd, 7 + n, -1.0, 1.0), synth.uniform(k, m * sd, 11 + k, -1.0, 1.0).reshape(k, m, sd).transpose(1, 0, 2).copy()
    if k > 4:
        cb[:, k - 1] = cb[:, 1]
        cb[:, 2] = 0.0
    if n > 8:
        x[3], x[4, 0], x[5, :sd], x[6] = 0.0, np.nan, np.inf, 1e30
        x[8, :sd] = cb[0, min(1, k - 1)]
        cb[0, k // 2, 0] = np.nan
        cb[m - 1, k - 2, sd - 1] = np.inf
    out_o, codes_o = oracle.pq_quantize(cb, x, METRICS[name])
    out, codes = vq.ProductQuantizer.from_codebooks(cb, getattr(vq.Distance, name)).quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(out, out_o.view(np.float16), equal_nan=True)


@pytest.mark.parametrize("m,sd,k,last", [(16, 8, 256, 686), (4, 8, 100, 4540), (8, 8, 33, 3371), (5, 4, 256, 11_200), (3, 8, 20, 6666), (4, 5, 100, 7000)])
def test_encode_on_both_sides_of_the_line_between_the_kernels(oracle, ctx, m, sd, k, last):
    """`last` rows are the most that one launch encodes, one more goes to the kernels for many rows (three launches where the tensor
    cores take the shape): both give the oracle's codes."""
    cb = synth.uniform(k, m * sd, 11 + k, -1.0, 1.0).reshape(k, m, sd).transpose(1, 0, 2).copy()
    cb[:, k - 1] = cb[:, 1]
    x = synth.uniform(last + 1, m * sd, 7, -1.0, 1.0)
    x[5] = cb[:, 1].reshape(-1)
    x[last // 2, 0] = np.nan
    out_o, codes_o = oracle.pq_quantize(cb, x, METRICS["Euclidean"])
    q = vq.ProductQuantizer.from_codebooks(cb, vq.Distance.Euclidean)
    launches = []
    for n in (last, last + 1):
        before = ctx.launch_count()
        out, codes = q.quantize(x[:n], return_codes=True)
        launches.append(ctx.launch_count() - before)
        assert np.array_equal(codes, codes_o[:n])
        assert np.array_equal(out, out_o[:n].view(np.float16), equal_nan=True)
    assert launches[0] == 1 and (launches[1] == 3 if sd == 8 and m % 4 == 0 else launches[1] >= 1)


@pytest.mark.parametrize("dim,k,last", [(128, 256, 12_500), (61, 256, 12_499), (33, 90, 34_500), (24, 5, 106_250)])
def test_residual_encode_on_both_sides_of_the_line_between_the_kernels(oracle, ctx, dim, k, last):
    """As above: one launch for all stages, or several per stage."""
    x = synth.gaussian_mixture(last + 1, dim, 5)
    books = 0.2 * synth.normal(2 * k, dim, 3).reshape(2, k, dim)
    books[0, 0], books[1, k - 1] = x[0], books[1, k // 2]
    out_o, codes_o, _ = oracle.rvq_quantize(books, 0.01, x, METRICS["Euclidean"])
    q = vq.ResidualQuantizer.from_codebooks(books, 0.01, vq.Distance.Euclidean)
    launches = []
    for n in (last, last + 1):
        before = ctx.launch_count()
        out, codes = q.quantize(x[:n], return_codes=True)
        launches.append(ctx.launch_count() - before)
        assert np.array_equal(codes, codes_o[:n])
        assert np.array_equal(out, out_o[:n].view(np.float16), equal_nan=True)
    assert launches[0] == 1 < launches[1]


@pytest.mark.parametrize("name", ["SquaredEuclidean", "Euclidean", "CosineDistance", "Manhattan"])
@pytest.mark.parametrize("n,dim,k,stages", [(1, 128, 256, 8), (17, 33, 64, 3), (40, 15, 7, 2), (700, 64, 130, 4)])
def test_direct_residual_encode_bit_exact(oracle, name, n, dim, k, stages):
    """All stages in one launch: rows that end early (their residual is a centroid), ties, NaN rows, ragged chunks."""
    x = synth.gaussian_mixture(n, dim, 5)
    books = 0.2 * synth.normal(stages * k, dim, 3).reshape(stages, k, dim)
    books[0, 0] = x[0]
    if n > 8:
        x[5, dim - 1] = np.nan
        books[1, k - 1] = books[1, k // 2]
    out_o, codes_o, _ = oracle.rvq_quantize(books, 0.01, x, METRICS[name])
    out, codes = vq.ResidualQuantizer.from_codebooks(books, 0.01, getattr(vq.Distance, name)).quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(out, out_o.view(np.float16), equal_nan=True)


@pytest.mark.parametrize("n,m,k", [(3000, 16, 256), (4097, 12, 200), (30_000, 4, 33)])
@pytest.mark.parametrize("special", [False, True])
def test_cosine_encode_on_tensor_cores_bit_exact(oracle, n, m, k, special):
    """Unit vectors on the tensor cores, near-ties to the exact scan: parallel centroids, zero, tiny, huge and NaN norms on both
    sides (each voids what it has to)."""
    rng = np.random.default_rng(n + k)
    x, cb = rng.normal(size=(n, m * 8)).astype(np.float32), rng.normal(size=(m, k, 8)).astype(np.float32)
    cb[:, 7] = 2.0 * cb[:, 3]          # the same direction: distances differ in the last bits only
    x[:50] = cb[:, 3].reshape(-1)
    if special:
        cb[0, 5], cb[1, 0, 2], cb[2, 9] = 0.0, np.nan, cb[2, 9] * 1e-30
        cb[3, 11] = 1e25
        x[60], x[61], x[62], x[63, 1] = 0.0, x[61] * 1e-25, x[62] * 1e20, np.nan
    q = vq.ProductQuantizer.from_codebooks(cb, vq.Distance.CosineDistance)
    out, codes = q.quantize(x, return_codes=True)
    out_o, codes_o = oracle.pq_quantize(cb, x, METRICS["CosineDistance"])
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(out, out_o.view(np.float16), equal_nan=True)


@pytest.mark.parametrize("n,dim,k", [(2000, 17, 2), (1300, 33, 31), (700, 61, 256), (1025, 100, 40), (3000, 128, 200)])
def test_full_width_training_of_any_width_bit_exact(oracle, n, dim, k):
    """Images padded to whole K steps (dim not a multiple of 16, rows not a multiple of 16 bytes), dead clusters, residual updates
    with the next stage's images."""
    from tests.golden import reference_known_answers as ka
    x = synth.gaussian_mixture(n, dim, dim, components=5)
    x[n // 2: n // 2 + 40] = x[3]
    so, sg = RecordingSeeder(4), RecordingSeeder(4)
    cb_o, _res, _norms = oracle.rvq_fit(x, 3, k, 4, 1e-6, ka.EUCLID, so.init_stage, so.draw)
    rq = vq.ResidualQuantizer.fit(x, 3, k, 4, 1e-6, vq.Distance.Euclidean, 4, init=sg.init_stage, draw=sg.draw, accumulate=vq.ACCUM_ORDERED)
    assert np.array_equal(rq.codebooks, cb_o) and by_stream(so.draws) == by_stream(sg.draws)


@pytest.mark.parametrize("n,dim,k", [(180_001, 61, 40), (70_000, 128, 33)])
def test_large_residual_encode_with_rows_that_end_early_bit_exact(oracle, n, dim, k):
    x = synth.gaussian_mixture(n, dim, 9)
    books = 0.1 * synth.normal(3 * k, dim, 3).reshape(3, k, dim)
    books[0, :k // 2] = x[:k // 2]
    books[2, 5] = books[2, 1]
    eps = float(np.float32(np.sqrt(np.sum((x[k] - books[0, 1]).astype(np.float64) ** 2))))  # some rows end within rounding of it
    x[100:100 + k // 2] = x[:k // 2]
    x[n - 1, dim - 1], x[n - 2, 0] = np.nan, np.inf
    out_o, codes_o, _ = oracle.rvq_quantize(books, eps, x, METRICS["Euclidean"])
    out, codes = vq.ResidualQuantizer.from_codebooks(books, eps, vq.Distance.Euclidean).quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o)
    assert np.array_equal(out, out_o.view(np.float16), equal_nan=True)


def test_image_dot_products_within_half_of_the_bound(ctx):
    from tests.test_gpu_dense_tc import _dots
    for n, dim, k, scale in ((1000, 128, 256, 1.0), (777, 61, 100, 1e3), (4097, 17, 2, 1e-4)):
        rng = np.random.default_rng(n)
        x, cb = (scale * rng.normal(size=(n, dim))).astype(np.float32), (scale * rng.normal(size=(k, dim))).astype(np.float32)
        dots, _ = _dots(ctx, x, cb)
        err = np.abs(dots[:, :k] - x.astype(np.float64) @ cb.astype(np.float64).T)
        # (the half norm is added back in f32 for this comparison: its own rounding is allowed for)
        norm = np.linalg.norm(x, axis=1)[:, None] * np.linalg.norm(cb, axis=1).max() + (np.linalg.norm(cb, axis=1) ** 2)[None, :] * 0.01
        assert (err <= 3.5e-6 * norm).all(), float((err / norm).max())


@pytest.mark.parametrize("n,dim,depth", [(1, 5, 3), (2, 33, 3), (1025, 7, 12), (2049, 64, 4), (9000, 40, 3), (20_000, 32, 6), (5000, 1, 20)])
def test_tree_build_bit_exact(oracle, n, dim, depth):
    """One-warp and streaming statistics, odd widths, nodes of one CTA and of a cluster, levels beyond the ones the host launches
    blindly, heavily repeated values (ranks inside runs of equal keys, nodes that cannot be split), negative values and zeros."""
    x = synth.normal(n, dim, n + dim)
    x[:, 0] = np.round(2 * x[:, 0]) * 40
    x[n // 2:, dim // 2] = -0.0
    cent_o, left_o, right_o = oracle.tsvq_fit(x, depth)
    cent, left, right = vq.TSVQ(x, depth, vq.Distance.Euclidean).tree()
    assert np.array_equal(left, left_o) and np.array_equal(right, right_o)
    assert np.array_equal(cent, cent_o)


@pytest.mark.parametrize("n,m,sd,k,skew", [(70_000, 16, 8, 256, False), (66_000, 5, 4, 17, False), (9000, 3, 16, 256, True),
                                           (70_001, 7, 12, 100, True), (4097, 2, 32, 256, False), (66_001, 1, 100, 256, True), (5000, 2, 36, 33, False), (1, 1, 8, 1, False), (140_000, 6, 8, 200, True)])
def test_unordered_sums_follow_the_rows(n, m, sd, k, skew):
    """Small whole numbers have sums that are exact in any order, so unordered sums (all rows in the first iteration, moved rows
    after it) must train the same codebooks as ordered ones: one to four sub-spaces per CTA, rows in no whole pieces, queues
    that run over because most rows share a cluster."""
    x = np.round(4 * synth.normal(n, m * sd, n + sd)).astype(np.float32)
    if skew:
        x[: n - n // 8] = x[0]
    init = np.stack([np.random.default_rng(s).permutation(n)[:k] for s in range(m)]).astype(np.uint32)
    fast, ordered = (vq.ProductQuantizer.fit(x, m, k, 6, vq.Distance.SquaredEuclidean, 1, init_idx=init, accumulate=a) for a in (vq.ACCUM_FAST, vq.ACCUM_ORDERED))
    assert np.array_equal(fast.codebooks, ordered.codebooks)


@pytest.mark.parametrize("metric", ["Euclidean", "SquaredEuclidean"])
@pytest.mark.parametrize("n,dim", [(1, 3), (5, 32), (203, 33), (130, 64), (77, 100), (66, 127), (1030, 256), (40, 260)])
def test_tree_lookup_exact_where_the_children_are_close(oracle, n, dim, metric):
    """Rows on the children's midplane (ties and last-bit differences decide), NaN, infinities, values whose squares vanish or
    overflow; rows in whole 16-byte pieces and not, one to eight pieces per lane, and the width above which the tile kernel runs."""
    x = synth.normal(n + 400, dim, n * dim)
    distance = getattr(vq.Distance, metric)
    tree = vq.TSVQ(x[n:], 6, distance)
    cent, left, right = tree.tree()
    x = x[:n].copy()
    inner = np.flatnonzero((left >= 0) & (right >= 0))
    for i in range(0, n, 2):
        j = inner[i % len(inner)]
        x[i] = (cent[left[j]] + cent[right[j]]) / 2
    for i, v in zip(range(3, n, 7), [np.nan, np.inf, -np.inf, 1e30, 1e-30, 2e19, 0.0]):
        x[i, i % dim:] = v
    got, leaf = tree.quantize(x, return_leaf=True)
    want, leaf_o = oracle.tsvq_quantize(cent, left, right, x, METRICS[metric])
    assert np.array_equal(np.asarray(leaf), leaf_o)
    assert np.array_equal(np.asarray(got).view(np.uint16), want)
