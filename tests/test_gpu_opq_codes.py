"""The cross-covariance whose first factor is gathered from codes (no reconstruction in memory) against f64."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.golden import reference_known_answers as ka

pytestmark = pytest.mark.gpu


# rows of a stage (32), of a CTA's share and of all SMs not full; sub-spaces of 4 and 8 values; codebooks up to a byte's last code
@pytest.mark.parametrize("n,dim,m,k,metric", [(32 * 148 * 3 + 1, 128, 16, 256, "Euclidean"), (4096, 128, 32, 256, "SquaredEuclidean"),
                                              (20_031, 32, 4, 37, "Euclidean"), (33_000, 32, 8, 16, "SquaredEuclidean"),
                                              (9_999, 96, 12, 200, "CosineDistance"), (7_777, 64, 16, 255, "Euclidean")])
def test_rotation_of_one_outer_iteration(oracle, n, dim, m, k, metric):
    """src/opq.rs:146-183 from the identity: A = sum y x^T with y the centroids of the oracle's codes, rotation = V U^T, the
    transposed polar factor of A.  The last row weighs as much as all others, the first a tenth."""
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, dim)).astype(np.float32)
    x[-1] *= np.float32(np.sqrt(n))
    x[0] *= np.float32(np.sqrt(0.1 * n))
    oq = vq.OptimizedProductQuantizer.fit(x, m, k, 2, 1, getattr(vq.Distance, metric), 5)
    cb = oq.codebooks
    name = {"Euclidean": ka.EUCLID, "SquaredEuclidean": ka.SQ, "CosineDistance": ka.COSINE}[metric]
    _, codes = oracle.opq_quantize(np.eye(dim, dtype=np.float32), cb, x, name)
    y = np.concatenate([cb[s][codes[:, s]] for s in range(m)], axis=1).astype(np.float64)
    a = y.T @ x.astype(np.float64)
    u, sv, vt = np.linalg.svd(a)
    # the entries of A carry 4e-6 of the sum of their terms' magnitudes (as the product of two matrices in memory); a polar factor moves by at
    # most |dA|_F / sigma_min, and is rounded to f32 (entries up to 1) after an iteration that ends at 1e-6
    bound = 4e-6 * np.linalg.norm(np.abs(y).T @ np.abs(x)) / sv[-1] + 2e-6
    assert bound < 0.05, bound
    assert np.linalg.norm(oq.rotation - (u @ vt).T) <= bound
