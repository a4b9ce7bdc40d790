"""The rotation matrix of the optimized product quantizer (polar factor in f64) at the edges of its tiles: one 16 x 16 tile, chunks of 128 values that
are not full, several of them, and matrices whose tiles need the kernel with few registers."""
import numpy as np
import pytest

import vq_b200 as vq
from tests.golden import reference_known_answers as ka

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,m", [(16, 4), (48, 3), (112, 14), (144, 18), (272, 34), (288, 36), (400, 50), (512, 64)])
def test_rotation_is_the_polar_factor(oracle, dim, m):
    """src/opq.rs:172-190 from the identity: A = sum y x^T, rotation = V U^T."""
    n, k = 4000, 64
    rng = np.random.default_rng(dim)
    # directions of weight 1 to 1/2 keep A far from singular and from a multiple of an orthogonal matrix
    x = (rng.normal(size=(n, dim)) * np.geomspace(1.0, 0.5, dim)).astype(np.float32)
    oq = vq.OptimizedProductQuantizer.fit(x, m, k, 2, 1, vq.Distance.Euclidean, 5)
    cb = oq.codebooks
    _, codes = oracle.opq_quantize(np.eye(dim, dtype=np.float32), cb, x, ka.EUCLID)
    y = np.concatenate([cb[s][codes[:, s]] for s in range(m)], axis=1).astype(np.float64)
    u, sv, vt = np.linalg.svd(y.T @ x.astype(np.float64))
    # entries of A: 4e-6 of the sum of their terms' magnitudes (f32 products and partial sums); a polar factor moves by at most
    # |dA|_F / sigma_min; rounded to f32 at the end: dim entries of 2^-25 in a Frobenius norm
    bound = 4e-6 * np.linalg.norm(np.abs(y).T @ np.abs(x)) / sv[-1] + dim * 2.0 ** -25 + 1e-9
    assert bound < 0.05, bound
    assert np.linalg.norm(oq.rotation - (u @ vt).T) <= bound
