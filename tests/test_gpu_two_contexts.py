"""Two contexts of a GPU, each driven by a thread of its own."""
import threading

import numpy as np
import pytest

import vq_b200 as vq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ks", [(1024, 640), (256, 100)])
def test_fits_with_different_numbers_of_centroids(ks):
    """The same kernels, with different needs of shared memory at the same time: neither thread's launches may depend on what the other has asked for."""
    rng = np.random.default_rng(1)
    x = rng.random((3_000, 16), dtype=np.float32)
    contexts = [vq.Context(0) for _ in ks]

    def fit(context, k):
        return vq.ProductQuantizer.fit(x, 2, k, 10, vq.Distance.Euclidean, 7, ctx=context).codebooks

    want = [fit(c, k) for c, k in zip(contexts, ks)]
    problems = []

    def work(which):
        try:
            for _ in range(100):
                if not np.array_equal(fit(contexts[which], ks[which]), want[which]):
                    problems.append(f"k {ks[which]}: other codebooks")
        except Exception as e:  # reported by the test
            problems.append(f"k {ks[which]}: {e}")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not problems, problems[:3]
