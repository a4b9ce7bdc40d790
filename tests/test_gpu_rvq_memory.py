"""Residual quantizers where the rows' images (a second copy of the rows) do not fit beside them: piece by piece, same results."""
import os
import subprocess
import sys

import numpy as np
import pytest

from vq_b200 import synth

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _child(code, *args, **env):
    res = subprocess.run([sys.executable, "-c", code, *args], cwd=ROOT, env=dict(os.environ, **env), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                         timeout=600)
    assert res.returncode == 0 and b"child ok" in res.stdout, res.stdout.decode()[-3000:]


PIECES = """
import sys
import numpy as np
import vq_b200 as vq
import oracle
from tests.util import METRICS, RecordingSeeder, by_stream
from vq_b200 import synth

oracle.build()
for n, dim, k in ((1025, 128, 40), (5000, 61, 256), (2048, 32, 7)):
    x = synth.gaussian_mixture(n, dim, dim, components=5)
    so, sg = RecordingSeeder(4), RecordingSeeder(4)
    cb_o, _res, _norms = oracle.rvq_fit(x, 3, k, 4, 1e-6, METRICS["Euclidean"], so.init_stage, so.draw)
    rq = vq.ResidualQuantizer.fit(x, 3, k, 4, 1e-6, vq.Distance.Euclidean, 4, init=sg.init_stage, draw=sg.draw, accumulate=vq.ACCUM_ORDERED)
    assert np.array_equal(rq.codebooks, cb_o) and by_stream(so.draws) == by_stream(sg.draws)
for n, dim, k in ((20_001, 128, 256), (34_600, 33, 90)):
    x = synth.gaussian_mixture(n, dim, 9)
    books = 0.1 * synth.normal(3 * k, dim, 3).reshape(3, k, dim)
    books[0, :k // 2] = x[:k // 2]
    x[n - 1, dim - 1] = np.nan
    out_o, codes_o, _ = oracle.rvq_quantize(books, 0.3, x, METRICS["Euclidean"])
    q = vq.ResidualQuantizer.from_codebooks(books, 0.3, vq.Distance.Euclidean)
    out, codes = q.quantize(x, return_codes=True)
    assert np.array_equal(codes, codes_o) and np.array_equal(out, out_o.view(np.float16), equal_nan=True)
    assert np.array_equal(q.quantize(x), out, equal_nan=True)
print("child ok")
"""


@pytest.mark.parametrize("rows", ["1024", "9984"])
def test_images_of_some_rows_at_a_time_give_the_same_results(rows):
    _child(PIECES, VQB_IMAGE_ROWS=rows)


TIGHT = """
import sys
import numpy as np
import torch
import vq_b200 as vq

n, dim, mib = 1_000_000, 128, 1 << 20
x = torch.from_numpy(np.load(sys.argv[1])).cuda()
fit = lambda rows: vq.ResidualQuantizer.fit(rows, 2, 64, 4, 1e-6, vq.Distance.SquaredEuclidean, 7).codebooks
fit(x[:100_000])  # loads the kernels
torch.cuda.synchronize()
free, _ = torch.cuda.mem_get_info()
# room for the residuals (488 MiB) and some of the images (488 MiB), not for all
hog = torch.empty(free - (488 + 330) * mib, dtype=torch.uint8, device="cuda")
got, want = fit(x), np.load(sys.argv[2])
assert np.array_equal(got[0], want[0]) and np.isfinite(got).all()
print("child ok")
"""


def test_fit_where_the_images_of_all_rows_do_not_fit(tmp_path):
    """Whole numbers, whose sums are exact in any order: the same first codebook with a GPU that is all but full (the second
    stage's residuals are no whole numbers)."""
    import vq_b200 as vq
    x = np.round(8 * synth.gaussian_mixture(1_000_000, 128, 3)).astype(np.float32)
    paths = [os.path.join(str(tmp_path), f) for f in ("x.npy", "want.npy")]
    np.save(paths[0], x)
    np.save(paths[1], vq.ResidualQuantizer.fit(x, 2, 64, 4, 1e-6, vq.Distance.SquaredEuclidean, 7).codebooks)
    _child(TIGHT, *paths)
