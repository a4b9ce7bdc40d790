"""Product-quantizer encodes where the working memory of the tensor path (a byte per row and sub-space) does not fit: piece by piece, with the
same results."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _child(code, *args, **env):
    res = subprocess.run([sys.executable, "-c", code, *args], cwd=ROOT, env=dict(os.environ, **env), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                         timeout=600)
    assert res.returncode == 0 and b"child ok" in res.stdout, res.stdout.decode()[-3000:]


PIECES = """
import numpy as np
import torch
import vq_b200 as vq
import oracle
from tests.golden import reference_known_answers as ka

oracle.build()
rng = np.random.default_rng(8)
for n, m, sd, k in ((9_999, 16, 8, 256), (13_313, 9, 4, 100), (20_481, 7, 8, 64)):
    x = rng.random((n, m * sd), dtype=np.float32)
    cb = rng.random((m, k, sd), dtype=np.float32)
    for dist, name in ((vq.Distance.Euclidean, ka.EUCLID), (vq.Distance.CosineDistance, ka.COSINE)):
        q = vq.ProductQuantizer.from_codebooks(cb, dist)
        out_o, codes_o = oracle.pq_quantize(cb, x, name)
        out, codes = q.quantize(torch.from_numpy(x).cuda(), return_codes=True)
        assert np.array_equal(codes.cpu().numpy(), codes_o) and np.array_equal(out.cpu().numpy(), out_o.view(np.float16))
        out, codes = q.quantize(x, return_codes=True)
        assert np.array_equal(codes, codes_o) and np.array_equal(out, out_o.view(np.float16))
print("child ok")
"""


@pytest.mark.parametrize("rows", ["128", "6656"])
def test_codes_of_some_rows_at_a_time_give_the_same_results(rows):
    _child(PIECES, VQB_CODE_ROWS=rows)


TIGHT = """
import sys
import torch
import vq_b200 as vq
from vq_b200 import synth

n, m, sd, k, mib = 6_000_000, 32, 4, 64, 1 << 20
cb = synth.uniform01(m * k, sd, 3).reshape(m, k, sd)
q = vq.ProductQuantizer.from_codebooks(cb, vq.Distance.Euclidean)
x = torch.rand(n, m * sd, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
out = torch.empty(n, m * sd, device="cuda", dtype=torch.float16)
q.quantize(x[:100_000], out=out[:100_000])  # loads the kernels
torch.cuda.synchronize()
free, _ = torch.cuda.mem_get_info()
hog = torch.empty(free - int(sys.argv[1]) * mib, dtype=torch.uint8, device="cuda")
q.quantize(x, out=out)  # 183 MiB of codes
torch.cuda.synchronize()
del hog
torch.cuda.empty_cache()  # (the comparison loads kernels of its own)
books = torch.from_numpy(cb).cuda()
for r0 in (0, 1_234_567, n - 5000):
    _, codes = q.quantize(x[r0:r0 + 5000], return_codes=True)  # the one-launch kernel
    want = torch.stack([books[s][codes[:, s].long()] for s in range(m)], dim=1).reshape(5000, -1).half()
    assert torch.equal(out[r0:r0 + 5000], want)
print("child ok")
"""


@pytest.mark.parametrize("mib", [120, 16])
def test_encode_in_a_gpu_that_is_all_but_full(mib):
    _child(TIGHT, str(mib))
