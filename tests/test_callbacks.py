"""What runs inside a callback of a fit: the context's lock is held there, by the very thread that calls back."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name", ["test_call_lock", "test_host_wait"])
def test_host_side_waits(tmp_path, name):
    """The lock of a context knows its holder; the host's wait for a result has an end and says what it waited for."""
    exe = os.path.join(str(tmp_path), name)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-o", exe, os.path.join(ROOT, "tests", "cpp", name + ".cpp")])
    res = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=60)
    assert res.returncode == 0, res.stdout.decode()


INSIDE = """
import gc
import numpy as np
import vq_b200 as vq
from vq_b200 import synth

x = synth.uniform01(3000, 16, 5)
keep = vq.ProductQuantizer.from_codebooks(synth.uniform01(2 * 32, 8, 1).reshape(2, 32, 8), vq.Distance.Euclidean)
want = keep.quantize(x)
x[1000:] = x[0]  # dead clusters: draws
refused = []

def cyclic_garbage():
    q = vq.ProductQuantizer.from_codebooks(synth.uniform01(2 * 32, 8, 2).reshape(2, 32, 8), vq.Distance.Euclidean)
    q.self = q

def fit(inside):
    calls = []

    def draw(stream, n):
        calls.append(n)
        inside(len(calls))
        return (len(calls) * 7919) % n

    books = vq.ProductQuantizer.fit(x, 2, 64, 4, vq.Distance.Euclidean, 3, draw=draw, accumulate=vq.ACCUM_ORDERED).codebooks
    assert len(calls) > 2
    return books

def inside(call):
    if call == 1:
        gc.collect()  # destroys the quantizers of cyclic_garbage()
    if call == 2:
        try:
            keep.quantize(x)
        except vq.BackendError as e:
            refused.append(e.code)

gc.disable()
for _ in range(3):
    cyclic_garbage()
books = fit(inside)
assert refused == [104], refused
assert np.array_equal(books, fit(lambda call: None))
assert np.array_equal(keep.quantize(synth.uniform01(3000, 16, 5)), want)
print("inside ok")
"""


@pytest.mark.gpu
def test_garbage_collection_and_calls_inside_a_draw_callback():
    """Quantizers that only the garbage collector finds are destroyed inside a draw callback (the thread would wait for itself for good); a
    call there is refused; the fit goes on as if neither had happened."""
    res = subprocess.run([sys.executable, "-c", INSIDE], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=300)
    assert res.returncode == 0 and b"inside ok" in res.stdout, res.stdout.decode()[-3000:]
