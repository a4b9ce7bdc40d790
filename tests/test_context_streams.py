"""Which stream a call runs on when several threads share a context.  A stand-in of the library counts here, so no GPU is needed."""
import sys
import threading
import time
import types

import numpy as np
import pytest

import vq_b200 as vq
from vq_b200 import _lib


class FakeLibrary:
    """The stream is the context's, as in include/vqb.h; every call lets the other threads run, as ctypes does."""

    def __init__(self):
        self.stream, self.ran_on, self.lock = None, [], threading.Lock()

    def _set(self, stream):
        with self.lock:
            self.stream = stream
        time.sleep(0.0003)
        return 0

    def vqb_ctx_set_stream(self, handle, stream):
        return self._set(stream.value or 0)

    def vqb_ctx_reset_stream(self, handle):
        return self._set(None)

    def vqb_bq_quantize(self, handle, threshold, low, high, ptr, size, out):
        with self.lock:
            self.ran_on.append((threading.current_thread().name, self.stream))
        time.sleep(0.0003)
        return self.fails(ptr) if hasattr(self, "fails") else 0

    def vqb_last_error(self, handle):
        return self.error.encode()

    def vqb_ctx_destroy(self, handle):
        return 0


class FakeTensor:
    """As much of a CUDA tensor as the package looks at."""
    is_cuda, dtype, shape = True, "float32", (4,)

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 4096

    def numel(self):
        return 4

    def get_device(self):
        return 0

    def new_empty(self, shape, dtype=None):
        return FakeTensor()


@pytest.fixture
def fake(monkeypatch):
    library, current = FakeLibrary(), threading.local()
    torch = types.ModuleType("torch")
    torch.Tensor, torch.float32, torch.float16, torch.uint8, torch.int32 = FakeTensor, "float32", "float16", "uint8", "int32"
    torch._C = types.SimpleNamespace(_cuda_getCurrentRawStream=lambda device: current.stream)
    monkeypatch.setitem(sys.modules, "torch", torch)
    monkeypatch.setattr(_lib, "load", lambda: library)
    library.vqb_ctx_create = lambda device, out: 0
    library.vqb_bq_fit = lambda *args: 0
    library.current = current
    return library


def test_every_call_runs_on_its_own_threads_stream(fake):
    ctx = vq.Context(0)
    q = vq.BinaryQuantizer.fit(0.0, 0, 1, ctx=ctx)
    start = threading.Barrier(3)

    def work(stream):
        fake.current.stream = stream
        start.wait()
        for _ in range(60):
            q.quantize(np.zeros(4, np.float32) if stream is None else FakeTensor())

    threads = [threading.Thread(target=work, args=(s,), name=str(s)) for s in (0, 7, None)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(fake.ran_on) == 180
    wrong = [(name, stream) for name, stream in fake.ran_on if name != str(stream)]
    assert not wrong, f"{len(wrong)} of 180 calls on another thread's stream"


def test_the_stream_is_told_only_when_it_changes_and_a_pinned_one_stays(fake):
    told = []
    fake._set = lambda stream: (told.append(stream), setattr(fake, "stream", stream), 0)[2]
    ctx = vq.Context(0)
    q = vq.BinaryQuantizer.fit(0.0, 0, 1, ctx=ctx)
    for stream in (5, 5, 0, 0):
        fake.current.stream = stream
        q.quantize(FakeTensor())
    q.quantize(np.zeros(4, np.float32))
    q.quantize(np.zeros(4, np.float32))
    assert told == [5, 0, None]
    ctx.use_stream(9)
    q.quantize(FakeTensor())
    q.quantize(np.zeros(4, np.float32))
    assert told == [5, 0, None, 9] and [s for _, s in fake.ran_on[-2:]] == [9, 9]


def test_a_failure_carries_its_own_message(fake):
    """The message is the context's too: it is read before another thread's call may replace it."""
    def fails(ptr):
        mine = threading.current_thread().name
        fake.error = mine
        return 2

    fake.fails = fails
    last_error = fake.vqb_last_error
    fake.vqb_last_error = lambda handle: (time.sleep(0.0003), last_error(handle))[1]
    q = vq.BinaryQuantizer.fit(0.0, 0, 1, ctx=vq.Context(0))
    mixed = []

    def work():
        for _ in range(30):
            try:
                q.quantize(np.zeros(4, np.float32))
            except vq.InvalidParameter as e:
                if str(e) != threading.current_thread().name:
                    mixed.append(str(e))

    threads = [threading.Thread(target=work, name=f"thread {i}") for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not mixed
