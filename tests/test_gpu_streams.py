"""Calls of one context on several streams: they share the context's scratch and have to follow each other, whoever waits for what."""
import threading

import numpy as np
import pytest

import vq_b200 as vq
from vq_b200 import synth

pytestmark = pytest.mark.gpu


def _quantizers():
    books = [synth.uniform01(16 * 256, 8, 3 + i).reshape(16, 256, 8) for i in range(2)]
    return [vq.ProductQuantizer.from_codebooks(b, vq.Distance.Euclidean) for b in books]


def test_calls_on_two_streams_follow_each_other():
    """Two quantizers, two streams, nobody waits: the operand tiles of one call are the next one's, and a
    quantizer is destroyed while its last call may still run."""
    import torch
    x = torch.from_numpy(synth.uniform01(300_000, 128, 9)).cuda()
    host = synth.uniform01(900, 128, 4)
    a, b = _quantizers()
    want = [q.quantize(x, return_codes=True)[1].clone() for q in (a, b)]
    want_host = a.quantize(host)
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.default_stream()]
    torch.cuda.synchronize()
    got = []
    for turn in range(12):
        for i, q in enumerate((a, b)):
            with torch.cuda.stream(streams[(turn + i) % 3]):
                got.append((i, q.quantize(x, return_codes=True)[1]))
        if turn % 4 == 1:
            assert np.array_equal(a.quantize(host), want_host)
        if turn % 4 == 3:
            del q
            a, b = _quantizers()
    torch.cuda.synchronize()
    for i, codes in got:
        assert torch.equal(codes, want[i])


def test_threads_with_streams_of_their_own():
    import torch
    x = torch.from_numpy(synth.uniform01(100_000, 128, 9)).cuda()
    quantizers = _quantizers()
    want = [q.quantize(x, return_codes=True)[1].clone() for q in quantizers]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            got = [quantizers[i].quantize(x, return_codes=True)[1] for _ in range(20)]
            stream.synchronize()
            wrong.extend(i for codes in got if not torch.equal(codes, want[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_a_captured_call_stays_out_of_the_order():
    import torch
    x = torch.from_numpy(synth.uniform01(50_000, 128, 9)).cuda()
    a, b = _quantizers()
    want_a, want_b = (q.quantize(x, return_codes=True)[1].clone() for q in (a, b))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        codes = a.quantize(x, return_codes=True)[1]
    got_b = b.quantize(x, return_codes=True)[1]
    graph.replay()
    assert torch.equal(codes, want_a) and torch.equal(got_b, want_b)


@pytest.mark.parametrize("m,sd,k,n", [(16, 8, 256, 30_000), (7, 8, 100, 30_000), (9, 4, 60, 30_000), (64, 4, 50, 600_000)])
def test_a_captured_encode_replays_after_larger_calls(m, sd, k, n):
    """The first call of a context may be a captured one, and its graph replays correctly after larger calls of the context and between
    them: nothing that it works with is given back meanwhile.  (Codes of up to 32 MiB lie in the context, more in the graph.)"""
    import torch
    x = torch.rand(2 * n, m * sd, device="cuda", generator=torch.Generator("cuda").manual_seed(9))
    books = synth.uniform01(m * k, sd, 3).reshape(m, k, sd)
    rows = x[:n].clone()
    want, want_all = (vq.ProductQuantizer.from_codebooks(books, vq.Distance.Euclidean).quantize(r, return_codes=True) for r in (rows, x))
    ctx = vq.Context(0)
    q = vq.ProductQuantizer.from_codebooks(books, vq.Distance.Euclidean, ctx=ctx)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, codes = q.quantize(rows, return_codes=True)
    for turn in range(3):
        out.zero_(), codes.zero_()
        graph.replay()
        assert torch.equal(codes, want[1]) and torch.equal(out, want[0])
        got = q.quantize(x, return_codes=True)  # larger than anything before it
        assert torch.equal(got[1], want_all[1]) and torch.equal(got[0], want_all[0])
        rows.copy_(x[n:] if turn == 0 else x[:n])  # the graph reads its rows anew
        graph.replay()
        assert torch.equal(codes, want_all[1][n:] if turn == 0 else want[1])
        rows.copy_(x[:n])
    del graph
