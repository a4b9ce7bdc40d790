"""Residual encodes that are captured into a graph."""
import ctypes as C

import pytest

import vq_b200 as vq
from vq_b200 import synth

pytestmark = pytest.mark.gpu


def quantizer(seed, stages):
    return vq.ResidualQuantizer.from_codebooks((0.3 * synth.normal(stages * 256, 128, seed)).reshape(stages, 256, 128), 0.01, vq.Distance.Euclidean)


@pytest.mark.parametrize("n", [2_000, 5_000])
def test_captured_encode_replays_beside_other_encodes_of_the_context(n):
    """Codebook images, and the counter of those that are there, are the call's own: neither side sees the other's."""
    import torch

    a, b = quantizer(3, 8), quantizer(4, 5)
    xa, xb = (torch.from_numpy(synth.gaussian_mixture(rows, 128, seed)).cuda() for rows, seed in ((n, 7), (n + 777, 8)))
    want_a, want_b = (tuple(t.clone() for t in q.quantize(x, return_codes=True)) for q, x in ((a, xa), (b, xb)))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = a.quantize(xa, return_codes=True)
    torch.cuda.synchronize()
    side, main = torch.cuda.Stream(), torch.cuda.Stream()
    got_b = []
    for _ in range(200):
        with torch.cuda.stream(side):
            graph.replay()
        with torch.cuda.stream(main):
            got_b.append(b.quantize(xb, return_codes=True))
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(out, want_a))
    assert all(torch.equal(g, w) for got in got_b for g, w in zip(got, want_b))


@pytest.mark.parametrize("n", [2_000, 12_500])
def test_graph_of_an_encode_of_few_rows_has_several_instances(n):
    """A graph with memory of its own may be instantiated once at a time; such an encode needs none."""
    import torch

    x = torch.from_numpy(synth.gaussian_mixture(n, 128, 7)).cuda()
    q = quantizer(3, 8)
    want, want_codes = (t.clone() for t in q.quantize(x, return_codes=True))
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        out, codes = q.quantize(x, return_codes=True)
    runtime = C.CDLL("libcudart.so.12")
    instances = []
    try:
        for _ in range(2):
            instance = C.c_void_p()
            assert runtime.cudaGraphInstantiate(C.byref(instance), C.c_void_p(graph.raw_cuda_graph()), C.c_ulonglong(0)) == 0
            instances.append(instance)
        for instance in instances:
            out.zero_(), codes.zero_()
            torch.cuda.synchronize()
            assert runtime.cudaGraphLaunch(instance, C.c_void_p(0)) == 0
            torch.cuda.synchronize()
            assert torch.equal(out, want) and torch.equal(codes, want_codes)
    finally:
        for instance in instances:
            runtime.cudaGraphExecDestroy(instance)


@pytest.mark.parametrize("dim,k,stages,last", [(128, 256, 2, 1299), (96, 200, 4, 899), (64, 256, 8, 699), (32, 90, 2, 1949), (24, 5, 4, 1349), (61, 256, 4, 299),
                                               (33, 90, 2, 299)])
def test_encode_on_both_sides_of_the_tensor_cores_line(oracle, ctx, dim, k, stages, last):
    """The kernel for few rows needs no memory, the one on the tensor cores asks for some."""
    import numpy as np
    import torch
    from tests.util import METRICS

    x = synth.gaussian_mixture(last + 1, dim, 5)
    books = 0.2 * synth.normal(stages * k, dim, 3).reshape(stages, k, dim)
    books[0, 0], books[1, k - 1] = x[0], books[1, k // 2]
    out_o, codes_o, _ = oracle.rvq_quantize(books, 0.01, x, METRICS["Euclidean"])
    q = vq.ResidualQuantizer.from_codebooks(books, 0.01, vq.Distance.Euclidean)
    rows = torch.from_numpy(x).cuda()
    q.quantize(rows, return_codes=True) # (what the context keeps is there)
    asked = []
    for n in (last, last + 1):
        before = ctx.alloc_count()
        out, codes = q.quantize(rows[:n], return_codes=True)
        asked.append(ctx.alloc_count() - before)
        assert np.array_equal(codes.cpu().numpy(), codes_o[:n].view(np.int32))
        assert np.array_equal(out.cpu().numpy(), out_o[:n].view(np.float16), equal_nan=True)
    assert asked == [0, 1]
