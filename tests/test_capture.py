"""Calls that a program may capture into a CUDA graph of its own, after it has
factored once by an ordinary call: the replay gives the ordinary call's bits.
Static pivots on a two-level pattern are the case in point: the ordinary
Bunch-Kaufman call runs on K's fine rows, so the captured one is the first to
need the block form."""
import ctypes

import numpy as np
import pytest

import culip_b200 as cb
from problems import kkt

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _stream(blocking):
    if not blocking:
        return torch.cuda.Stream()
    s = ctypes.c_void_p()
    assert ctypes.CDLL("libcudart.so.12").cudaStreamCreate(ctypes.byref(s)) == 0
    return torch.cuda.ExternalStream(s.value)


def _stages(F, b, out):
    for stage, source, target in ((cb.LEFT, b, out[0]), (cb.MIDDLE, out[0], out[1]), (cb.RIGHT, out[1], out[2])):
        F.apply(stage, source, target)


@pytest.mark.parametrize("blocking", [False, True])
@pytest.mark.parametrize("pivot", [cb.PIV_STATIC, cb.PIV_BK])
def test_factorization_and_stages_in_a_callers_graph(pivot, blocking):
    rp, ci, v, bs = kkt("small")
    stream = _stream(blocking)
    h = cb.Handle(0, stream)
    P = cb.Pattern(h, rp, ci, bs, 0, 1.0, cb.F64)
    F, G = cb.Factor(P), cb.Factor(cb.Pattern(cb.Handle(0), rp, ci, bs, 0, 1.0, cb.F64))
    values = torch.from_numpy(v).cuda()
    b = torch.from_numpy(cb.normal_vector(2, len(rp) - 1)).cuda()
    out, want = ([torch.zeros_like(b) for _ in range(3)] for _ in range(2))
    torch.cuda.synchronize()
    F.compute(values)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        F.compute(values, pivot=pivot)
        _stages(F, b, out)
    for scale in (1.0, 3.0):  # the buffer's contents may change between replays
        values.copy_(torch.from_numpy(v).cuda() * scale)
        torch.cuda.synchronize()
        graph.replay()
        G.compute(values, pivot=pivot)
        _stages(G, b, want)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(out, want)), scale
