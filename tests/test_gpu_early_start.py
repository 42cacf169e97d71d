"""Stages that start while the previous one drains: chains of short transforms
without synchronisation, plain and captured, give the bits of the same chain
with a synchronisation after every call; the no-allocation transform refills
its tables between calls of different shapes."""
import ctypes

import numpy as np
import pytest

import dfft
from dfft._lib import lib

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32, 32), False), ((20, 18, 30), False), ((24, 16, 40), True), ((17, 9, 23), False), ((64, 48, 32), True)]


@pytest.mark.parametrize("precision", ["float64", "float32"])
def test_unsynchronised_chain(precision):
    import torch
    cdt = torch.complex128 if precision == "float64" else torch.complex64
    rdt = torch.float64 if precision == "float64" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(3)
    work = []
    for gin, real in SHAPES:
        gout = gin[:2] + (gin[2] // 2 + 1,) if real else gin
        p = dfft.Plan(gin, gout, (0, 1, 2), (2, 1, 1), (1, 2, 1), real_input=real, precision=precision, norm="ortho")
        x = torch.randn(p.buffer_elements("in"), dtype=rdt if real else cdt, device="cuda", generator=gen)
        work.append((p, x, torch.empty(p.buffer_elements("out"), dtype=cdt, device="cuda")))

    def chain(after):
        xs = [x.clone() for _, x, _ in work]
        after()
        for _ in range(10):
            for (p, _, y), x in zip(work, xs):
                dfft.execute(p, x, y, dfft.Direction.forward, stream=torch.cuda.current_stream().cuda_stream)
                after()
                dfft.execute(p, y, x, dfft.Direction.backward, stream=torch.cuda.current_stream().cuda_stream)
                after()
        return xs

    want = chain(torch.cuda.synchronize)
    got = chain(lambda: None)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        captured = chain(lambda: None)
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, captured))


def test_no_allocation_shapes_alternate():
    import torch
    gen = torch.Generator(device="cuda").manual_seed(4)
    shapes = [(16, 32, 64), (64, 16, 32), (32, 64, 16)]
    xs = [torch.randn(s, dtype=torch.complex128, device="cuda", generator=gen) for s in shapes]
    ys = [torch.empty_like(x) for x in xs]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for _ in range(20):
        for x, y in zip(xs, ys):
            assert lib.dfft_execute_local_c2c_noalloc(ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()),
                                                      *x.shape, 0, 0, 0, stream) == 0
    torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        ref = np.fft.fftn(x.cpu().numpy())
        assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)
