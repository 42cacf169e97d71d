"""Batches whose fields share memory: an output may lie where another field's
input was (every input is read before any output is written), also where the
fields' launches would otherwise run as independent chains (cubic fields of
different lengths).  Outputs against each plan's own dfft_execute on copies,
rel-L2 <= 1e-12; the captured launches show the order without running it."""
import ctypes

import pytest

import dfft

pytestmark = pytest.mark.gpu


def _fields(lengths):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(8)
    plans = [dfft.Plan((n,) * 3, (n,) * 3, (0, 1, 2), (2, 2, 1), (1, 2, 2)) for n in lengths]
    return plans, [torch.randn(n ** 3, dtype=torch.complex128, device="cuda", generator=gen) for n in lengths]


def _roots_reach_all_leaves(call):
    import torch
    graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        call(stream.cuda_stream)
    cudart = ctypes.CDLL("libcudart.so.12")  # the one torch has loaded
    raw, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cudart.cudaGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    a, b = [(ctypes.c_void_p * n.value)() for _ in range(2)]
    data = (ctypes.c_ubyte * (8 * n.value))()
    assert cudart.cudaGraphGetEdges_v2(raw, a, b, data, ctypes.byref(n)) == 0
    after = {}
    for x, y in zip(a, b):
        after.setdefault(x, set()).add(y)
    leaves = set(b) - set(a)

    def reach(x):
        seen, todo = set(), [x]
        while todo:
            for y in after.get(todo.pop(), ()):
                if y not in seen:
                    seen.add(y)
                    todo.append(y)
        return seen

    return all(leaves <= reach(x) for x in set(a) - set(b))


def test_order_of_the_launches():
    plans, xs = _fields([32, 64])
    batch, ys = dfft.Batch(plans), [x.clone() for x in xs]
    assert not _roots_reach_all_leaves(lambda s: batch.execute(xs, ys, dfft.Direction.forward, stream=s))
    both = xs[1].new_zeros(32 ** 3 + 64 ** 3)
    for ins, outs in [(xs, [xs[1][:32 ** 3], ys[1]]), (xs, [xs[1][-32 ** 3:], ys[1]]),
                      ([both[:32 ** 3], xs[1]], [ys[0], both[32 ** 3 - 8:-8]])]:
        assert _roots_reach_all_leaves(lambda s: batch.execute(ins, outs, dfft.Direction.forward, stream=s))


def test_output_over_another_fields_input():
    import torch
    plans, xs = _fields([32, 64, 48])
    batch = dfft.Batch(plans)
    want = []
    for p, x in zip(plans, xs):
        want.append(torch.empty_like(x))
        dfft.execute(p, x, want[-1], dfft.Direction.forward)
    torch.cuda.synchronize()
    for _ in range(20):
        ins = [x.clone() for x in xs]
        other = torch.empty_like(xs[1])
        outs = [ins[1][5 * 32 ** 3:6 * 32 ** 3], other, ins[1][:48 ** 3]]
        batch.execute(ins, outs, dfft.Direction.forward)
        torch.cuda.synchronize()
        for y, ref in zip(outs, want):
            assert torch.linalg.vector_norm(y - ref) <= 1e-12 * torch.linalg.vector_norm(ref)
