"""Which launches may start while the one before them in the stream drains:
those that read at most 128 MB, of one field or of a batch (its fields
together).  Read from the edges of the captured launches (a programmatic
dependency, or a full one)."""
import ctypes

import pytest

import dfft

pytestmark = pytest.mark.gpu


def _programmatic_edges(call):
    import torch
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    stream = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        call(stream.cuda_stream)
    cudart = ctypes.CDLL("libcudart.so.12")  # the one torch has loaded
    raw, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cudart.cudaGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    nodes = [(ctypes.c_void_p * n.value)() for _ in range(2)]
    data = (ctypes.c_ubyte * (8 * n.value))()  # cudaGraphEdgeData: from_port, to_port, type, 5 reserved bytes
    assert cudart.cudaGraphGetEdges_v2(raw, nodes[0], nodes[1], data, ctypes.byref(n)) == 0
    return sum(t == 1 for t in data[2::8]), n.value  # cudaGraphDependencyTypeProgrammatic


@pytest.mark.parametrize("n,count,early", [(64, 3, True), (192, 1, True), (192, 5, False), (384, 1, False)])
def test_rule(n, count, early):
    import torch
    shape = (n, n, n)
    plans = [dfft.Plan(shape, shape, (0, 1, 2), (2, 2, 1), (1, 2, 2), precision="float32") for _ in range(count)]
    xs = [torch.zeros(n ** 3, dtype=torch.complex64, device="cuda") for _ in plans]
    ys = [torch.empty_like(x) for x in xs]
    calls = []
    if count == 1:
        calls.append(lambda s: dfft.execute(plans[0], xs[0], ys[0], dfft.Direction.forward, stream=s))
    batch = dfft.Batch(plans)
    calls.append(lambda s: batch.execute(xs, ys, dfft.Direction.forward, stream=s))
    for call in calls:
        call(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        programmatic, edges = _programmatic_edges(call)
        assert edges == 2 and programmatic == (2 if early else 0)
