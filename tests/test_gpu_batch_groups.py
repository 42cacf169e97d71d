"""Batches whose fields share launches differently at every stage (non-cubic
fields: the groups of a stage join before the next), alone at every stage
(cubic fields: independent chains), beside fields whose stages launch on their
own (lengths without a batched tile): outputs against each plan's own
dfft_execute, rel-L2 <= 1e-12 (FP64) and 1e-6 (FP32)."""
import pytest

import dfft

pytestmark = pytest.mark.gpu

SETS = [[(32, 64, 48), (64, 32, 32), (48, 48, 64), (64, 32, 32)], [(32, 32, 32), (48, 48, 48), (32, 32, 32)],
        [(30, 32, 20), (64, 48, 32), (32, 32, 32)]]


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("shapes", SETS)
def test_groups(shapes, precision):
    import torch
    dt = torch.complex128 if precision == "float64" else torch.complex64
    tol = 1e-12 if precision == "float64" else 1e-6
    gen = torch.Generator(device="cuda").manual_seed(5)
    plans = [dfft.Plan(s, s, (0, 1, 2), (2, 2, 1), (1, 2, 2), precision=precision) for s in shapes]
    xs = [torch.randn(s[0] * s[1] * s[2], dtype=dt, device="cuda", generator=gen) for s in shapes]
    ys, zs = [torch.empty_like(x) for x in xs], [torch.empty_like(x) for x in xs]
    batch = dfft.Batch(plans)
    batch.execute(xs, ys, dfft.Direction.forward)
    batch.execute(ys, zs, dfft.Direction.backward)
    torch.cuda.synchronize()
    for p, x, y, z in zip(plans, xs, ys, zs):
        ref = torch.empty_like(x)
        dfft.execute(p, x, ref, dfft.Direction.forward)
        torch.cuda.synchronize()
        assert torch.linalg.vector_norm(y - ref) <= tol * torch.linalg.vector_norm(ref)
        assert torch.linalg.vector_norm(z - x) <= tol * torch.linalg.vector_norm(x)
