"""Navier-Stokes right-hand side on kept modes (line kernels along x, y, z)
and its adjoint, on the grids where they can go wrong: an odd number of grid
lines (the last has no partner), odd lengths, tiny axes, radices above 16
along each axis, tiles that are not full, and grids whose axes the kernels do
not take (the plan's transforms).  Forward against the numpy oracle, rel-L2 <=
1e-12 (FP64) and 1e-5 (FP32), the tolerances of the other solver tests; the
adjoint by <J d, c> = <d, J^T c>, where J d = (f(y + d) - f(y - d)) / 2 exactly
(f is quadratic), so the identity holds to rounding: 1e-12 of |J d| |c|
against about 1e-15 sqrt(terms)."""
import numpy as np
import pytest

import dfft
import ns_oracle as N

pytestmark = pytest.mark.gpu

NU, DT, LX = 0.01, 0.01, 2.0
ONE, PENCIL = ((1, 1, 1, 1), (1, 1, 1, 1)), ((1, 2, 2, 1), (1, 1, 2, 2))
GRIDS = [((9, 15, 20), PENCIL), ((25, 15, 36), PENCIL), ((8, 9, 8), ONE), ((12, 9, 15), PENCIL), ((50, 25, 12), PENCIL),
         ((320, 8, 8), PENCIL), ((8, 300, 8), PENCIL), ((8, 9, 360), PENCIL), ((8, 12, 512), ONE), ((48, 32, 64), PENCIL),
         ((17, 16, 16), PENCIL), ((16, 16, 11), ONE), ((4, 6, 8), ONE)]


def _plan(shape, topo, precision):
    nx, ny, nz = shape
    return dfft.Plan((3, nx, ny, nz), (3, nx, ny, nz // 2 + 1), (1, 2, 3), *topo, real_input=True, precision=precision)


def _spectrum(shape, seed):
    rng = np.random.default_rng(seed)
    k, _, inv = N.wavenumbers(*shape, LX)
    return N.projection(np.fft.rfftn(rng.standard_normal((3,) + shape), axes=(1, 2, 3)), k, inv)


def _dev(plan, a, precision):
    import torch
    c = np.complex128 if precision == "float64" else np.complex64
    return torch.from_numpy(np.ascontiguousarray(dfft.scatter_blocks(plan, a.astype(c), "out"))).cuda()


def _host(plan, t):
    return dfft.gather_blocks(plan, t.cpu().numpy(), "out").astype(np.complex128)


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a - b)) / np.linalg.norm(np.ravel(b)))


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("shape,topo", GRIDS)
def test_rhs_and_step(shape, topo, precision):
    import torch
    tol = 1e-12 if precision == "float64" else 1e-5
    plan = _plan(shape, topo, precision)
    ns = dfft.NavierStokes(plan, nu=NU, dt=DT, lx=LX)
    y = _spectrum(shape, 1)
    uk = _dev(plan, y, precision)
    dukdt = torch.full_like(uk, float("nan"))
    ns.rhs(uk, dukdt)
    ref_u, ref_f = N.rhs(y, NU, LX, shape)
    assert _rel(_host(plan, uk), ref_u) <= tol
    assert _rel(_host(plan, dukdt), ref_f) <= tol
    # cut modes hold zeros
    cut = N.alias_mask(*shape) == 0
    assert not _host(plan, dukdt)[:, cut].any() and not _host(plan, uk)[:, cut].any()
    uk = _dev(plan, y, precision)
    ns.step(uk)
    assert _rel(_host(plan, uk), N.rk4_step(y, NU, DT, LX, shape)) <= tol


@pytest.mark.parametrize("shape,topo", GRIDS)
def test_rhs_adjoint(shape, topo):
    import torch
    plan = _plan(shape, topo, "float64")
    ns = dfft.NavierStokes(plan, nu=NU, dt=DT, lx=LX)
    y, d, c = (_dev(plan, _spectrum(shape, s), "float64") for s in (1, 2, 3))

    def rhs(v):
        out = torch.empty_like(v)
        ns.rhs(v.clone(), out)
        return out

    jd = (rhs(y + d) - rhs(y - d)) / 2
    jtc = torch.full_like(y, float("nan"))
    ns.rhs_adjoint(y, c, jtc)
    lhs = float((jd.conj() * c).real.sum())
    rhs_ = float((d.conj() * jtc).real.sum())
    assert abs(lhs - rhs_) <= 1e-12 * float(torch.linalg.vector_norm(jd) * torch.linalg.vector_norm(c))


@pytest.mark.parametrize("precision", ["float64", "float32"])
def test_step_graph_mixed_fields(precision):
    """fields the line kernels take beside one they do not, in one graph."""
    import torch
    tol = 1e-12 if precision == "float64" else 1e-5
    states, uks, refs = [], [], []
    for i, shape in enumerate([(16, 20, 24), (16, 16, 11), (10, 9, 12), (9, 15, 12)]):
        plan = _plan(shape, PENCIL, precision)
        y = _spectrum(shape, i)
        states.append(dfft.NavierStokes(plan, nu=NU, dt=DT, lx=LX))
        uks.append(_dev(plan, y, precision))
        refs.append((plan, N.rk4_step(y, NU, DT, LX, shape)))
    for batched in (True, False):
        run = [u.clone() for u in uks]
        dfft.step_graph(states, run, batched=batched).launch()
        torch.cuda.synchronize()
        for u, (plan, ref) in zip(run, refs):
            assert _rel(_host(plan, u), ref) <= tol
