"""Real lines whose length has a prime factor above 13, and ones too long for
one stage, are transformed one by one: every line of a stack has its own
precision whatever its neighbours hold (forward, backward and both adjoints,
each line against its own norm), a line of zeros stays zero, and infinities and
NaNs stay in their line.  Lengths up to 512 take one kernel, longer ones
several.

Tolerance: 2^-53 or 2^-24 times 2 log2 m + 4, m the power of two the
convolution's 2 n - 1 points fit: a convolution is two FFTs of log2 m levels,
each of at most one unit of rounding in the norm, and the two chirp products,
the filter and the scaling."""
import numpy as np
import pytest

import dfft
from _gpu_util import _TORCH, out_extents

pytestmark = pytest.mark.gpu

ROWS, COLS = 7, 6


def _plan(n, precision):
    gin = (ROWS, COLS, n)
    return dfft.Plan(gin, out_extents(gin, (2,), True), (2,), (2, 1, 1), (1, 2, 1), real_input=True, precision=precision)


def _call(plan, fn, x, direction, src, dst, real_out):
    import torch
    dbl = plan.precision == "float64"
    dt = (np.float64 if dbl else np.float32) if real_out else (np.complex128 if dbl else np.complex64)
    a = torch.from_numpy(np.ascontiguousarray(dfft.scatter_blocks(plan, x, src))).cuda()
    b = torch.empty(plan.buffer_elements(dst), dtype=_TORCH[np.dtype(dt)], device="cuda")
    fn(plan, a, b, direction)
    torch.cuda.synchronize()
    return dfft.gather_blocks(plan, b.cpu().numpy(), dst)


def _forward(plan, x):
    return _call(plan, dfft.execute, x, dfft.Direction.forward, "in", "out", False)


def _backward(plan, y):
    return _call(plan, dfft.execute, y, dfft.Direction.backward, "out", "in", True)


def _stack(n, precision, complex_):
    """Lines of sizes 1e-12 .. 1e12 in an order that puts far ones side by side, and a line of zeros."""
    rng = np.random.default_rng(n)
    shape = (ROWS, COLS, n // 2 + 1 if complex_ else n)
    x = rng.standard_normal(shape)
    if complex_:
        x = x + 1j * rng.standard_normal(shape)
    size = 10.0 ** rng.permutation(np.repeat(np.arange(-12, 13, 4), ROWS * COLS // 7 + 1)[:ROWS * COLS]).reshape(ROWS, COLS, 1)
    size[1, 2] = 0.0
    x = x * size
    if precision == "float32":
        x = x.astype(np.complex64 if complex_ else np.float32)
    return x


CASES = [(n, p) for n in (17, 31, 34, 97, 119, 131, 157, 257, 383, 509, 512 + 9, 1009, 2 * 521) for p in ("float64", "float32")]
CASES += [(8192, "float64"), (16384, "float32")]


@pytest.mark.parametrize("n,precision", CASES)
def test_lines_keep_their_precision(n, precision):
    plan = _plan(n, precision)
    m = 1 << (2 * n - 2).bit_length()
    tol = (2.0 ** -53 if precision == "float64" else 2.0 ** -24) * (2 * np.log2(m) + 4)
    x, y = _stack(n, precision, False), _stack(n, precision, True)
    w = np.full(n // 2 + 1, 0.5)
    w[0] = 1.0
    if n % 2 == 0:
        w[-1] = 1.0
    got = {"forward": (_forward(plan, x), np.fft.rfft(x.astype(np.float64))),
           "backward": (_backward(plan, y), np.fft.irfft(y.astype(np.complex128), n)),
           "adjoint of forward": (_call(plan, dfft.execute_adjoint, y, dfft.Direction.forward, "out", "in", True),
                                  n * np.fft.irfft(w * y, n)),
           "adjoint of backward": (_call(plan, dfft.execute_adjoint, x, dfft.Direction.backward, "in", "out", False),
                                   np.fft.rfft(x.astype(np.float64)) / (w * n))}
    for what, (a, ref) in got.items():
        err = np.linalg.norm(a - ref, axis=2)
        assert np.all(err <= tol * np.linalg.norm(ref, axis=2)), (what, float(np.nanmax(err / np.linalg.norm(ref, axis=2))))


@pytest.mark.parametrize("n", [17, 131, 34, 521])
@pytest.mark.parametrize("precision", ["float64", "float32"])
def test_infinities_and_nans_stay_in_their_line(n, precision):
    plan = _plan(n, precision)
    x, y = _stack(n, precision, False), _stack(n, precision, True)
    bad = [(0, 0, np.inf), (2, 3, np.nan), (6, 5, -np.inf)]
    for run, src in ((_forward, x), (_backward, y)):
        clean, dirty = src.copy(), src.copy()
        keep = np.ones((ROWS, COLS), bool)
        for i, j, v in bad:
            clean[i, j] = 0.0
            dirty[i, j, 3] = v
            keep[i, j] = False
        a, b = run(plan, clean), run(plan, dirty)
        assert np.array_equal(a[keep], b[keep])
        assert not np.any(np.isfinite(b[~keep]).all(axis=1))
