"""Lines whose length has a prime factor above 13 are as exact as through a
convolution of the next power of two: rel-L2 of a stack of lines against
extended precision at most q sqrt(n / 2^k), 2^k >= 2 n - 1, with q the largest
that register passes over 2^k points measured at any such length up to 512
(q hardly depends on n: a convolution's rounding errors spread over its points)."""
import numpy as np
import pytest

import dfft
from _gpu_util import out_extents, run

pytestmark = pytest.mark.gpu

Q = {("float32", "c2c"): 3.1e-7, ("float32", "c2r"): 2.9e-7, ("float64", "c2c"): 5.6e-16, ("float64", "c2r"): 5.4e-16}


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("n", [17, 41, 68, 87, 114, 131, 157, 199, 261, 263, 268, 307, 328, 373, 404, 509])
def test_as_exact_as_a_power_of_two(n, precision):
    gin = (16, 16, n)
    rng = np.random.default_rng(n)
    real, cplx = (np.float64, np.complex128) if precision == "float64" else (np.float32, np.complex64)
    power = 1 << (2 * n - 2).bit_length()
    rel = lambda a, ref: float(np.sqrt((np.abs(a - ref) ** 2).sum() / (np.abs(ref) ** 2).sum()))  # noqa: E731
    got = {}
    plan = dfft.Plan(gin, gin, (2,), (2, 1, 1), (1, 2, 1), precision=precision)
    x = (rng.standard_normal(gin) + 1j * rng.standard_normal(gin)).astype(cplx)
    got["c2c"] = rel(run(plan, x), np.fft.fft(x.astype(np.clongdouble)))
    got["c2c inverse"] = rel(run(plan, x, forward=False), np.fft.ifft(x.astype(np.clongdouble)))
    plan = dfft.Plan(gin, out_extents(gin, (2,), True), (2,), (2, 1, 1), (1, 2, 1), real_input=True, precision=precision)
    x = rng.uniform(-1, 1, gin).astype(real)
    y = np.fft.rfft(x.astype(np.longdouble)).astype(cplx)
    got["r2c"] = rel(run(plan, x), np.fft.rfft(x.astype(np.longdouble)))
    got["c2r"] = rel(run(plan, y, forward=False), np.fft.irfft(y.astype(np.clongdouble), n))
    for what, e in got.items():
        assert e <= Q[precision, "c2r" if what == "c2r" else "c2c"] * (n / power) ** 0.5, (what, e)
