"""Plan creation for a length without a radix plan: its chirp and filter tables
(extended precision, on the host) are a few thousand products and a few hundred
sines, about a millisecond; a sum over all pairs of a 900-point convolution
takes about five."""
import time

import pytest

import dfft

pytestmark = pytest.mark.gpu


def _seconds(n):
    shape = (n, 16, 16)
    t = []
    for _ in range(6):
        start = time.perf_counter()
        plan = dfft.Plan(shape, shape, (0, 1, 2), (1, 1, 1), (1, 1, 1))
        t.append(time.perf_counter() - start)
        del plan
    return min(t[1:])  # the first one tunes the other axes


@pytest.mark.parametrize("n,smooth", [(431, 432), (449, 448), (383, 384)])
def test_chirp_tables(n, smooth):
    assert _seconds(n) <= _seconds(smooth) + 2.5e-3
