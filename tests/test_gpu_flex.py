"""Two-pass stages (lines of R1 R2 points from two register codelets, and the
chirp-z form of any other length) against the FP64 oracle.

Every codelet length appears as either radix, along the unit-stride axis and
across it; C2C and R2C both ways; blocks that divide evenly (separable
addressing), ragged ones (general tables) and exchange buffers cut along the
FFT axis; Fortran order.  Tolerances are those of the other stages: rel-L2
<= 1e-12 in FP64 and <= 1e-6 in FP32 (a transform of n <= 2^20 points in
precision eps has rel-L2 about eps log2 n: 2e-15 and 1e-6)."""
import numpy as np
import pytest

import dfft
import dfft_oracle as O
from _gpu_util import out_extents, random_input, run
from test_distributed import _case
from test_gpu_distributed import _run as _run_ranks

pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-12, "float32": 1e-6}

# both radices up to 10, up to 16, above 16 (a line each, every codelet twice),
# then lengths without a radix plan and ones whose convolution splits differently
LENGTHS = [4, 6, 12, 20, 30, 42, 56, 72, 90, 100, 22, 132, 156, 182, 210, 225, 240, 256, 125, 189, 162, 252, 300, 324,
           360, 420, 504, 600, 675, 756, 840, 960, 17, 19, 23, 31, 53, 97, 101, 113, 127, 131, 157, 257, 383]


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("n", LENGTHS)
def test_lengths(n, precision):
    """n along the unit-stride axis and across it, a tile that is not full, both directions."""
    for i, gin in enumerate([(n, 3, 11), (5, n, 18), (7, 3, n)]):
        for real in (False, True):
            plan = dfft.Plan(gin, out_extents(gin, (0, 1, 2), real), (0, 1, 2), (1, 3, 1), (3, 1, 1), real_input=real,
                             precision=precision)
            x = random_input(gin, real, 10 * n + i, precision)
            X = run(plan, x)
            ref = O.global_fft(x.astype(np.float64 if real else np.complex128), (0, 1, 2), real)
            assert O.rel_l2(X, ref) <= TOL[precision], (gin, real)
            assert O.rel_l2(run(plan, ref, forward=False), x) <= TOL[precision], (gin, real)


@pytest.mark.parametrize("layout", ["right", "left"])
@pytest.mark.parametrize("gin,tin,tout", [((30, 20, 36), (2, 2, 1), (1, 2, 2)), ((29, 25, 37), (2, 3, 1), (1, 2, 3)),
                                          ((50, 21, 26), (3, 1, 1), (1, 3, 1)), ((33, 40, 130), (1, 2, 1), (2, 1, 1))])
@pytest.mark.parametrize("real", [False, True])
def test_layouts(gin, tin, tout, layout, real):
    """even and ragged blocks, both memory orders, all normalisations."""
    axes = (0, 1, 2) if layout == "right" else (2, 1, 0)
    for norm in ("backward", "forward", "ortho", "none"):
        plan = dfft.Plan(gin, out_extents(gin, axes, real), axes, tin, tout, real_input=real, layout=layout, norm=norm)
        x = random_input(gin, real, 3)
        scale = {"backward": 1.0, "none": 1.0, "forward": 1.0 / x.size, "ortho": x.size ** -0.5}[norm]
        ref = O.global_fft(x, axes, real) * scale
        assert O.rel_l2(run(plan, x), ref) <= 1e-12
        back = run(plan, ref, forward=False)
        assert O.rel_l2(back, x * (x.size if norm == "none" else 1)) <= 1e-12


@pytest.mark.parametrize("n", [60, 131])
def test_literal_in_place(n):
    """The literal program runs the stages in place on per-rank blocks."""
    gin = (n, 20, 18)
    plan = dfft.Plan(gin, gin, (0, 1, 2), (2, 1, 1), (1, 2, 1), exec_mode="literal")
    x = random_input(gin, False, 4)
    ref = O.global_fft(x, (0, 1, 2), False)
    assert O.rel_l2(run(plan, x), ref) <= 1e-12
    assert O.rel_l2(run(plan, ref, forward=False), x) <= 1e-12


@pytest.mark.parametrize("precision", ["float64", "float32"])
@pytest.mark.parametrize("real", [False, True])
def test_exchange_buffers(real, precision):
    """Per-rank programs: lines cut into bins along the FFT axis (offsets from the axis table), padding kept zero."""
    _run_ranks(_case((20, 37, 30), (0, 1, 2), (2, 2, 1), (1, 2, 2), real), precision)


def test_batch_still_refuses_lengths_without_a_radix_plan():
    a = dfft.Plan((17, 16, 16), (17, 16, 16), (0, 1, 2), (2, 1, 1), (1, 2, 1))
    with pytest.raises(dfft.DistributedFFTError):
        dfft.Batch([a])
