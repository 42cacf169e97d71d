"""How the kernels of a stage address its lines, read from the host planner (no
GPU, no buffers): every kernel a stage may run must see the addressing it
handles.  The x axis of a field of 2^31 points has (n - 1) * stride < 2^31 <=
n * stride: still an affine side."""
import pytest

import dfft

OTHER, REGISTER, PAIR, PAIR_STREAM, PAIR_TMA, TWO_PASS_CHIRP = -1, 1, 2, 3, 4, 6  # DFFT_KERNEL_*


def _plan(gin, **kw):
    return dfft.Plan(gin, gin, (0, 1, 2), kw.pop("tin", (4, 4, 1)), kw.pop("tout", (1, 4, 4)), analyze_only=True, **kw)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("gin", [(1024, 1024, 2048), (512, 2048, 2048), (512, 1024, 4096), (768, 1024, 2732)])
def test_fields_of_2_31_points(gin, precision):
    """Sides whose last position lies below 2^31 elements keep base + position * stride, for whichever kernel runs."""
    reach = 0
    for program in range(4):
        stages = _plan(gin, precision=precision).stages(program)
        assert stages
        for s in stages:
            assert s.axis_table[0] == 0 and s.axis_table[1] == 0, (program, s.n, s.kernel)
            assert (s.n - 1) * max(s.stride) < 2 ** 31
            reach = max(reach, s.n * max(s.stride))
    assert reach >= 2 ** 31


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_fields_above_take_no_strided_kernel_on_tables(precision):
    """Past the bound a side is not affine: neither the TMA nor the two-line kernels may take the stage."""
    for gin in [(1024, 2048, 2048), (2048, 1024, 2048)]:
        p = _plan(gin, precision=precision)
        for program in range(4):
            for s in p.stages(program):
                if s.axis_table[0] or s.axis_table[1]:
                    assert s.kernel not in (PAIR, PAIR_STREAM, PAIR_TMA), (gin, program, s.kernel)


def test_two_pass_choice_leaves_the_addressing():
    """The two-pass kernel is a choice on these stages; sides and strides are those of the register kernels."""
    p = _plan((64, 96, 128), precision="float64")
    for program in range(4):
        for s in p.stages(program):
            assert s.two_pass and s.kernel == REGISTER and not s.axis_table[0] and not s.axis_table[1]


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("first,one_kernel", [(1, False), (2, False), (5, True), (8, True)])
def test_chirp_rows_across_a_short_axis(first, one_kernel, precision):
    """One chirp-z kernel only where its tiles (8 lines, 16 with short complex64 codelets) hold more than a quarter."""
    gin = (first, 16, 251, 32)
    p = dfft.Plan(gin, gin, (3, 2, 1), (1, 2, 1, 1), (1, 1, 1, 2), layout="left", precision=precision, analyze_only=True)
    for program in range(4):
        kernels = [s.kernel for s in p.stages(program)]
        assert (TWO_PASS_CHIRP in kernels) == one_kernel and (OTHER in kernels) != one_kernel
