"""Every kernel of the two-pass stage: each length of its table, and for each
convolution length a line that takes it, C2C and R2C / C2R, both ways, along
the unit-stride axis and across it, on separable and general layouts, against
the FP64 oracle (rel-L2 <= 1e-12 FP64, 1e-6 FP32, as everywhere).  Lengths that
have register kernels run it where the tuner picks it: a child process with a
tuning file that says so."""
import os
import subprocess
import sys

import pytest

from test_two_pass_lengths import groups

pytestmark = pytest.mark.gpu

PRECISIONS = ["float64", "float32"]
PLAIN = [m for g in groups("PLAIN") for m, _, _ in g]
REGISTER = [m for m, _, _ in groups("PLAIN")[0]]
CHIRP = sorted(m for g in groups("CHIRP") for m, _, _ in g)


def _line(m):
    """The longest line whose convolution has length m, and that has no radix plan."""
    for n in range((m + 1) // 2, 1, -1):
        power = 1 << (2 * n - 2).bit_length()
        rest = n
        for p in (2, 3, 5, 7, 11, 13):
            while rest % p == 0:
                rest //= p
        if rest > 1 and min(c for c in CHIRP if c >= 2 * n - 1 and 8 * c >= 5 * power) == m:
            return n
    raise AssertionError(m)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("n", sorted(set(PLAIN) - set(REGISTER)))
def test_lengths(n, precision):
    from _two_pass_child import TWO_PASS, check
    check(n, precision, TWO_PASS)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("m", CHIRP)
def test_convolution_lengths(m, precision):
    from _two_pass_child import TWO_PASS_CHIRP, check
    check(_line(m), precision, TWO_PASS_CHIRP)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_lengths_with_register_kernels(precision, tmp_path):
    cache = tmp_path / "tune"
    child = [sys.executable, os.path.join(os.path.dirname(os.path.abspath(__file__)), "_two_pass_child.py")]
    args = [precision, ",".join(map(str, REGISTER))]
    env = dict(os.environ, DFFT_TUNE_CACHE=str(cache))
    env.pop("DFFT_AUTOTUNE", None)
    subprocess.run(child + ["tune"] + args, env=env, check=True, timeout=600)
    tuned = [line.split() for line in cache.read_text().splitlines()]
    assert any(key.startswith("fast+flex:") for key, _ in tuned)
    # 400000: the two-pass kernel (Plan::autotune)
    cache.write_text("".join(f"{key} {400000 if key.startswith('fast+flex:') else value}\n" for key, value in tuned))
    done = subprocess.run(child + ["run"] + args, env=env, timeout=600, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr[-2000:]
