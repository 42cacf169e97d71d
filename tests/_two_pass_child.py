"""Child process of test_gpu_two_pass_all.py: `tune LENGTHS` creates the plans
(their stages are tuned into the file DFFT_TUNE_CACHE names), `run LENGTHS`
creates them again and checks them, every line stage on the two-pass kernel."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (os.path.join(ROOT, "distributed-fft-for-kokkos_b200"), os.path.join(ROOT, "oracle"), os.path.join(ROOT, "tests")):
    sys.path.insert(0, p)

import numpy as np  # noqa: E402

import dfft  # noqa: E402
import dfft_oracle as O  # noqa: E402
from _gpu_util import out_extents, random_input, run  # noqa: E402

TOL = {"float64": 1e-12, "float32": 1e-6}
TWO_PASS, TWO_PASS_CHIRP = 5, 6  # DFFT_KERNEL_*


def plans(n, precision):
    """n along the unit-stride axis, across it on whole (separable) and on ragged (general) layouts, tiles not full."""
    for gin, tin, tout in [((5, 3, n), (1, 3, 1), (3, 1, 1)), ((n, 3, 19), (1, 1, 1), (1, 1, 1)),
                           ((5, n, 19), (2, 1, 1), (1, 1, 2))]:
        for real in (False, True):
            yield gin, real, dfft.Plan(gin, out_extents(gin, (0, 1, 2), real), (0, 1, 2), tin, tout, real_input=real,
                                       precision=precision)


def check(n, precision, kernel):
    for gin, real, plan in plans(n, precision):
        for program in range(4):
            kernels = [s.kernel for s in plan.stages(program) if s.n == n]
            assert kernels == [kernel], (n, gin, real, program, kernels)
        x = random_input(gin, real, n, precision)
        ref = O.global_fft(x.astype(np.float64 if real else np.complex128), (0, 1, 2), real)
        assert O.rel_l2(run(plan, x), ref) <= TOL[precision], (n, gin, real)
        assert O.rel_l2(run(plan, ref, forward=False), x) <= TOL[precision], (n, gin, real)


if __name__ == "__main__":
    for length in sys.argv[3].split(","):
        if sys.argv[1] == "tune":
            for _ in plans(int(length), sys.argv[2]):
                pass
        else:
            check(int(length), sys.argv[2], TWO_PASS)
