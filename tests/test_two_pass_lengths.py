"""The two-pass kernel's length table: every entry a product of two codelet
lengths, once, and the lengths that plans try beside their register kernels in
one group (the first use of a group loads its image)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "distributed-fft-for-kokkos_b200", "csrc")


def groups(form):
    """[(m, R1, R2), ...] of every group of fft_flex_lengths.h: PLAIN or CHIRP."""
    text = open(os.path.join(CSRC, "fft_flex_lengths.h")).read().replace("\\\n", " ")
    found = re.findall(r"#define DFFT_FLEX_%s_\d+\(X\)(.*)" % form, text)
    return [[tuple(map(int, x)) for x in re.findall(r"X\((\d+), (\d+), (\d+)\)", body)] for body in found]


@pytest.mark.parametrize("form", ["PLAIN", "CHIRP"])
def test_entries(form):
    entries = [e for g in groups(form) for e in g]
    codelets = {int(r) for r in re.findall(r"struct Dft<T, (\d+)>", open(os.path.join(CSRC, "fft_codelet.cuh")).read())}
    assert len(entries) == len({m for m, _, _ in entries})
    for m, r1, r2 in entries:
        assert m == r1 * r2 and r1 >= r2 and {r1, r2} <= codelets


def test_register_lengths_share_a_group():
    register = {2 ** k for k in range(4, 12)} | {3 * 2 ** k for k in range(3, 9)}
    holding = [i for i, g in enumerate(groups("PLAIN")) if register & {m for m, _, _ in g}]
    assert holding == [0]
