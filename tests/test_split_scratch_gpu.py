"""The split form's programs of one commutator, which share a workspace of the
layout, against the FP64 form and against themselves."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, part_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gen", [False, True])
def test_split_programs_share_no_scratch(gen):
    """The ladders and the particle-hole product slice their operands into the
    same workspace.  Repeated commutators are bitwise equal and within the
    8-slice bar of the FP64 form (1e-12 per part), the first one included,
    whose workspaces grow."""
    n, R = 6, 10
    P, O = qd.Layout(n, R), oracle.Layout(n, R)
    a, b = qd.random_operator(P, -1, 900), qd.random_operator(P, 1, 901)
    if gen:  # only fph and Vpphh: the other branches of a generator-like operator
        parts, g = dict(part_slices(O)), np.zeros_like(a)
        for name in ("fph", "Vpphh"):
            g[parts[name]] = a[parts[name]]
        a = g
    A, B, C = qd.FullHam(P, -1, a), qd.FullHam(P, 1, b), qd.FullHam(P, 1)
    P.split = 0
    qd.commutator(A, B, C, True)
    ref = C.download()
    P.split = 8
    first = None
    for _ in range(20):
        qd.commutator(A, B, C, True)
        got = C.download()
        if first is None:
            first = got
            compare_parts(O, got, ref, 1e-12, atol=1e-14)  # a part that cancels holds its terms' rounding
        assert np.array_equal(got, first)
    for X in (A, B, C):
        X.close()
