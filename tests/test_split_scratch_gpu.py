"""The split form's programs of one commutator, which share a workspace of the
layout, against the FP64 form, against themselves and against the pieces."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, numpy_random_op, part_slices

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


@pytest.mark.parametrize("n,R", [(2, 4), (6, 8)])
@pytest.mark.parametrize("slices", [3, 6])
def test_split_one_body_is_the_sliced_111(n, R, slices):
    """The one-body part of a commutator in the split form is the sliced 111
    plus the FP64 121 and 221, to the bar of the plain form (1e-12 per part);
    a 111 in FP64 would differ by the slices' truncation (1e-8 with three)."""
    P, O = qd.Layout(n, R), oracle.Layout(n, R)
    rng = np.random.default_rng(n + R)
    a, b = (numpy_random_op(O, h, rng, conserve=True) for h in (-1, 1))
    A, B = qd.FullHam(P, -1, a), qd.FullHam(P, 1, b)
    C, D, w1, w2 = (qd.FullHam(P, 1) for _ in range(4))
    P.split = slices
    qd.commutator(A, B, C, True)
    qd.set_to_zero(D)
    qd.commutator_111(A, B, D)
    P.split = 0
    qd.commutator_121(A, B, D)
    qd.commutator_221(A, B, D, w1, w2)
    got, want = C.download(), D.download()
    for name, s in dict(part_slices(O)).items():
        if name in ("fhh", "fpp", "fph"):
            assert np.abs(got[s] - want[s]).max() <= 1e-12 * np.abs(want[s]).max(), name


def test_new_layouts_in_recycled_memory():
    """A layout's tables are in place before its first kernels read them, also
    in memory that an earlier layout's tables left: every new layout's first
    commutator is bitwise that of the first one, in both forms."""
    first = {}
    for k in range(8):
        n, R = ((6, 8), (12, 7))[k % 2]
        P = qd.Layout(n, R)
        A, B, C = qd.random_operator(P, -1, 5), qd.random_operator(P, 1, 6), qd.FullHam(P, 1)
        A, B = qd.FullHam(P, -1, A), qd.FullHam(P, 1, B)
        for slices in (3, 0):
            P.split = slices
            qd.commutator(A, B, C, True)
            out = C.download()
            assert np.array_equal(out, first.setdefault((n, slices), out))
        for X in (A, B, C):
            X.close()
        P.close()
