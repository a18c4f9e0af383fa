"""commutator_122 where one operand's one-body part couples holes to
particles only and the other operand is not generator-like on the left: from
a million entries on these run through the tiles that skip vanishing legs
(k_122_tile), with their bucketings timed on the first call.  Against the
oracle, as part of a commutator and by itself."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, numpy_random_op, part_slices
from test_known_zero_gpu import generator_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 12])
@pytest.mark.parametrize("left", ["dense", "fph, Vpphh, Vppph"])
@pytest.mark.parametrize("ha,hb", [(-1, 1), (1, -1)])
def test_against_oracle(gpu, n, left, ha, hb):
    R = 11
    O = oracle.Layout(n, R)
    assert O.neq >= 1000000
    rng = np.random.default_rng(n)
    a, b = numpy_random_op(O, ha, rng), numpy_random_op(O, hb, rng)
    if left == "dense":
        b = generator_of(O, b)  # [H, Omega]
    else:
        keep = generator_of(O, a)
        ix = dict(part_slices(O))["Vppph"]
        keep[ix] = a[ix]
        a = keep
    oA, oB = oracle.Op(O, ha, a), oracle.Op(O, hb, b)
    P = qd.Layout(n, R)
    A, B, C = qd.FullHam(P, ha, a), qd.FullHam(P, hb, b), qd.FullHam(P, 1)
    for pandya in (True, False):
        oC = oracle.Op(O, 1)
        oracle.commutator(oA, oB, oC, pandya)
        C.upload(np.full(P.neq, 7.0))
        qd.commutator(A, B, C, pandya=pandya)
        first = C.download()
        # the bar of test_onebody_gpu.py: parts that cancel hold rounding noise of their terms
        compare_parts(O, first, oC.get(), rtol=1e-12, atol=1e-14)
        qd.commutator(A, B, C, pandya=pandya)
        np.testing.assert_array_equal(C.download(), first)
    assert "masks A=" in P.tuning()
    D, oD = qd.FullHam(P, 1), oracle.Op(O, 1)
    qd.commutator_122(A, B, D)
    oracle.commutator_122(oA, oB, oD)
    compare_parts(O, D.download(), oD.get(), rtol=1e-12, atol=1e-14)
