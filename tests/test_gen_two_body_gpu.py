"""Two-body part of [A, B] for a generator-like A (only fph and Vpphh): 122
with every ladder, and the particle-hole channel, against the oracle.  Block sizes around the 64-row tiles,
and 1 to more than 16 hh pairs a block (the ladder panels' sizes are 4, 8 and
16; blocks with more keep the grouped GEMM); B with parts known to be zero."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, numpy_random_op, part_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(2, 4), (6, 6), (12, 8), (20, 8), (20, 10), (30, 8), (42, 9)])
@pytest.mark.parametrize("ha,hb", [(-1, 1), (1, -1), (1, 1)])
@pytest.mark.parametrize("dead", [(), ("Vpppp", "Vhhhh"), ("Vpphh",), ("Vppph", "Vphhh")])
@pytest.mark.parametrize("pandya", [False, True])
def test_generator_two_body(gpu, n, R, ha, hb, dead, pandya):
    O = oracle.Layout(n, R)
    rng = np.random.default_rng(7 * R + n)
    a, b = numpy_random_op(O, ha, rng), numpy_random_op(O, hb, rng)
    parts = dict(part_slices(O))
    g = np.zeros_like(a)
    for p in ("fph", "Vpphh"):
        g[parts[p]] = a[parts[p]]
    for p in dead:
        b[parts[p]] = 0.0
    oA, oB, oC = oracle.Op(O, ha, g), oracle.Op(O, hb, b), oracle.Op(O, 1)
    oracle.commutator(oA, oB, oC, pandya)
    P = qd.Layout(n, R)
    A, B, C = qd.FullHam(P, ha, g), qd.FullHam(P, hb, b), qd.FullHam(P, 1)
    C.upload(np.full(P.neq, 7.0))  # every entry is written
    qd.commutator(A, B, C, pandya=pandya)
    # 1e-12 relative per part, as everywhere; a part that cancels exactly in
    # the reference may hold the rounding of its terms
    compare_parts(O, C.download(), oC.get(), rtol=1e-12, atol=1e-14)
