"""E0 and the one-body part of a whole commutator of operators that conserve
(m_l, m_s), against the oracle: group sizes around the 4 x 4 register tiles
(R = 3 .. 11: one to six states a group), particle counts around the eight
per CTA, all herm combinations and a generator-like left operand; and that a
caller's write through a raw pointer is never taken for conserving."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, numpy_random_op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(2, 2), (2, 3), (6, 4), (12, 5), (6, 8), (20, 9), (12, 11)])
@pytest.mark.parametrize("ha,hb", [(-1, 1), (1, 1), (1, -1)])
@pytest.mark.parametrize("gen", [False, True])
def test_onebody_matches_oracle(gpu, n, R, ha, hb, gen):
    O = oracle.Layout(n, R)
    rng = np.random.default_rng(100 * R + n)
    a, b = numpy_random_op(O, ha, rng), numpy_random_op(O, hb, rng)
    if gen:
        g = np.zeros_like(a)
        mp = O.m - n
        o = 1 + n * n + mp * mp
        g[o:o + mp * n] = a[o:o + mp * n]
        for q in range(O.nblock):
            nh, npp, s = int(O.dims[q, 0]), int(O.dims[q, 2]), int(O.offs[q, 2])
            g[s:s + npp * nh] = a[s:s + npp * nh]
        a = g
    oA, oB, oC = oracle.Op(O, ha, a), oracle.Op(O, hb, b), oracle.Op(O, 1)
    oracle.commutator(oA, oB, oC, False)
    P = qd.Layout(n, R)
    A, B, C = qd.FullHam(P, ha, a), qd.FullHam(P, hb, b), qd.FullHam(P, 1)
    C.upload(np.full(P.neq, 7.0))
    qd.commutator(A, B, C, pandya=False)
    # 1e-12 relative per part; a part that cancels exactly in the reference
    # may hold rounding noise of its terms (entries ~ 0.1, at most m^2 terms)
    compare_parts(O, C.download(), oC.get(), rtol=1e-12, atol=1e-14)


def test_write_through_a_raw_pointer(gpu):
    import torch

    n, R = 6, 5
    O = oracle.Layout(n, R)
    rng = np.random.default_rng(3)
    a, b, c = (numpy_random_op(O, h, rng) for h in (-1, 1, 1))
    dense = numpy_random_op(O, 1, rng, conserve=False)
    P = qd.Layout(n, R)
    A, B, C, D = qd.FullHam(P, -1, a), qd.FullHam(P, 1, b), qd.FullHam(P, 1), qd.FullHam(P, -1)
    view = torch.as_tensor(qd.DeviceView(C), device="cuda")
    qd.commutator(A, B, C, pandya=False)  # C conserves (m_l, m_s) now
    P.synchronize()
    view.copy_(torch.from_numpy(dense))   # and now it does not
    torch.cuda.synchronize()
    qd.commutator(A, C, D, pandya=False)
    oA, oC, oD = oracle.Op(O, -1, a), oracle.Op(O, 1, dense), oracle.Op(O, -1)
    oracle.commutator(oA, oC, oD, False)
    compare_parts(O, D.download(), oD.get(), rtol=1e-12, atol=1e-14)
