"""BCH_EXPAND on a basis above 8 M entries, where a term's update of HS runs
where C_pppp is made, against the series summed from explicit commutators:
the first call (eager), and the calls that capture and replay the step."""
import numpy as np
import pytest

import qd_imsrg_b200 as qd

pytestmark = pytest.mark.gpu

# the reference's coefficients, as it writes them (magnus_IMSRG.f90, BCH_EXPAND)
COF = (1.0, 0.5, 0.166666666666666666, 0.04166666666666666, 0.0083333333333333333, 0.001388888888888, 1.984126984e-4,
       2.48015873e-5, 2.755731922e-6, 2.755731922e-7, 2.505210839e-8)


@pytest.mark.parametrize("n,R", [(2, 16), (6, 15)])
@pytest.mark.parametrize("pandya", [False, True])
def test_split_update_is_the_series(gpu, n, R, pandya):
    P = qd.Layout(n, R)
    assert P.neq >= 8_000_000
    a, b = qd.random_operator(P, -1, 31 + n), qd.random_operator(P, 1, 32 + n)
    g = np.zeros_like(a)
    mp = P.msp - n
    o = 1 + n * n + mp * mp
    g[o:o + mp * n] = 0.02 * a[o:o + mp * n]
    for q in range(P.nblock):
        nh, npp, s = int(P.dims[q, 0]), int(P.dims[q, 2]), int(P.offs[q, 2])
        g[s:s + npp * nh] = 0.02 * a[s:s + npp * nh]
    G, H, HS = qd.FullHam(P, -1, g), qd.FullHam(P, 1, b), qd.FullHam(P, 1)
    ws = [qd.FullHam(P, 1) for _ in range(5)]
    hcc, occ = qd.CCMat(P, 1.0), qd.CCMat(P, -1.0)
    nt = [qd.bch_expand(HS, G, H, *ws, hcc, occ, pandya=pandya)]
    outs = [HS.download()]
    for _ in range(3):
        nt.append(qd.bch_expand(HS, G, H, *ws, hcc, occ, pandya=pandya))
        outs.append(HS.download())
    assert len(set(nt)) == 1 and nt[0] >= 2
    X, Y = qd.FullHam(P, 1, b), qd.FullHam(P, 1)
    want = b.copy()
    for cof in COF[: nt[0]]:
        qd.commutator(G, X, Y, pandya)
        want += cof * Y.download()
        X, Y = Y, X
    # the same products in another order of additions: the bar of a commutator
    # against the oracle, on the largest entry
    for out in outs:
        assert np.abs(out - want).max() <= 1e-12 * np.abs(want).max()
