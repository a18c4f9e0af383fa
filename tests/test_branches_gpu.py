"""The side streams of a layout come into use after its first calls: every
call gives the bits of the first one, and the first one the oracle's values."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, numpy_random_op
from test_known_zero_gpu import generator_of

pytestmark = pytest.mark.gpu

CALLS = 8  # past the first two, which run on one stream


@pytest.mark.parametrize("n,R", [(2, 3), (6, 6), (12, 9)])
@pytest.mark.parametrize("gen", [False, True])
@pytest.mark.parametrize("pandya", [False, True])
@pytest.mark.parametrize("split", [0, 4])
def test_commutator(gpu, n, R, gen, pandya, split):
    O = oracle.Layout(n, R)
    rng = np.random.default_rng(31 * R + n)
    a, b = numpy_random_op(O, -1, rng), numpy_random_op(O, 1, rng)
    if gen:
        a = generator_of(O, a)
    P = qd.Layout(n, R)
    P.split = split
    A, B = qd.FullHam(P, -1, a), qd.FullHam(P, 1, b)
    out = [qd.FullHam(P, 1) for _ in range(CALLS)]
    for C in out:  # nothing waits between the calls
        qd.commutator(A, B, C, pandya=pandya)
    first = out[0].download()
    for C in out[1:]:
        np.testing.assert_array_equal(C.download(), first)
    if split == 0:
        oA, oB, oC = oracle.Op(O, -1, a), oracle.Op(O, 1, b), oracle.Op(O, 1)
        oracle.commutator(oA, oB, oC, pandya)
        compare_parts(O, first, oC.get(), rtol=1e-12, atol=1e-14)


def test_eom_product(gpu):
    import torch

    P = qd.Layout(6, 6)
    H = qd.FullHam(P, 1, qd.random_operator(P, 1, 4))
    v = torch.from_numpy(np.random.default_rng(2).normal(size=sum(qd.eom_dim(P, 1, 0)))).cuda()
    w = [qd.eom_matvec_target(H, 1, 0, v) for _ in range(CALLS)]
    for x in w[1:]:
        assert torch.equal(x, w[0])
