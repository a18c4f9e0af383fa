"""What the library knows to be zero in an operator is never trusted where
that may have changed: after a caller's write through a raw pointer, and in
the result of a flow, whose buffers change places."""
import numpy as np
import pytest

import oracle
import qd_imsrg_b200 as qd
from helpers import compare_parts, numpy_random_op, part_slices, synth_hamiltonian

pytestmark = pytest.mark.gpu


def generator_of(O, v):
    """fph and Vpphh of v alone."""
    g = np.zeros_like(v)
    n, mp = O.n, O.m - O.n
    o = 1 + n * n + mp * mp
    g[o:o + mp * n] = v[o:o + mp * n]
    for q in range(O.nblock):
        nh, npp, s = int(O.dims[q, 0]), int(O.dims[q, 2]), int(O.offs[q, 2])
        g[s:s + npp * nh] = v[s:s + npp * nh]
    return g


@pytest.mark.parametrize("before", ["upload", "zero", "copy"])
@pytest.mark.parametrize("pandya", [False, True])
def test_dense_write_after_a_mask_was_set(gpu, before, pandya):
    import torch

    n, R = 6, 5
    O = oracle.Layout(n, R)
    rng = np.random.default_rng(17)
    a, b = numpy_random_op(O, -1, rng), numpy_random_op(O, 1, rng)
    P = qd.Layout(n, R)
    A, B, C = qd.FullHam(P, -1), qd.FullHam(P, 1, b), qd.FullHam(P, 1)
    view = torch.as_tensor(qd.DeviceView(A), device="cuda")
    if before == "upload":
        A.upload(generator_of(O, a))
    elif before == "copy":
        qd.copy_arrays(qd.FullHam(P, -1, generator_of(O, a)), A)
    else:
        qd.set_to_zero(A)
    P.synchronize()
    view.copy_(torch.from_numpy(a))
    torch.cuda.synchronize()
    qd.commutator(A, B, C, pandya=pandya)
    oA, oB, oC = oracle.Op(O, -1, a), oracle.Op(O, 1, b), oracle.Op(O, 1)
    oracle.commutator(oA, oB, oC, pandya)
    compare_parts(O, C.download(), oC.get(), rtol=1e-12, atol=1e-14)
    assert qd.mat_2_norm(A) == pytest.approx(float(np.linalg.norm(a[1:])), rel=1e-12)
    qd.add_arrays(A, 2.0, B, 1.0, C)
    np.testing.assert_allclose(C.download(), 2.0 * a + b, rtol=1e-14, atol=1e-15)


def test_eom_product_of_a_written_hamiltonian(gpu):
    import torch

    n, R = 6, 5
    O = oracle.Layout(n, R)
    h = numpy_random_op(O, 1, np.random.default_rng(5))
    P = qd.Layout(n, R)
    H, ref = qd.FullHam(P, 1), qd.FullHam(P, 1, h)
    view = torch.as_tensor(qd.DeviceView(H), device="cuda")
    qd.set_to_zero(H)
    P.synchronize()
    view.copy_(torch.from_numpy(h))
    torch.cuda.synchronize()
    v = np.random.default_rng(6).normal(size=sum(qd.eom_dim(P, 1, 0)))
    got = np.asarray(qd.eom_matvec_target(H, 1, 0, v))
    want = np.asarray(qd.eom_matvec_target(ref, 1, 0, v))
    assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)


@pytest.mark.parametrize("steps", [1, 2])
def test_result_of_a_short_flow(gpu, steps):
    n, R = 6, 5
    O = oracle.Layout(n, R)
    rng = np.random.default_rng(23)
    h, b = synth_hamiltonian(O, rng), numpy_random_op(O, -1, rng)
    for name, ix in part_slices(O):
        if name in ("Vppph", "Vphhh"):
            h[ix] = 0.0  # in H, but not in the evolved operator
    P = qd.Layout(n, R)
    H, HS = qd.FullHam(P, 1, h), qd.FullHam(P, 1)
    f = qd.Flow(H, HS)
    for _ in range(steps):
        assert f.step().accepted
    f.close()  # HS is the caller's again
    hs = HS.download()
    ix = dict(part_slices(O))["Vppph"]
    assert np.abs(hs[ix]).max() > 1e-6
    B, C = qd.FullHam(P, -1, b), qd.FullHam(P, 1)
    qd.commutator(HS, B, C, pandya=True)
    oA, oB, oC = oracle.Op(O, 1, hs), oracle.Op(O, -1, b), oracle.Op(O, 1)
    oracle.commutator(oA, oB, oC, True)
    compare_parts(O, C.download(), oC.get(), rtol=1e-12, atol=1e-13)
