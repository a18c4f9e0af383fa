"""Gradients of the warm-start network over many chunks of 32 rows: counts
that the summing threads do not share evenly (9, 33), K slices of dW2 with a
shorter last one, and fewer rows after more in one network (the workspace is
kept); against the numpy statement with the bars of test_mlp_gpu.py."""
import numpy as np
import pytest

from oracle import mlp as om

pytestmark = pytest.mark.gpu

GROUPS = [(om.O_W1, om.O_B1), (om.O_B1, om.O_W2), (om.O_W2, om.O_B2), (om.O_B2, om.O_W3), (om.O_W3, om.O_B3),
          (om.O_B3, om.NPARAM)]


@pytest.mark.parametrize("rows", [(288,), (1056,), (8192, 96), (1056, 288, 1056)])
def test_gradient_and_loss(gpu, rows):
    import torch

    from qd_imsrg_b200.warmstart import MLP

    m = MLP(0, seed=11)
    p = m.params().astype(np.float64)
    rng = np.random.default_rng(sum(rows))
    for n in rows:
        X = rng.normal(0, 1, (n, om.NI)).astype(np.float32)
        T = rng.normal(0, 1, n).astype(np.float32)
        g = torch.empty(om.NPARAM, dtype=torch.float32, device="cuda")
        dX, dT = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
        loss = m.grad(dX, dT, g)
        got = g.cpu().numpy()
        ref, lref = om.grad(p, X, T)
        assert loss == pytest.approx(lref, rel=2e-3)
        for lo, hi in GROUPS:
            err = np.linalg.norm(got[lo:hi] - ref[lo:hi]) / max(np.linalg.norm(ref[lo:hi]), 1e-30)
            assert err < 5e-3, (n, lo, hi, err)
        assert m.grad(dX, dT, g) == loss and np.array_equal(g.cpu().numpy(), got)
    m.close()
