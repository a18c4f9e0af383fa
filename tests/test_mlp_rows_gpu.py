"""The warm-start network's kernels take rows in chunks of 32: forward with a
last chunk of 1 to 32 rows, gradients from one chunk on, against the numpy
statement with the bars of test_mlp_gpu.py."""
import numpy as np
import pytest

from oracle import mlp as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 95])
def test_rows(gpu, n):
    import torch

    from qd_imsrg_b200.warmstart import MLP

    m = MLP(0, seed=5)
    p = m.params().astype(np.float64)
    rng = np.random.default_rng(n)
    X = rng.normal(0, 1, (n, om.NI)).astype(np.float32)
    dX = torch.from_numpy(X).cuda()
    y = torch.empty(n, dtype=torch.float32, device="cuda")
    m.forward(dX, y)
    yref, _ = om.forward(p, X)
    assert np.allclose(y.cpu().numpy(), yref, rtol=2e-3, atol=2e-3 * np.abs(yref).max())
    if n % 32 == 0:
        T = rng.normal(0, 1, n).astype(np.float32)
        g = torch.empty(om.NPARAM, dtype=torch.float32, device="cuda")
        loss = m.grad(dX, torch.from_numpy(T).cuda(), g)
        gref, lref = om.grad(p, X, T)
        assert loss == pytest.approx(lref, rel=2e-3)
        assert np.linalg.norm(g.cpu().numpy() - gref) <= 5e-3 * np.linalg.norm(gref)
    m.close()
