"""Workspaces of the warm-start network: a network that is only evaluated
holds the two arrays its forward pass reads, 1.5 KB a row of the largest
batch (rounded up to 1,024 rows), not the gradient's."""
import pytest

from oracle import mlp as om

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65536, 262144 + 5])  # the second: in chunks of 2^18 rows
def test_forward_holds_only_its_own_arrays(gpu, n):
    import torch

    from qd_imsrg_b200.warmstart import MLP

    m = MLP(0, seed=7)
    X = torch.zeros((n, om.NI), dtype=torch.float32, device="cuda")
    y = torch.empty(n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    m.forward(X, y)
    torch.cuda.synchronize()
    held = free - torch.cuda.mem_get_info()[0]
    # H1 in bfloat16 and Z2 in float32, 256 each; allocations in 2 MiB granules
    assert held <= min(n, 1 << 18) * 256 * (2 + 4) + 2 * (2 << 20)
    m.close()
