"""LRTRUNC without a tolerance: the rank is the number of singular values above zero (at most the limit),
as it is with one, and the columns beyond it are zero."""
import numpy as np
import pytest

from test_gpu_lowrank import TOL, execute
from test_gpu_vm import dev, rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("k,r", [(8, 0), (8, 3), (17, 16), (32, 5), (1, 0)])
def test_no_tolerance_drops_what_is_zero(pp, gctx, k, r):
    """The columns beyond r are exactly zero, so is the rest of the Gram matrix: nothing is rounded."""
    rng = np.random.default_rng(k + r)
    U, V = np.linalg.qr(rng.standard_normal((64, k)))[0], rng.standard_normal((50, k))
    V[:, rng.permutation(k)[r:]] = 0.0
    dU, dV, dr = dev(U), dev(V), dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=17, m=64, n=50, k=k, o=k, beta=0.0), {0: dU, 1: dV, 5: dr})
    assert dr.item() == r
    assert torch.count_nonzero(dU[:, r:]).item() == 0 and torch.count_nonzero(dV[:, r:]).item() == 0
    if r:
        assert rel(dU.cpu().numpy() @ dV.cpu().numpy().T, U @ V.T) < TOL
