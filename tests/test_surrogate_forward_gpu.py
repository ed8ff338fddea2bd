"""The fused inference kernel at the sizes where its tiles meet the grid: one block, one tile per
block, the second and third group of a block, several rounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from xyce_b200 import surrogate as S  # noqa: E402


@pytest.mark.parametrize("n", [1, 128, 129, 148 * 128, 148 * 128 + 1, 3 * 148 * 128 - 5, 3 * 148 * 128 + 1, 150_000])
def test_fused_forward_sizes(n):
    """The same BF16 roundings and products as the layer-by-layer path in the same order: equal bits."""
    rng = np.random.default_rng(n)
    net = S.SurrogateMLP(seed=6, max_batch=n)
    X = rng.uniform(-1, 1, (n, S.N_IN)).astype(np.float32)
    ref = net.forward(X).clone()
    net.Y.fill_(7.0)
    got = net.forward_fused(n)
    torch.cuda.synchronize()
    net.k.check_err()
    assert torch.equal(got, ref)
    assert (net.Y[n:] == 7.0).all()
