"""The fused training step against the layer-by-layer one on the same network and batch: sizes around
a 128-row tile and around one tile per block, and several tiles per block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from xyce_b200 import surrogate as S  # noqa: E402


@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 128, 148 * 128 + 1, 40_000])
def test_fused_training_step_matches_layer_by_layer(n):
    """Both round the same activations and gradients to BF16 and sum the same FP32 products over the
    batch, in different orders: chains of at most 256 + 148 additions on either side, so a sum
    differs by at most 2 x 404 x 2^-24 = 4.9e-5 of the sum of its terms' magnitudes. Adam's first
    step moves a weight by lr g / (|g| + eps): at most lr, and the same where the gradients are."""
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (n, S.N_IN)).astype(np.float32)
    T = rng.standard_normal((n, S.N_OUT)).astype(np.float32)
    a, b = (S.SurrogateMLP(seed=3, max_batch=n) for _ in range(2))
    cfg = S.AdamConfig(lr=1e-3)
    loss = a.train_step(X, T, cfg)
    m, Bp = b._load_inputs(X)
    b.T[:n] = torch.as_tensor(T, device="cuda")
    b._forward(Bp)
    b.backward(m, Bp)
    b.adam_step(cfg)
    torch.cuda.synchronize()
    a.k.check_err()
    b.k.check_err()
    assert torch.equal(a.Y[:n], b.Y[:n])
    assert torch.allclose(loss, b.sq[:n].mean() / S.N_OUT, rtol=1e-6)
    dz = [b.dZ[l][:Bp].double().abs() for l in range(4)] + [b.dY16[:Bp].double().abs()]
    h = [b.X32[:Bp].double().abs()] + [b.H[l][:Bp].double().abs() for l in range(4)]
    for l in range(5):
        gw, gb = dz[l].T @ h[l], dz[l].sum(0)
        assert ((a.gW[l] - b.gW[l]).abs() <= 4.9e-5 * gw + 1e-30).all(), l
        assert ((a.gb[l] - b.gb[l]).abs() <= 4.9e-5 * gb + 1e-30).all(), l
        assert (a.W[l] - b.W[l]).abs().max() <= 2 * cfg.lr
        same = (a.gW[l] == b.gW[l])
        assert torch.equal(a.W[l][same], b.W[l][same])
        assert torch.equal(a.W16[l], a.W[l].to(torch.bfloat16)) and torch.equal(a.W16T[l], a.W16[l].t())
    # Twice on the same state: the same bits.
    c = S.SurrogateMLP(seed=3, max_batch=n)
    c.train_step(X, T, cfg)
    assert all(torch.equal(u, v) for u, v in zip(a.W + a.b + a.gW + a.gb, c.W + c.b + c.gW + c.gb))
