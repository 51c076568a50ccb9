"""One training step of the tensor-core network: gradients, Adam and images.

Two steps against an FP32 Adam on the host, fed with the gradients that the
library returns for the same parameters, at one sample, the edges of a tile, the
batch in use, and more than one tile per SM.  The step lr * mhat / (sqrt(vhat) + eps) takes
about ten FP32 roundings (10 * 2^-24 = 6e-7 relative; 2e-6 allowed), the
parameter one (2^-23 of it allowed).  The second step starts from the first's
moments, and the network's outputs after it match the oracle for the parameters
read back, so the BF16 images follow the master weights (the forward test's
bounds).
"""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 8192, 128 * 148 + 1, 128 * 311 + 64])
def test_step_is_adam_on_the_gradients(cuda, n):
    from q_psdm_b200 import surrogate as S
    rng = np.random.default_rng(n)
    x = rng.uniform(-1.0, 1.0, (n, 5)).astype(np.float32)
    t = np.stack([np.sin(x[:, 0]) + x[:, 1], x[:, 2] * x[:, 3] - x[:, 4]], 1).astype(np.float32)
    net = S.Mlp(0, params=M.init_params(3, out_scale=1.0).astype(np.float32))
    net.set_scaling(np.zeros(5, np.float32), np.ones(5, np.float32), (1.0, 0.5))
    f = np.float32
    lr, b1, b2, eps = f(1e-3), f(0.9), f(0.999), f(1e-8)
    p = net.params()
    m, v = np.zeros_like(p), np.zeros_like(p)
    for step in (1, 2):
        loss, g = net.gradients(x, t)
        assert net.train_step(x, t, float(lr), want_loss=True) == loss
        m = b1 * m + (f(1) - b1) * g
        v = b2 * v + (f(1) - b2) * g * g
        c1, c2 = f(1) / (f(1) - b1 ** f(step)), f(1) / (f(1) - b2 ** f(step))
        d = lr * (m * c1) / (np.sqrt(v * c2) + eps)
        q = net.params()
        assert np.all(np.abs(q - (p - d)) <= 2e-6 * lr + 2.0 ** -23 * np.abs(p))
        assert np.any(q != p)
        p = q
    y = net.forward(x).cpu().numpy()
    net.status()
    yb, _, _ = M.forward(p.astype(np.float64), x, np.zeros(5), np.ones(5), bf16_ops=True)
    scale = np.sqrt(np.mean(yb ** 2))
    assert np.abs(y - yb).max() < 2e-2 * scale
    if n > 1:
        assert np.sqrt(np.mean((y - yb) ** 2)) < 2e-3 * scale
