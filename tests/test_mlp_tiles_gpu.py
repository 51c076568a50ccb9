"""Network inference at the edges of its tiles: 64 samples to a tile, a tile to
an SM before a second team of a CTA has one, six teams, then further rounds.

A sample's outputs do not depend on where it lies: any number of samples, from
any first one, gives the bits that one call over all of them gives (whose values
the forward test holds against the oracle), and nothing past the last is
written."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu

TOTAL = 64 * 148 * 6 + 200


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, 64 * 148, 64 * 148 + 1, 64 * 148 * 6 + 65])
@pytest.mark.parametrize("first", [0, 37, 64])
def test_outputs_do_not_depend_on_the_tile(cuda, n, first):
    import torch
    from q_psdm_b200 import surrogate as S
    rng = np.random.default_rng(1)
    x = torch.from_numpy(rng.uniform(-1.0, 1.0, (TOTAL, 5)).astype(np.float32)).cuda()
    net = S.Mlp(0, params=M.init_params(4, out_scale=1.0).astype(np.float32))
    net.set_scaling(np.zeros(5, np.float32), np.ones(5, np.float32), (1.0, 1.0))
    every = net.forward(x)
    part = torch.full((n + 64, 2), 7.0, device="cuda")
    net.forward(x[first:first + n].contiguous(), out=part)
    net.status()
    assert torch.equal(part[:n], every[first:first + n])
    assert bool((part[n:] == 7.0).all())
