"""Real transforms two signals at a time: odd batches, lengths with repeated
factors (Stockham passes), every small factor, rows aligned to 4 bytes only.

Tolerance: that of the batched transforms' own test, 3e-7 log2(n) of the
largest bin (some eps per pass of a float transform)."""
import numpy as np
import pytest

from q_psdm_b200 import _lib

pytestmark = pytest.mark.gpu


def _tol(n):
    return 3e-7 * max(1.0, np.log2(n))


# 2 x: one factor each, coprime products (16, 9 among them), repeated factors
LENGTHS = [4, 6, 8, 10, 14, 18, 22, 26, 32, 64, 98, 128, 162, 242, 250, 288, 338, 1024, 1440,
           4752, 5040, 12012, 12798 // 2 * 2 - 6]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("batch,shift", [(1, 0), (5, 0), (4, 1)])
def test_r2c_c2r(cuda, n, batch, shift):
    import torch
    L = _lib.lib()
    if L.qpsdm_fft_r2c(8, n, 0, 8, None) != 0:
        pytest.fail("batch 0 is refused")
    rng = np.random.default_rng(n + batch)
    x = rng.standard_normal((batch, n)).astype(np.float32)
    buf = torch.zeros(batch * n + 1, dtype=torch.float32, device="cuda")
    dx = buf[shift:shift + batch * n]
    dx.copy_(torch.from_numpy(x).reshape(-1))
    y = torch.empty((batch, n // 2 + 1, 2), dtype=torch.float32, device="cuda")
    rc = L.qpsdm_fft_r2c(dx.data_ptr(), n, batch, y.data_ptr(), None)
    ref = np.fft.rfft(x.astype(np.float64), axis=1)
    if rc == 1:  # a factor outside {2, 3, 5, 7, 11, 13}
        m = n // 2
        for q in (2, 3, 5, 7, 11, 13):
            while m % q == 0:
                m //= q
        assert m != 1
        return
    assert rc == 0
    torch.cuda.synchronize()
    got = y.cpu().numpy().astype(np.float64)
    assert np.abs(got[..., 0] + 1j * got[..., 1] - ref).max() <= _tol(n) * np.abs(ref).max()
    out = torch.zeros(batch * n + 1, dtype=torch.float32, device="cuda")
    z = out[shift:shift + batch * n]
    assert L.qpsdm_fft_c2r(y.data_ptr(), n, batch, z.data_ptr(), None) == 0
    torch.cuda.synchronize()
    back = z.cpu().numpy().reshape(batch, n) / n
    assert np.abs(back - x).max() <= 4 * _tol(n) * np.abs(x).max()
    assert float(out[0 if shift else -1]) == 0.0
