"""Which transform lengths are taken: 2 m with m up to 6399 and no factor outside
{2, 3, 5, 7, 11, 13}.  The rest are refused before anything is planned or
allocated, also lengths with more factors than a plan has passes for."""
import numpy as np
import pytest

from q_psdm_b200 import _lib

EINVAL = 1


def _smooth(m):
    for q in (2, 3, 5, 7, 11, 13):
        while m % q == 0:
            m //= q
    return m == 1


def test_refused_lengths():
    """The pointers are never read: every one of these calls is refused."""
    L = _lib.lib()
    big = [2 * m for m in (6400, 6435, 6480, 2 ** 26, 3 * 2 ** 25, 3 ** 18, 15 * 2 ** 26, 2 ** 29)]
    rough = [2 * m for m in range(1, 6400, 7) if not _smooth(m)] + [12792, 2 * 6397]
    for n in big + rough + [3, 9, 2 ** 31 - 1]:
        assert L.qpsdm_fft_r2c(64, n, 1, 64, None) == EINVAL, n
        assert L.qpsdm_fft_c2r(64, n, 1, 64, None) == EINVAL, n


@pytest.mark.gpu
@pytest.mark.parametrize("m", [6370, 6336, 6300, 6250, 6272, 6237, 6160, 6006, 5632, 5005, 4095])
@pytest.mark.parametrize("batch", [1, 4])
def test_longest_lengths(cuda, m, batch):
    """Against float64, to the bound of the shorter lengths' test (3e-7 log2(n) of
    the largest bin): two-buffer lengths, even and odd, and prime-factor ones."""
    import torch
    L, n = _lib.lib(), 2 * m
    tol = 3e-7 * np.log2(n)
    x = np.random.default_rng(m).standard_normal((batch, n)).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    y = torch.empty((batch, m + 1, 2), dtype=torch.float32, device="cuda")
    assert L.qpsdm_fft_r2c(dx.data_ptr(), n, batch, y.data_ptr(), None) == 0
    torch.cuda.synchronize()
    got = y.cpu().numpy().astype(np.float64)
    ref = np.fft.rfft(x.astype(np.float64), axis=1)
    assert np.abs(got[..., 0] + 1j * got[..., 1] - ref).max() <= tol * np.abs(ref).max()
    z = torch.empty_like(dx)
    assert L.qpsdm_fft_c2r(y.data_ptr(), n, batch, z.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert np.abs(z.cpu().numpy() / n - x).max() <= 4 * tol * np.abs(x).max()
