"""t* through zones without attenuation (1/Q = 0: water, an elastic overburden):
the blocks below them are reached although t* does not change in them.
Against the float64 relaxation of test_eikonal_blocks_gpu, with its bounds.
Grids and sources lie on model nodes, where the model is sampled exactly."""
import ctypes as C

import numpy as np
import pytest

from q_psdm_b200 import _lib
from tests.test_eikonal_blocks_gpu import _reference

pytestmark = pytest.mark.gpu
H = 20.0


def _block(x, y, z):
    return ((x >= 20 * H) & (x <= 32 * H) & (y >= 8 * H) & (y <= 22 * H) &
            (z >= 12 * H) & (z <= 26 * H))


MODELS = {
    "above": lambda x, y, z: np.where(z <= 9 * H, 0.0, 0.02),
    "deep": lambda x, y, z: np.where(_block(x, y, z), 0.03, 0.0),
    "middle": lambda x, y, z: np.where((z > 5 * H) & (z <= 14 * H), 0.0, 0.01),
    "none": lambda x, y, z: 0.0 * (x + y + z),
}


@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("nx,ny,nz", [(40, 25, 31), (33, 1, 30), (17, 24, 41)])
def test_tstar_below_zero_attenuation(cuda, name, nx, ny, nz):
    import torch
    v0, kz, r0, ns = 1800.0, 0.5, 3.0, 2
    vel = lambda x, y, z: v0 + kz * z + 0.05 * x + 0.02 * y
    invq = MODELS[name]
    mx, my, mz = nx + 6, ny + 6, nz
    Z, Y, X = np.meshgrid(np.arange(mz) * H, np.arange(my) * H, np.arange(mx) * H, indexing="ij")
    dv = torch.from_numpy(vel(X, Y, Z).astype(np.float32)).cuda()
    dq = torch.from_numpy(invq(X, Y, Z).astype(np.float32)).cuda()
    src = np.array([[0, 0, 0, 0], [nx // 2 + 4, ny // 2 + 3, 4, 3]], np.float32) * H
    n = nx * ny * nz * ns
    dsrc = torch.from_numpy(src).cuda()
    work = torch.empty(4 * n + 4, dtype=torch.float32, device="cuda")
    T = torch.empty(n, dtype=torch.float32, device="cuda")
    S = torch.empty_like(T)
    model = _lib.EikModel(mx, my, mz, H, 0.0, 0.0, v0, kz)
    grid = _lib.EikGrid(nx, ny, nz, H)
    rc = _lib.lib().qpsdm_eikonal_solve(dv.data_ptr(), dq.data_ptr(), C.byref(model),
                                        dsrc.data_ptr(), ns, C.byref(grid), r0 * H, 2000,
                                        work.data_ptr(), T.data_ptr(), S.data_ptr(), None)
    assert rc == 0
    torch.cuda.synchronize()
    T, S = (a.cpu().numpy().reshape(ns, nz, ny, nx).astype(np.float64) for a in (T, S))
    for s in range(ns):
        rt, rs = _reference(vel, invq, H, src[s, :2].astype(float), src[s, 2:].astype(float),
                            (nz, ny, nx), r0 * H, v0, kz)
        assert np.abs(T[s] - rt).max() <= 1e-4, s
        assert np.abs(S[s] - rs).max() <= 0.02 * rs.max(), s
