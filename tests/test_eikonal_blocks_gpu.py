"""The relaxation in active blocks: grids that are no multiple of a block,
thinner than one, sources anywhere, against a float64 relaxation of the same
scheme over the whole grid (numpy Jacobi).

Tolerances: traveltime 1e-4 s of up to 1 s, the FP32 update's rounding (the
three-sided solution cancels s^2 - 3 (...): some 3e-6 s per node, and a node
only moves down) over the grid's some 50 nodes a side; t*, smooth in the
weights, 2 % of its largest value."""
import ctypes as C

import numpy as np
import pytest

from q_psdm_b200 import _lib

pytestmark = pytest.mark.gpu
INF = 1e30


def _reference(vel, invq, h, src, origin, shape, r0, v0, kz):
    nz, ny, nx = shape
    z, y, x = np.meshgrid(np.arange(nz) * h, origin[1] + np.arange(ny) * h,
                          origin[0] + np.arange(nx) * h, indexing="ij")

    def at(m, x, y, z):  # the model is linear in every axis: trilinear is exact
        return m(x, y, z)
    r2 = (x - src[0]) ** 2 + (y - src[1]) ** 2
    start = r2 + z * z <= r0 * r0
    # the held start values are the scheme's input: the analytic time with its
    # argument in FP32, as the solver has it (1 + a small number near the source)
    f4 = lambda a: np.asarray(a, np.float32)
    r = np.sqrt(f4(r2))
    arg = f4(1.0) + f4(kz * kz) * (r * r + f4(z) * f4(z)) / (f4(2.0 * v0) * f4(v0 + kz * z))
    bg = np.arccosh(np.maximum(arg.astype(np.float64), 1.0)) / kz
    T = np.where(start, bg, INF)
    f = h / at(vel, x, y, z)

    def near(A, ax, fill):
        lo, hi = np.full_like(A, fill), np.full_like(A, fill)
        sl = [slice(None)] * 3
        a, b = list(sl), list(sl)
        a[ax], b[ax] = slice(1, None), slice(None, -1)
        lo[tuple(a)] = A[tuple(b)]
        hi[tuple(b)] = A[tuple(a)]
        return lo, hi
    for _ in range(8 * sum(shape)):
        m = np.sort(np.stack([np.minimum(*near(T, a, INF)) for a in range(3)]), 0)
        t = m[0] + f
        s2 = m[0] + m[1]
        t = np.where((t > m[1]) & (m[1] < INF),
                     0.5 * (s2 + np.sqrt(np.maximum(2 * f * f - (m[0] - m[1]) ** 2, 0))), t)
        s3 = s2 + m[2]
        d3 = s3 * s3 - 3.0 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2 - f * f)
        t = np.where((m[0] + f > m[1]) & (t > m[2]) & (m[2] < INF),
                     (s3 + np.sqrt(np.maximum(d3, 0))) / 3.0, t)
        new = np.where(start | (m[0] >= INF), T, np.minimum(T, t))
        if not (new < T - 1e-13).any():
            break
        T = new
    num, den, S = [], 0.0, np.where(start, T * at(invq, src[0], src[1], 0.0), 0.0)
    for a in range(3):
        lo, hi = near(T, a, INF)
        w = np.maximum(T - np.minimum(lo, hi), 0.0) * (np.minimum(lo, hi) < T) / (h * h)
        num.append((a, lo <= hi, w))
        den = den + w
    qf = at(invq, x, y, z) / at(vel, x, y, z) ** 2
    free = ~start & (den > 0)
    for _ in range(8 * sum(shape)):
        n = qf.copy()
        for a, low, w in num:
            lo, hi = near(S, a, 0.0)
            n += w * np.where(low, lo, hi)
        new = np.where(free, n / np.where(den > 0, den, 1.0), S)
        if np.array_equal(new, S):
            break
        S = new
    return T, S


@pytest.mark.parametrize("nx,ny,nz,r0", [(16, 8, 4, 3.0), (17, 9, 5, 3.0), (2, 1, 2, 1.0),
                                         (33, 1, 30, 3.0), (40, 25, 21, 3.0), (31, 24, 40, 12.0),
                                         (64, 16, 8, 2.0)])
def test_solve_matches_float64(cuda, nx, ny, nz, r0):
    import torch
    h, v0, kz, ns = 20.0, 1800.0, 0.5, 3
    vel = lambda x, y, z: v0 + kz * z + 0.05 * x + 0.02 * y
    invq = lambda x, y, z: 0.01 + 1e-6 * x + 2e-6 * z
    mx, my, mz = nx + 10, ny + 10, nz
    Z, Y, X = np.meshgrid(np.arange(mz) * h, np.arange(my) * h, np.arange(mx) * h, indexing="ij")
    dv = torch.from_numpy(vel(X, Y, Z).astype(np.float32)).cuda()
    dq = torch.from_numpy(invq(X, Y, Z).astype(np.float32)).cuda()
    rng = np.random.default_rng(nx)
    src = np.zeros((ns, 4), np.float32)
    src[:, 2:] = np.rint(rng.uniform(0, 9 * h, (ns, 2)))
    src[0, :2] = src[0, 2:]  # a source at its grid's corner
    src[1:, 0] = src[1:, 2] + np.rint(rng.uniform(0, (nx - 1) * h, ns - 1))
    src[1:, 1] = src[1:, 3] + np.rint(rng.uniform(0, (ny - 1) * h, ns - 1))
    n = nx * ny * nz * ns
    dsrc = torch.from_numpy(src).cuda()
    work = torch.empty(4 * n + 4, dtype=torch.float32, device="cuda")
    T = torch.empty(n, dtype=torch.float32, device="cuda")
    S = torch.empty_like(T)
    model = _lib.EikModel(mx, my, mz, h, 0.0, 0.0, v0, kz)
    grid = _lib.EikGrid(nx, ny, nz, h)
    rc = _lib.lib().qpsdm_eikonal_solve(dv.data_ptr(), dq.data_ptr(), C.byref(model),
                                        dsrc.data_ptr(), ns, C.byref(grid), r0 * h, 2000,
                                        work.data_ptr(), T.data_ptr(), S.data_ptr(), None)
    assert rc == 0
    torch.cuda.synchronize()
    T, S = (a.cpu().numpy().reshape(ns, nz, ny, nx).astype(np.float64) for a in (T, S))
    for s in range(ns):
        rt, rs = _reference(vel, invq, h, src[s, :2].astype(float), src[s, 2:].astype(float),
                            (nz, ny, nx), r0 * h, v0, kz)
        assert np.abs(T[s] - rt).max() <= 1e-4, s
        assert np.abs(S[s] - rs).max() <= 0.02 * rs.max(), s
