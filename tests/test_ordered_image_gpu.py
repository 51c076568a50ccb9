"""The plain and compat kernels add every point's traces in submission order
whatever the image size, the number of warps that share a point, the tile's
shape or the dip limits: bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from q_psdm_b200 import engine as E
from q_psdm_b200 import synth, tables
from tests.cuda_util import d2h

pytestmark = pytest.mark.gpu
X0, Y0 = 500000.0, 4000000.0


def _headers(nxi, ntr, seed):
    rng = np.random.default_rng(seed)
    h = np.empty((ntr, 4))
    s = np.repeat(rng.uniform(0.2, 0.8, (ntr + 6) // 7) * nxi * 10.0, 7)[:ntr]  # runs of a source
    h[:, 0], h[:, 1] = s, 40.0
    h[:, 2] = s + rng.uniform(-900, 900, ntr)
    h[:, 3] = rng.uniform(-300, 300, ntr)
    h += np.array([X0, Y0] * 2)
    h[0] = (X0 + 50, Y0, X0 + 50, Y0)  # zero offset above a node
    return np.rint(h * 100).astype(np.int32)


def _dips(kind, nxi, nzi):
    rng = np.random.default_rng(3)
    if kind == "reference":
        return np.stack(synth.dip_fields(nxi, nzi, float(np.radians(3.0))))
    lo = {"varied": 0.35, "crossed": -0.02}[kind]  # crossed: lower limit above the upper
    v = rng.uniform(min(lo, 0.05), max(lo, 0.05), (4, nxi, nzi)).astype(np.float32)
    v[0::2] *= -1
    return v


def _engine(nxi, nzi, nt, taper, **kw):
    p = E.static_params(nxi=nxi, nzi=nzi, ntl=nt, dt=0.002, dxi=10.0, dyi=10.0, dzi=10.0,
                        scaled=0.01, fxv=X0, fyv=Y0 - 4000.0, nxv=nxi, nyv=1000, taperzone=taper,
                        max_batch=600, **kw)
    return p, E.Engine(p)


@pytest.mark.parametrize("nxi,nzi,ntr", [(128, 100, 600), (33, 11, 300), (300, 257, 500),
                                         (512, 397, 300), (720, 500, 200), (1024, 600, 120)])
@pytest.mark.parametrize("dips,taper", [("reference", 8.0), ("varied", 8.0), ("varied", 0.0),
                                        ("crossed", 2.0)])
def test_compat_equals_oracle(cuda, nxi, nzi, ntr, dips, taper):
    hdr = _headers(nxi, ntr, nxi)
    p, eng = _engine(nxi, nzi, 1010, taper)
    d = _dips(dips, nxi, nzi)
    try:
        tc = (4, nxi - 3)
        eng.set_line(fxi=X0, cyi=Y0, dips=d, ttt_cdp1=tc[0], ttt_cdp2=tc[1])
        eng.begin_offset(E.offset_params(p, 0, nxi, aznx1=70, aznx2=75, azny1=40, azny2=40))
        eng.submit(E.encode_su(*hdr.T, np.zeros((ntr, 1010), np.float32), dt_us=2000, scalco=-100))
        img = eng.get_image(False)
        npt = eng.counters()[1]
        pi, pg = eng.gate_device_ptrs()
        ints, geom = d2h(pi, (ntr, 8), np.int32), d2h(pg, (ntr, 4), np.float32)
    finally:
        eng.close()
    ok = ints[:, 0] == 3
    assert ok.sum() > ntr // 4
    ip = O.ImageParams(nzi=nzi, nxb=nxi, ixstart=0, nt=p.nffti, dt1=p.dt1, dxi=10.0, dzi=10.0,
                       taperzone=p.taperzone, tcdp1=tc[0] - 1, tcdp2=tc[1] - 1)
    ref, n = O.image_compat(ip, geom[ok], np.ascontiguousarray(ints[ok][:, [4, 5, 7]]),
                            [np.ascontiguousarray(x.ravel()) for x in d])
    assert npt == n
    assert np.array_equal(img, ref.reshape(nxi, nzi))


def test_plain_blocks_bit_equal(cuda):
    """640 x 500 points in one block (one warp per column) against narrower
    blocks of the same line (2, 4 and 8 warps per column), blocks whose tiles
    straddle table cells, and two batches."""
    nxi, nzi, nt, ntr = 640, 500, 600, 400
    sv = synth.config2(0)
    tfn = lambda px, py, x, z: synth.traveltime(sv, np.hypot(px - x, py), z)
    tab = tables.build_line_tables(tfn, lambda *a: tfn(*a) / 80.0, fci=1, nxi=nxi, dxi=10.0,
                                   zmax=(nzi - 1) * 10.0, dzii=80.0, nxi1=16, nzi1=64,
                                   surf_dx=320, surf_dy=320, half_x=1600.0, half_y=640.0)
    hdr = _headers(nxi, ntr, 5)
    rng = np.random.default_rng(8)
    rec = E.encode_su(*hdr.T, rng.standard_normal((ntr, nt)).astype(np.float32), dt_us=2000,
                      scalco=-100)
    d = _dips("varied", nxi, nzi)
    full = {}
    for kahan in (0, 1):
        p, eng = _engine(nxi, nzi, nt, 8.0, mode=1, panel_dtype=0, nbins=4, dtstar=0.002,
                         dzii=80.0, kahan=kahan)
        try:
            eng.set_line(fxi=X0, cyi=Y0, dips=d, tables=tab.as_engine_dict())
            for lo, hi in ((0, nxi), (160, 460), (240, 400), (304, 340), (163, 471), (301, 333)):
                eng.begin_offset(E.offset_params(p, lo, hi, aznx1=90, aznx2=90, azny1=40,
                                                 azny2=40))
                eng.submit(rec[:150])
                eng.submit(rec[150:])
                img = eng.get_image(False)
                if lo == 0:
                    full[kahan] = img
                    assert np.abs(img).max() > 0
                assert np.array_equal(img, full[kahan][lo:hi]), (kahan, lo, hi)
        finally:
            eng.close()
