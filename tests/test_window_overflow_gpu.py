"""Table entries past any time window (1e30, the float maximum, infinities, NaN)
at some nodes: a pair whose traveltime is past the window is not imaged,
whatever it is.  The plain form against its FP32 restatement, bit for bit; the
original batched kernels against the plain form (2e-5 of the image peak, the
bound they are held to), with equal point-trace counts."""
import copy

import numpy as np
import pytest

from oracle import oracle as O
from tests.cuda_util import d2h
from tests.physics_case import engine, gate, make_case, records

pytestmark = pytest.mark.gpu
BAD = {"1e30": 1e30, "max": np.finfo(np.float32).max, "inf": np.inf, "-inf": -np.inf, "nan": np.nan}


def marked_case(bad, table="ttt", **kw):
    """A case with the value `bad` in a table: at one surface node of every
    depth, at one depth node and at scattered entries."""
    c = make_case(**{**dict(nshots=2, rstep=2), **kw})
    tab = c["tab"] = copy.copy(c["tab"])
    a = getattr(tab, table).copy()
    setattr(tab, table, a)
    plane = tab.nxi1 * tab.nzi1
    for k in range(tab.nxg * tab.nzg):
        d = tab.desc[k]
        n = int(d["nys"]) * int(d["nxs"])
        cell = a[d["idx"]:d["idx"] + n * plane].reshape(n, tab.nxi1, tab.nzi1)
        if k % 3 == 0:
            cell[n // 2 + 3] = bad
        if k % 3 == 1:
            cell[:, k % tab.nxi1, tab.nzi1 // 2] = bad
        cell.ravel()[k::2011] = bad
    return c


def image(c, rec, **kw):
    eng, _, _ = engine(c, **{**dict(panel_dtype=0, max_batch=rec.shape[0]), **kw})
    try:
        eng.submit(rec)
        return eng.get_image(False), eng.stats()
    finally:
        eng.close()


@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("table", ["ttt", "qqq"])
def test_plain_bit_exact(cuda, bad, table):
    c = marked_case(BAD[bad], table)
    sv, tab, rec = c["sv"], c["tab"], records(c)
    eng, p, _ = engine(c, panel_dtype=0, form=0, max_batch=rec.shape[0])
    try:
        eng.submit(rec)
        img = np.asarray(eng.get_image(False), np.float32).ravel()
        st = eng.stats()
        pan = d2h(eng.panels_device_ptrs()[0], (rec.shape[0], p.nbins, p.nffti), np.float32)
    finally:
        eng.close()
    ints, geom = gate(c)
    a = O.P32(nzi=sv.nzi, nxb=c["nxb"], ixstart=c["ixstart"], nt=p.nffti, nbins=p.nbins,
              dt1=p.dt1, dxi=p.dxi, dzi=p.dzi, taperzone=p.taperzone, dtstar=p.dtstar,
              dzii=p.dzii, tcdp1=tab.cdp1 - sv.fci, tcdp2=tab.cdp2 - sv.fci, nxg=tab.nxg,
              nzg=tab.nzg, nxi1=tab.nxi1, nzi1=tab.nzi1)
    with np.errstate(invalid="ignore"):
        ref, npt, nimg = O.image_plain_fp32(a, ints, geom, pan, c["dips"], tab.as_engine_dict())
    assert nimg > 0 and np.isfinite(ref).all()
    assert (st["point_traces"], st["imaged"]) == (npt, nimg)
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("variant", [1, 3, 6, 13])
@pytest.mark.parametrize("bad", list(BAD))
def test_original_kernels_equal_plain(cuda, bad, variant):
    c = marked_case(BAD[bad])
    rec = records(c)
    plain, s0 = image(c, rec, form=0)
    img, s1 = image(c, rec, form=1, variant=variant)
    assert s1["point_traces"] == s0["point_traces"]
    assert np.isfinite(img).all()
    assert np.abs(img - plain).max() <= 2e-5 * np.abs(plain).max()
