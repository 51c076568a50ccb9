"""Table cells past the 65,535 of a launch grid's second dimension: the image of
the last columns of a line of 66,100 one-cdp cells equals, bit for bit, the
image from a table of those columns alone (same sums, same cell centres)."""
import numpy as np
import pytest

from q_psdm_b200 import engine as E
from q_psdm_b200 import synth, tables

pytestmark = pytest.mark.gpu
NXI, NZI, NT, LO, HI = 66100, 40, 400, 65900, 66060


@pytest.mark.parametrize("paired", [True, False])
@pytest.mark.parametrize("form,variant", [(0, 0), (1, 26), (1, 13)])
def test_cells_past_a_grid(cuda, form, variant, paired):
    sv = synth.config1(0)
    tfn = lambda px, py, x, z: synth.traveltime(sv, np.hypot(px - x, py), z)
    # v(z): one block, relative to its cell's centre, serves every cell
    one = tables.build_line_tables(tfn, lambda *a: tfn(*a) / 60.0, fci=1, nxi=1, dxi=10.0,
                                   zmax=(NZI - 1) * 10.0, dzii=40.0, nxi1=1, nzi1=16, surf_dx=40,
                                   surf_dy=40, half_x=800.0, half_y=400.0)
    rng = np.random.default_rng(1)
    ntr = 200
    mid = rng.uniform(LO + 20, HI - 20, ntr) * 10.0
    off = rng.uniform(-150, 150, ntr)
    hdr = np.rint(100 * np.stack([mid - off, np.full(ntr, 30.0), mid + off,
                                  rng.uniform(-60, 60, ntr)], 1)).astype(np.int64)
    rec = E.encode_su(*hdr.T, rng.standard_normal((ntr, NT)).astype(np.float32), dt_us=2000,
                      scalco=-100)
    p = E.static_params(nxi=NXI, nzi=NZI, ntl=NT, dt=0.002, dxi=10.0, dyi=10.0, dzi=10.0,
                        scaled=0.01, fxv=0.0, fyv=-2000.0, nxv=NXI, nyv=400, max_batch=ntr,
                        mode=1, panel_dtype=0, nbins=4, dtstar=0.002, dzii=40.0, form=form,
                        variant=variant)
    dips = np.empty((4, NXI, NZI), np.float32)
    dips[0::2], dips[1::2] = -0.3, 0.3
    eng, out = E.Engine(p), []
    try:
        for cdp1, n in ((1, NXI), (LO - 99, NXI - LO + 100)):
            d = np.repeat(one.desc[:1], n)
            dq = d.copy()
            qqq = one.qqq
            if not paired:
                dq["idx"] += 16
                qqq = np.concatenate([np.zeros(16, np.float32), qqq])
            raw = lambda a: a.view(np.uint8).reshape(-1, 16).copy()
            eng.set_line(fxi=0.0, cyi=0.0, dips=dips, tables=dict(
                nxg=n, nzg=1, nxi1=1, nzi1=one.nzi1, cdp1=cdp1, cdp2=NXI, ttt_desc=raw(d),
                qqq_desc=raw(dq), ttt=one.ttt, qqq=qqq))
            eng.begin_offset(E.offset_params(p, LO, HI, aznx1=30, aznx2=30, azny1=30, azny2=30))
            eng.submit(rec)
            out.append((eng.get_image(False), eng.stats()))
    finally:
        eng.close()
    (a, sa), (b, sb) = out
    assert np.abs(b).max() > 0 and sb["point_traces"] > 0
    assert sa == sb
    assert np.array_equal(a, b)
