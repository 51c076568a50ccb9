"""The fast batched form holds two depths per thread and may split a tile's
members into parts: the edges of both, against the plain form with FP32 panels.

Tolerance: 2e-5 of the image peak (the bound the batched form is held to
point by point: FP32 rounding of some 1e3 sums in another order, and of the
approximate reciprocals, 1e-7 each); point-trace counts are equal."""
import numpy as np
import pytest

from tests.physics_case import DTSTAR, engine, make_case, records
from q_psdm_b200 import synth, tables

pytestmark = pytest.mark.gpu


def _case(nzi, ixend, dzii, nzi1):
    """Config 1's two gathers into a line of ixend x nzi points; nzi1: depth
    nodes of a table cell (0: one cell over all depths)."""
    c = make_case(nshots=2, rstep=2, ixend=ixend)
    sv = c["sv"]
    sv.nzi = nzi
    c["dips"] = np.stack([d.ravel() for d in synth.dip_fields(
        sv.nxi, nzi, float(c["static"]["contract"]))])
    zmax = (nzi - 1) * sv.dzi
    c["tab"] = tables.build_line_tables(
        lambda px, py, x, z: synth.traveltime(sv, np.hypot(px - x, py), z),
        lambda px, py, x, z: synth.traveltime(sv, np.hypot(px - x, py), z) / sv.q,
        fci=sv.fci, nxi=sv.nxi, dxi=sv.dxi, zmax=zmax, dzii=dzii, nxi1=16,
        nzi1=nzi1 or int(zmax // dzii) + 2, surf_dx=40, surf_dy=40, half_x=1000.0, half_y=500.0)
    return c


def _image(c, rec, **kw):
    eng, _, _ = engine(c, panel_dtype=0, dtstar=DTSTAR, **kw)
    try:
        eng.submit(rec)
        return eng.get_image(False), eng.stats()
    finally:
        eng.close()


@pytest.mark.parametrize("nzi,ixend,dzii,nzi1,ntr", [
    (100, 128, 40.0, 0, 512),   # pairs inside one depth interval, tiles in parts
    (97, 125, 40.0, 0, 512),    # a last pair with one point, ragged columns
    (100, 128, 30.0, 0, 512),   # pairs that straddle depth nodes
    (100, 128, 40.0, 0, 60),    # too few members to split
    (96, 128, 160.0, 2, 512),   # the lower node in the cell below
    (99, 128, 40.0, 8, 512),    # tiles that straddle depth cells
])
@pytest.mark.parametrize("variant,kahan", [(26, 0), (27, 1), (20, 0), (15, 0)])
def test_depth_pairs_equal_plain(cuda, nzi, ixend, dzii, nzi1, ntr, variant, kahan):
    c = _case(nzi, ixend, dzii, nzi1)
    rec = records(c)
    rec = rec[np.linspace(0, rec.shape[0] - 1, ntr).astype(int)]
    plain, s0 = _image(c, rec, form=0, kahan=kahan)
    img, s1 = _image(c, rec, form=1, kahan=kahan, variant=variant)
    amp = np.abs(plain).max()
    assert amp > 0
    assert s1["point_traces"] == s0["point_traces"]
    assert np.abs(img - plain).max() <= 2e-5 * amp


@pytest.mark.parametrize("share", [False, True])
def test_cells_that_share_a_block(cuda, share):
    """Cells with several depths whose descriptors point at one block: the
    node under a cell's last one depends on the cell, not on the block."""
    c = _case(96, 128, 160.0, 2)
    tab = c["tab"]
    if share:  # every x cell reads the first x cell's data; its last depth cell the first's
        for k in range(tab.nxg * tab.nzg):
            tab.desc["idx"][k] = tab.desc["idx"][0 if k % tab.nzg == tab.nzg - 1 else k % tab.nzg]
    rec = records(c)
    plain, s0 = _image(c, rec, form=0)
    img, s1 = _image(c, rec, form=1, variant=26)
    assert s1["point_traces"] == s0["point_traces"]
    assert np.abs(img - plain).max() <= 2e-5 * np.abs(plain).max()
