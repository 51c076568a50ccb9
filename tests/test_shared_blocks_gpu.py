"""Table cells whose blocks share data image, bit for bit, what the same cells
with blocks of their own do: the same values by the same kernel."""
import copy

import numpy as np
import pytest

from q_psdm_b200 import synth, tables
from tests.physics_case import make_case, records
from tests.test_window_overflow_gpu import image

pytestmark = pytest.mark.gpu


def _own_blocks(tab):
    """The tables with every cell's block copied out, one after the other."""
    own = copy.copy(tab)
    own.desc = tab.desc.copy()
    n = [int(d["nys"]) * int(d["nxs"]) * tab.nxi1 * tab.nzi1 for d in tab.desc]
    cut = [slice(int(d["idx"]), int(d["idx"]) + k) for d, k in zip(tab.desc, n)]
    own.desc["idx"] = np.cumsum([0] + n[:-1])
    own.ttt = np.concatenate([tab.ttt[c] for c in cut])
    own.qqq = np.concatenate([tab.qqq[c] for c in cut])
    return own


def _equal(c, tab, **kw):
    rec = records(c)
    a, sa = image(dict(c, tab=tab), rec, **kw)
    b, sb = image(dict(c, tab=_own_blocks(tab)), rec, **kw)
    assert np.abs(b).max() > 0
    assert sa == sb
    assert np.array_equal(a, b)


@pytest.mark.parametrize("nzi1", [2, 7])
@pytest.mark.parametrize("kw", [dict(form=0), dict(form=1, variant=26), dict(form=1, variant=3)])
def test_columns_share_their_blocks(cuda, kw, nzi1):
    """v(z) tables of several depth cells, kept once for all x cells."""
    c = make_case(nshots=2, rstep=2)
    sv = c["sv"]
    tfn = lambda px, py, x, z: synth.traveltime(sv, np.hypot(px - x, py), z)
    tab = tables.build_line_tables(tfn, lambda *a: tfn(*a) / sv.q, fci=sv.fci, nxi=sv.nxi,
                                   dxi=sv.dxi, zmax=(sv.nzi - 1) * sv.dzi, dzii=80.0, nxi1=16,
                                   nzi1=nzi1, surf_dx=40, surf_dy=40, half_x=1000.0, half_y=500.0)
    assert tab.nzg > 1
    tab.desc["idx"] = np.tile(tab.desc["idx"][:tab.nzg], tab.nxg)
    _equal(c, tab, **kw)


@pytest.mark.parametrize("step", [16 * 26, 26, 37])  # whole planes, a cdp, neither
def test_blocks_that_overlap_plain(cuda, step):
    c = make_case(nshots=2, rstep=2)
    tab = copy.copy(c["tab"])
    assert (tab.nzg, tab.nxi1, tab.nzi1) == (1, 16, 26)
    tab.desc = tab.desc.copy()
    tab.desc["idx"] = step * np.arange(tab.nxg)
    _equal(c, tab, form=0)
