"""The fast batched form computes a pair of depths, and two members, together:
what it computes for a point or a member that takes no part must not reach the
image.  Every fast variant against the plain form, FP32 panels: 2e-5 of the
image peak (the bound the batched form is held to point by point), equal
point-trace counts, every value finite."""
import numpy as np
import pytest

from q_psdm_b200 import tables
from tests.physics_case import make_case, records
from tests.test_window_overflow_gpu import BAD, image, marked_case

pytestmark = pytest.mark.gpu
FAST = list(range(14, 28))


def _check(c, rec, variant, kahan):
    plain, s0 = image(c, rec, form=0, kahan=kahan)
    img, s1 = image(c, rec, form=1, kahan=kahan, variant=variant)
    amp = np.abs(plain).max()
    assert np.isfinite(plain).all() and amp > 0
    assert s1["point_traces"] == s0["point_traces"]
    assert np.isfinite(img).all()
    assert np.abs(img - plain).max() <= 2e-5 * amp


@pytest.mark.parametrize("variant,kahan", [(v, v & 1) for v in FAST] + [(16, 1), (18, 1)])
@pytest.mark.parametrize("shots", [(5, 6), (6, 5)])
def test_first_source_off_the_tables(cuda, shots, variant, kahan):
    """Two shots 260 m apart on tables that reach 320 m, and of the second one
    the few traces that image tiles where the tables do not cover the first:
    every member list there ends in a member of the second shot alone."""
    c = make_case(shots=shots, rstep=2)
    sv = c["sv"]
    c["tab"] = tables.linear_gradient_tables(sv, fci=sv.fci, nxi=sv.nxi, dxi=sv.dxi,
                                             zmax=(sv.nzi - 1) * sv.dzi, sub=4, nxi1=16,
                                             half_x=320.0, half_y=500.0)
    h = c["hdr"] * sv.scaled
    x, y = h[:, 2] - sv.fxv, h[:, 3] - sv.fyv
    far = (x <= 405) if shots[0] == 6 else (x >= 865)
    second = np.arange(len(h)) >= len(h) // 2
    near_y = np.abs(0.5 * (h[:, 1] + h[:, 3]) - c["cyi"]) <= 25
    pick = ~second | (second & far & near_y)
    assert 0 < (pick & second).sum() < 16
    _check(c, records(c)[pick], variant, kahan)


@pytest.mark.parametrize("bad,variant,kahan", [("inf", v, 0) for v in FAST] +
                         [(b, v, k) for b in BAD for v, k in ((15, 0), (20, 1), (27, 1))])
def test_nodes_past_the_window(cuda, bad, variant, kahan):
    c = marked_case(BAD[bad])
    _check(c, records(c), variant, kahan)


@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("table,ntr", [("qqq", 512), ("ttt", 60)])
def test_nodes_past_the_bins_and_unsplit(cuda, bad, table, ntr):
    c = marked_case(BAD[bad], table)
    rec = records(c)
    _check(c, rec[np.linspace(0, rec.shape[0] - 1, ntr).astype(int)], 26, 0)
