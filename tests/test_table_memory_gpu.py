"""Line tables in little device memory: where the (t, t*) quads do not fit, the
float tables alone, which always were enough, serve the line."""
import copy

import numpy as np
import pytest

from tests.physics_case import engine, make_case, records

pytestmark = pytest.mark.gpu
N = 24 << 20  # entries: 192 MB as two float tables, 384 MB as quads


def _case():
    c = make_case(nshots=2, rstep=2)
    tab = c["tab"] = copy.copy(c["tab"])
    pad = np.zeros(N - tab.ttt.size, np.float32)
    tab.ttt, tab.qqq = np.concatenate([tab.ttt, pad]), np.concatenate([tab.qqq, pad])
    return c


def _image(c, rec, left=None, **kw):
    """The image; left: device bytes that set_line finds free."""
    import torch
    small = dict(c, tab=make_case(nshots=1, rstep=8)["tab"])
    eng, _, o = engine(small, panel_dtype=0, max_batch=rec.shape[0], **kw)
    try:
        torch.cuda.empty_cache()
        hold = None if left is None else torch.empty(torch.cuda.mem_get_info()[0] - left,
                                                     dtype=torch.uint8, device="cuda")
        sv = c["sv"]
        before = torch.cuda.mem_get_info()[0]
        eng.set_line(fxi=c["fxi"], cyi=c["cyi"], dips=c["dips"].reshape(4, sv.nxi, sv.nzi),
                     tables=c["tab"].as_engine_dict())
        used = before - torch.cuda.mem_get_info()[0]
        del hold
        torch.cuda.empty_cache()
        eng.begin_offset(o)
        eng.submit(rec)
        return eng.get_image(False), eng.stats(), used
    finally:
        eng.close()


def test_quads_do_not_fit(cuda):
    c = _case()
    rec = records(c)
    a, sa, _ = _image(c, rec, form=0)
    b, sb, used = _image(c, rec, 330 << 20, form=0)
    assert used <= 8 * N + (40 << 20)
    assert np.abs(a).max() > 0 and sa == sb and np.array_equal(a, b)
    for variant in (26, 3):
        b, sb, _ = _image(c, rec, 330 << 20, form=1, variant=variant)
        assert sb["point_traces"] == sa["point_traces"]
        assert np.abs(b - a).max() <= 2e-5 * np.abs(a).max()
