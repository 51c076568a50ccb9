"""The tuner's results are shared by the engines of a process whose image kernels
do the same: an engine with float tables, or whose batches are split otherwise,
times for itself, a second of its kind takes the result over."""
import numpy as np
import pytest

from tests.physics_case import engine, make_case, records

pytestmark = pytest.mark.gpu


def _tuned(c, rec, paired=True):
    """(variant, whether this engine timed the variants itself)."""
    eng, p, o = engine(c, panel_dtype=0, nbins=6, form=1, max_batch=1024)
    try:
        if not paired:  # the t* data 16 entries further on
            sv, t = c["sv"], c["tab"].as_engine_dict()
            d = c["tab"].desc.copy()
            d["idx"] += 16
            t["qqq_desc"] = d.view(np.uint8).reshape(-1, 16).copy()
            t["qqq"] = np.concatenate([np.zeros(16, np.float32), t["qqq"]])
            eng.set_line(fxi=c["fxi"], cyi=c["cyi"], dips=c["dips"].reshape(4, sv.nxi, sv.nzi),
                         tables=t)
            eng.begin_offset(o)
        eng.submit(rec)
        eng.get_image(False)
        t = eng.tuning()
        return t["variant"], max(t["variant_ms"]) > 0
    finally:
        eng.close()


def test_tuned_apart(cuda):
    c = make_case(nshots=1, ixstart=3, ixend=119)  # a shape no other test images
    rec = records(c)
    small = rec[400:460]
    kinds = [dict(rec=small), dict(rec=rec), dict(rec=rec, paired=False)]
    first = [_tuned(c, **k) for k in kinds]
    again = [_tuned(c, **k) for k in kinds]
    assert [own for _, own in first] == [True] * 3
    assert [own for _, own in again] == [False] * 3
    assert [v for v, _ in again] == [v for v, _ in first]
