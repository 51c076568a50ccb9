"""Compensated sums of an image whose tiles' members are split into parts.

A gather goes in as one batch (in parts), then negated in small batches (not
split): what is left is the sums' rounding alone.  A compensated sum rounds
each value it adds (half an ulp of the value), a part kept as one float the
part's sum: at the diffractors, where values add up coherently, some 60 times
as much per part, 8 times in the total.  So the residual there is held to twice
that of a run whose batches are all too small to be split."""
import numpy as np
import pytest

from tests.physics_case import engine, make_case, records

pytestmark = pytest.mark.gpu


def _residual(c, variant, pieces):
    rec = records(c)
    neg = records(dict(c, traces=-c["traces"]))
    eng, _, _ = engine(c, panel_dtype=0, form=1, variant=variant, kahan=1, max_batch=rec.shape[0])
    try:
        for r in np.array_split(rec, pieces):
            eng.submit(np.ascontiguousarray(r))
        img = eng.get_image(False).copy()
        for r in np.array_split(neg, 13):
            eng.submit(np.ascontiguousarray(r))
        return img, eng.get_image(False)
    finally:
        eng.close()


@pytest.mark.parametrize("variant", [13, 26, 15, 27])
def test_parts_keep_their_compensation(cuda, variant):
    c = make_case(nshots=1)
    img, split = _residual(c, variant, 1)
    _, whole = _residual(c, variant, 10)  # 103 traces: one part
    top = np.abs(img) >= np.quantile(np.abs(img), 0.99)
    rms = lambda a: float(np.sqrt(np.mean(np.square(a[top], dtype=np.float64))))
    assert np.abs(img).max() > 0 and rms(whole) > 0
    assert rms(split) <= 2.0 * rms(whole)
