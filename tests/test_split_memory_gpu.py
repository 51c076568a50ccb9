"""An offset group begun in little device memory: where the sums of split tiles
do not fit (32 MB per grouping set), tiles are not split.  The image equals the
plain form's to the bound of the batched form (2e-5 of the peak)."""
import numpy as np
import pytest

from q_psdm_b200 import engine as E
from q_psdm_b200 import synth, tables

pytestmark = pytest.mark.gpu
X0, Y0, NXI, NZI, NT, NTR = 500000.0, 4000000.0, 640, 500, 600, 300


def _image(left=None, **kw):
    import torch
    sv = synth.config2(0)
    tfn = lambda px, py, x, z: synth.traveltime(sv, np.hypot(px - x, py), z)
    tab = tables.build_line_tables(tfn, lambda *a: tfn(*a) / 80.0, fci=1, nxi=NXI, dxi=10.0,
                                   zmax=(NZI - 1) * 10.0, dzii=80.0, nxi1=16, nzi1=64,
                                   surf_dx=320, surf_dy=320, half_x=1600.0, half_y=640.0)
    rng = np.random.default_rng(4)
    s = rng.uniform(0.3, 0.7, NTR) * NXI * 10.0
    hdr = np.stack([X0 + s, np.full(NTR, Y0), X0 + s + rng.uniform(-600, 600, NTR),
                    Y0 + rng.uniform(-100, 100, NTR)], 1)
    rec = E.encode_su(*np.rint(hdr * 100).astype(np.int32).T,
                      rng.standard_normal((NTR, NT)).astype(np.float32), dt_us=2000, scalco=-100)
    p = E.static_params(nxi=NXI, nzi=NZI, ntl=NT, dt=0.002, dxi=10.0, dyi=10.0, dzi=10.0,
                        scaled=0.01, fxv=X0, fyv=Y0 - 4000.0, nxv=NXI, nyv=1000, max_batch=NTR,
                        mode=1, panel_dtype=0, nbins=4, dtstar=0.002, dzii=80.0, **kw)
    eng = E.Engine(p)
    try:
        eng.set_line(fxi=X0, cyi=Y0, dips=np.stack(synth.dip_fields(NXI, NZI, 0.05)),
                     tables=tab.as_engine_dict())
        torch.cuda.empty_cache()
        hold = None if left is None else torch.empty(torch.cuda.mem_get_info()[0] - left,
                                                     dtype=torch.uint8, device="cuda")
        eng.begin_offset(E.offset_params(p, 0, NXI, aznx1=60, aznx2=60, azny1=40, azny2=40))
        del hold
        torch.cuda.empty_cache()
        eng.submit(rec)
        return eng.get_image(False), eng.stats()
    finally:
        eng.close()


@pytest.mark.parametrize("kahan", [0, 1])
def test_no_room_for_parts(cuda, kahan):
    plain, s0 = _image(form=0, kahan=kahan)
    for left in (None, 24 << 20):
        img, s1 = _image(left, form=1, variant=26, kahan=kahan)
        assert s1["point_traces"] == s0["point_traces"]
        assert np.abs(plain).max() > 0
        assert np.abs(img - plain).max() <= 2e-5 * np.abs(plain).max()
