"""A band whose taper would end below its flat part (f3 > f4, set after the
parameters' initialisation) has a sharp edge at f3: the panels keep all of it.
Bound: relative 1e-5 in the 2-norm, ten times what two FP32 transforms of a
dozen passes and a rounded filter leave (some 1e-6)."""
import numpy as np
import pytest

from oracle import oracle as O
from q_psdm_b200 import engine as E
from tests.cuda_util import d2h
from tests.physics_case import CONTRACT, DT, DTSTAR, NBINS, NTL, TAPERZONE, THRESHOLD, gate, \
    make_case, records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f3,f4", [(90.0, 60.0), (60.0, 90.0)])
def test_panels_of_a_sharp_band(cuda, f3, f4):
    c = make_case(nshots=1, rstep=8)
    sv, st, rec = c["sv"], c["static"], records(c)
    p = E.static_params(nxi=sv.nxi, nzi=sv.nzi, ntl=NTL, dt=float(DT), dxi=sv.dxi, dyi=sv.dyi,
                        dzi=sv.dzi, fci=sv.fci, scaled=sv.scaled, fxv=sv.fxv, fyv=sv.fyv,
                        nxv=sv.nxi, nyv=sv.nyi, fc=c["fc"], threshold=THRESHOLD,
                        contract=CONTRACT, taperzone=TAPERZONE, dzii=c["tab"].dzii, mode=1,
                        panel_dtype=0, nbins=NBINS, dtstar=DTSTAR, max_batch=rec.shape[0])
    p.f3, p.f4 = f3, f4
    eng = E.Engine(p)
    try:
        eng.set_line(fxi=c["fxi"], cyi=c["cyi"], dips=c["dips"].reshape(4, sv.nxi, sv.nzi),
                     tables=c["tab"].as_engine_dict())
        az = c["az"]
        eng.begin_offset(E.offset_params(p, 0, sv.nxi, aznx1=az[0], aznx2=az[1], azny1=az[2],
                                         azny2=az[3]))
        eng.submit(rec)
        eng.get_image(False)
        got = d2h(eng.panels_device_ptrs()[0], (rec.shape[0], p.nbins, p.nffti), np.float32)
    finally:
        eng.close()
    ok = gate(c)[0][:, 0] == 3
    assert ok.sum() > 10
    filt = O.physics_filter(st["nfft"], DT, f3, f4, c["fc"], THRESHOLD, NBINS, DTSTAR)
    want = O.physics_panels(c["traces"][ok], DT, st["nfft"], st["nffti"], filt)
    assert np.linalg.norm(got[ok] - want) <= 1e-5 * np.linalg.norm(want)
