"""set_line and begin_offset that fail for device memory: nothing is submitted,
replayed from a graph or read until they have been called again, and then the
engine images as before.  (Before, the buffers that the failed call had freed
stayed in use.)"""
import ctypes as C

import numpy as np
import pytest

from q_psdm_b200 import _lib
from q_psdm_b200 import engine as E
from tests.physics_case import engine, make_case, records

pytestmark = pytest.mark.gpu
ENOMEM, ESTATE = 3, 4


def _code(f, *a):
    with pytest.raises(E.QpsdmError) as x:
        f(*a)
    return x.value.code


def _set(c, eng):
    sv = c["sv"]
    eng.set_line(fxi=c["fxi"], cyi=c["cyi"], dips=c["dips"].reshape(4, sv.nxi, sv.nzi),
                 tables=c["tab"].as_engine_dict())


def _refused(eng, rec):
    assert _code(eng.submit, rec) == ESTATE
    assert _code(eng.get_image, False) == ESTATE


@pytest.mark.parametrize("form", [0, 1])
def test_set_line_without_memory(cuda, form):
    c = make_case(nshots=1, rstep=2)
    rec = records(c)
    eng, p, o = engine(c, form=form, variant=26 if form else 0, use_graph=1)
    try:
        for _ in range(3):  # eager, captured, replayed
            eng.submit(rec)
        want = eng.get_image(False).copy()
        keep = []
        sv, lp = c["sv"], None
        lp = eng._line_params(keep, fxi=c["fxi"], cyi=c["cyi"],
                              dips=c["dips"].reshape(4, sv.nxi, sv.nzi),
                              tables=c["tab"].as_engine_dict())
        lp.ttt_len = lp.qqq_len = 1 << 38  # allocated before any of it is read
        assert _lib.lib().qpsdm_set_lines(eng.h, C.byref(lp), 1) == ENOMEM
        _refused(eng, rec)
        _set(c, eng)
        _refused(eng, rec)
        eng.begin_offset(o)
        for _ in range(3):
            eng.submit(rec)
        assert np.array_equal(eng.get_image(False), want)
    finally:
        eng.close()


@pytest.mark.parametrize("form", [0, 1])
def test_begin_offset_without_memory(cuda, form):
    import torch
    c = make_case(nshots=1, rstep=2)
    rec = records(c)
    eng, p, o = engine(c, form=form, variant=26 if form else 0, use_graph=1, max_batch=1 << 15)
    try:
        for _ in range(3):
            eng.submit(rec)
        want = eng.get_image(False).copy()
        big = E.offset_params(p, 0, p.nxi, aznx1=40, aznx2=40, azny1=30, azny2=30)
        big.nww = big.nsb // 2 + 1 - big.nf1  # spectra of every frequency: more than is left
        torch.cuda.empty_cache()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), dtype=torch.uint8,
                           device="cuda")
        rc = _code(eng.begin_offset, big)
        del hold
        torch.cuda.empty_cache()
        assert rc == ENOMEM
        _refused(eng, rec)
        eng.begin_offset(o)
        for _ in range(3):
            eng.submit(rec)
        assert np.array_equal(eng.get_image(False), want)
    finally:
        eng.close()
