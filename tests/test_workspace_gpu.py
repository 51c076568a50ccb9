"""The workspace that a network handle keeps for the table calls: a call that
needs a larger one gives the kept one back first, so that it fits where a new
handle's call does; results as a new handle's, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from q_psdm_b200 import _lib
from q_psdm_b200 import surrogate as S

pytestmark = pytest.mark.gpu


def _line(ncell, dev):
    """A gate call's arguments for ncell cells of 4 x 4 points on 3 x 3 nodes."""
    import torch
    desc = np.zeros(ncell, S.DESC_DTYPE)
    desc["nys"] = desc["nxs"] = 3
    desc["dys"] = desc["dxs"] = 100
    desc["idx"] = np.arange(ncell) * 9 * 16
    ttt = torch.linspace(0.1, 2.0, ncell * 9 * 16, device=dev)
    ln = _lib.SurLine(ncell, 1, 4, 4, 0, 10.0, 40.0, 500.0, 1800.0, 0.5, 60.0)
    return ln, desc, ttt, torch.zeros(9 * ncell, device=dev)


def _gate(mlp, args):
    ln, desc, ttt, err = args
    return _lib.lib().qpsdm_surrogate_gate(mlp.h, C.byref(ln), desc.ctypes.data, ttt.data_ptr(),
                                           int(ttt.numel()), err.data_ptr(), None)


def test_larger_workspace_in_little_memory(cuda):
    import torch
    params = S.init_params(3)
    mlp, fresh = S.Mlp(0, params=params), S.Mlp(0, params=params)
    small, large, want = (_line(n, mlp.dev) for n in (8, 50000, 50000))
    try:
        assert _gate(mlp, small) == 0
        assert _gate(fresh, want) == 0
        fresh.close()
        torch.cuda.empty_cache()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (60 << 20), dtype=torch.uint8,
                           device="cuda")
        rc = _gate(mlp, large)
        del hold
        torch.cuda.empty_cache()
        assert rc == 0
        assert float(want[3].max()) > 0 and torch.equal(large[3], want[3])
    finally:
        mlp.close()
        fresh.close()
