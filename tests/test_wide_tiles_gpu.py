"""The 16 x 16 tiles that the autotuner mostly picks, with half-precision panels,
against the FP64 oracle: its bounds for FP16 (2.5e-4) and BF16 panels (1e-3)."""
import pytest

from tests.physics_case import engine, make_case, nrmse, oracle_run, records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ixstart", [0, 30])  # 30: tiles that straddle table cells
def test_wide_tiles(cuda, ixstart):
    c = make_case(nshots=2, ixstart=ixstart, ixend=126)
    ref, npt, _ = oracle_run(c)
    for variant in (26, 27):
        for dtype, bound in ((2, 2.5e-4), (1, 1e-3)):
            eng, _, _ = engine(c, panel_dtype=dtype, form=1, variant=variant)
            try:
                eng.submit(records(c))
                img = eng.get_image(False)
                assert eng.counters()[1] == npt
                assert eng.tuning()["variant"] == variant - 1
            finally:
                eng.close()
            assert nrmse(img, ref) <= bound, (variant, dtype)
