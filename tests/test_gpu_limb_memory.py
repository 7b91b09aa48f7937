"""The FP64 form's limb rows (fx_words of 8 bytes each for Y and W, and one word of
exponents, per observation) come with a handle's first FP64 solve; a handle that
runs the mixed form only does not have them."""
import pytest

import psba_gb300 as P
from psba_gb300 import scenes

pytestmark = pytest.mark.gpu
WORDS = {6: 24, 11: 48, 16: 60}


@pytest.mark.parametrize("cnp", [6, 11, 16])
def test_limb_rows_come_with_the_first_fp64_solve(cnp):
    sc = scenes.arc_scene(seed=5, n_cams=5, n_pts=60, arc_deg=12.0, min_views=3)
    if cnp > 6:
        sc = scenes.with_intrinsics(sc, cnp, seed=1)
    with P.Solver(sc) as s:
        made = s.device_bytes()
        s.levmar(allow_switch=0, max_iter=2, precision=P.PREC_MIXED)
        assert s.device_bytes() == made
        s.reset_params()
        first = s.levmar(allow_switch=0, max_iter=2)
        assert s.device_bytes() == made + sc.n_obs * 8 * (2 * WORDS[cnp] + 1)
        s.reset_params()
        assert s.levmar(allow_switch=0, max_iter=2).final_cost == first.final_cost
        assert s.device_bytes() == made + sc.n_obs * 8 * (2 * WORDS[cnp] + 1)
