"""psba_set_wait_limit bounds the triangular solves' waits too.  Two cameras make a
reduced system of one 16 x 16 tile, whose factor waits for nothing: with one poll
a wait, only the solve's waits for its one block can run out."""
import numpy as np
import pytest

import psba_gb300 as P
from psba_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refine", [0, 1])
def test_a_wait_that_runs_out_is_reported_and_the_handle_recovers(refine):
    sc = scenes.arc_scene(seed=2, n_cams=2, n_pts=30, arc_deg=10.0, min_views=2)
    kw = dict(allow_switch=0, max_iter=4, refine=refine)
    with P.Solver(sc) as fresh:
        want = fresh.levmar(**kw)
    with P.Solver(sc) as s:
        for _ in range(3):
            s.set_wait_limit(1)
            with pytest.raises(P.PSBAError, match="wait budget"):
                s.levmar(**kw)
            s.set_wait_limit(0)
            s.reset_params()
            got = s.levmar(**kw)
            assert got.final_cost == want.final_cost
            assert np.array_equal(got.cams, want.cams) and np.array_equal(got.pts, want.pts)
            s.reset_params()
