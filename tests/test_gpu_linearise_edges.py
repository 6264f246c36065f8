"""The point, camera and pair passes at the edges of their chunks: three cameras that
all see every point, with as many points as fit, just fill and just overflow
a chunk of 24 observations or of 16 (FP64) and 32 (FP32) contributions, and a
few of each.  Two LM steps: FP64 against the oracle at the drop-in contract's
bounds (cost 1e-8, parameters 1e-6), mixed within 1e-5 of the FP64 cost
(test_gpu_mixed.py's bar for inexact solves, its direct bar 1e-6 being for
thousands of points)."""
import numpy as np
import pytest

from tests.parity_util import COST_RTOL, PARAM_RTOL, param_errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [15, 16, 17, 23, 24, 25, 31, 32, 33, 48, 49, 64, 65, 97])
def test_chunk_edges(oracle_mod, points):
    from rpba_b200 import scenes
    blk = scenes.to_block(scenes.arc_scene(seed=40 + points, n_cams=3, n_pts=points, track_mean=50.0, outlier_frac=0.0))
    assert (np.diff(blk.pt_obs_off) == 3).sum() >= points - 3  # (a point may leave an image)
    _check_steps(oracle_mod, blk)


@pytest.mark.parametrize("points", [16, 17, 24, 33])
def test_long_tracks(oracle_mod, points):
    """Tracks of up to 40 observations: the point pass takes eight points'
    observations 32 at a time, whichever point they belong to."""
    from rpba_b200 import scenes
    blk = scenes.to_block(scenes.arc_scene(seed=90 + points, n_cams=40, n_pts=points, track_mean=60.0, track_max=40,
                                           outlier_frac=0.0))
    assert np.diff(blk.pt_obs_off).max() > 32
    _check_steps(oracle_mod, blk)


def _check_steps(oracle_mod, blk):
    import rpba_b200 as rb
    kw = dict(robust=False, max_lm_iterations=2)
    st, ora, rep_o, _ = oracle_mod.calc_plsa(blk, rb.make_options(solver=rb.SOLVER_DIRECT, **kw))
    assert st == 0

    def solve(precision):
        with rb.Solver(blk, solver=rb.SOLVER_DIRECT, precision=precision, **kw) as S:
            st, rep = S.solve()
            assert st == 0
            return rep, S.state()

    rep, out = solve(rb.PREC_FP64)
    assert abs(rep["cost"] - rep_o["cost"]) <= COST_RTOL * rep_o["cost"]
    err = param_errors(out, ora)
    assert max(err.values()) <= PARAM_RTOL, err
    rep32, _ = solve(rb.PREC_MIXED)
    assert abs(rep32["cost"] - rep["cost"]) <= 1e-5 * rep["cost"]
