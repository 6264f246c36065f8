"""The forms of the persistent PCG give the same bits: a solve with the form
the library chooses, and the same solve with the blocks streamed, and gathered
from global memory (test hook), end in the same state, byte for byte.  Each
form is the one that ran (asked back from the handle)."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (scene, size, points a camera) -> the library's form, FP64 and FP32.  Off-diagonal
# blocks: 3, 36, 528; 528 of fewer than seven contributions (the streamed
# form's products in memory of their own); 14.6k; 22k (FP64: each stage's only
# group stays) and 35k; 65k, the most a warp a group holds on 148 SMs, and 83k
CASES = [("arc", 3, 150, "resident", "resident"), ("arc", 9, 150, "resident", "resident"),
         ("arc", 33, 150, "resident", "resident"), ("arc", 33, 10, "resident", "resident"),
         ("city", (4, 60), 120, "resident", "resident"), ("city", (4, 75), 120, "streamed", None),
         ("city", (6, 75), 120, "streamed", None), ("city", (7, 95), 120, None, "resident"),
         ("city", (8, 100), 120, None, "streamed")]


@functools.lru_cache(maxsize=1)
def _block(kind, size, per):
    from rpba_b200 import scenes
    if kind == "arc":
        return scenes.to_block(scenes.arc_scene(seed=5, n_cams=size, n_pts=per * size))
    return scenes.to_block(scenes.city_scene(seed=8, n_clusters=size[0], cams_per_cluster=size[1],
                                             n_pts=per * size[0] * size[1]))


def _state(blk, form, **kw):
    import rpba_b200 as rb
    with rb.Solver(blk, **kw) as S:
        S.debug_pcg_form(form)
        st, rep = S.solve()
        assert st == 0
        out = S.state()
        ran = S.kernel_stats()["_rcs"]["pcg_form"]
    arrays = [getattr(out, n) for n in ("pmat", "K", "distpara", "XX", "pt_obs_off", "pt_obs_image", "pt_obs_slot")]
    return ran, [a.tobytes() for a in arrays], [rep[k] for k in ("linear_solves", "pcg_iterations", "pcg_fallbacks", "cost")]


@pytest.mark.parametrize("kind,size,per,fp64,fp32", CASES)
def test_forms_give_the_same_bits(kind, size, per, fp64, fp32):
    import rpba_b200 as rb
    blk = _block(kind, size, per)
    # the drop-in form; the relative stop rule, without and with the coarse space
    solvers = (dict(solver=rb.SOLVER_PCG), dict(solver=rb.SOLVER_LEARNED, pcg_tolerance=1e-4, coarse_aggregates=-1),
               dict(solver=rb.SOLVER_LEARNED, pcg_tolerance=1e-4, coarse_aggregates=0))
    for prec, chosen, others in ((rb.PREC_FP64, fp64, ("streamed", "gathered")), (rb.PREC_MIXED, fp32, ("streamed",))):
        if chosen is None:
            continue
        for kw in solvers:
            ran, state, rep = _state(blk, 0, precision=prec, **kw)
            assert ran == chosen, (prec, kw)
            for other in others:
                r, s, p = _state(blk, {"streamed": 2, "gathered": 3}[other], precision=prec, **kw)
                assert r == other
                assert p == rep and s == state, (prec, kw, other, p, rep)
            assert np.isfinite(rep[-1])
