"""The forms of the PCG kernels at their edges: systems of one group of 32
blocks, of a chunk with groups to spare, the last that keep their items or
groups resident and the first that stream them -- FP64 and mixed, with and
without the coarse space, against the FP64 direct solve.  An inexact solve at
1e-6 that converges ends within 1e-6 of the direct solver's RMS (the bar of
test_gpu_learned.py); FP32 blocks add up to 1e-6 (test_gpu_mixed.py); the bar
here is 1e-5, since the fewest cameras leave the least averaging."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (scene, cameras): off-diagonal blocks 3, 36, 528; 14.6k, about 20k (FP64:
# resident and streamed items), 65k and 83k (FP32: 75.7k blocks are one group
# for each warp of 148 CTAs)
CASES = [("arc", 3), ("arc", 9), ("arc", 33), ("city", (4, 60)), ("city", (4, 75)), ("city", (7, 95)), ("city", (8, 100))]


@pytest.mark.parametrize("kind,size", CASES)
def test_pcg_forms_reach_direct(kind, size):
    import rpba_b200 as rb
    from rpba_b200 import scenes
    if kind == "arc":
        blk = scenes.to_block(scenes.arc_scene(seed=5, n_cams=size, n_pts=150 * size))
    else:
        blk = scenes.to_block(scenes.city_scene(seed=8, n_clusters=size[0], cams_per_cluster=size[1],
                                                n_pts=120 * size[0] * size[1]))

    def solve(**kw):
        S = rb.Solver(blk, **kw)
        st, rep = S.solve()
        out = S.state()
        S.close()
        assert st == 0 and np.isfinite(out.XX).all() and np.isfinite(out.pmat).all(), kw
        return rep

    ref = solve(solver=rb.SOLVER_DIRECT)
    for prec in (rb.PREC_FP64, rb.PREC_MIXED):
        for coarse in (-1, 0):
            rep = solve(solver=rb.SOLVER_LEARNED, precision=prec, pcg_tolerance=1e-6, coarse_aggregates=coarse)
            # (FP32 block-Jacobi alone may run out of iterations and be solved directly)
            assert rep["pcg_fallbacks"] == 0 or (prec == rb.PREC_MIXED and coarse == -1), (prec, coarse)
            assert abs(rep["rms"] - ref["rms"]) <= 1e-5 * ref["rms"], (prec, coarse, rep["rms"], ref["rms"])
