"""Bounded device waits that run out one at a time (test hook): the kernel
leaves, the call ends with the device-timeout status instead of hanging, and
the same handle then gives what a fresh one gives, byte for byte."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LIMIT = 20_000_000  # ns


def _city(clusters, cams):
    from rpba_b200 import scenes
    return scenes.to_block(scenes.city_scene(seed=8, n_clusters=clusters, cams_per_cluster=cams,
                                             n_pts=120 * clusters * cams))


def _arc():
    from rpba_b200 import scenes
    return scenes.to_block(scenes.arc_scene(seed=5, n_cams=20, n_pts=2000))


def _same(a, b):
    return all(np.array_equal(getattr(a, n), getattr(b, n), equal_nan=True)
               for n in ("pmat", "K", "distpara", "XX", "pt_obs_off", "pt_obs_image", "pt_obs_slot"))


def _runs_out(S, which, call):
    import rpba_b200 as rb
    S.debug_wait_fault(which, LIMIT)
    t0 = time.perf_counter()
    with pytest.raises(rb.RpbaError) as e:
        call()
    assert e.value.status == 6, e.value
    assert time.perf_counter() - t0 < 30.0
    S.debug_wait_fault(0, 0)


# a copy that never completes, in each form of the PCG: FP64 items resident,
# groups resident (22k blocks), groups streamed (35k); FP32 a group a warp,
# groups streamed (83k) -- with and without the coarse space
@pytest.mark.parametrize("scene,precision", [("arc", "fp64"), ((4, 75), "fp64"), ((6, 75), "fp64"), ("arc", "mixed"),
                                             ((8, 100), "mixed")])
def test_copy_that_never_completes(scene, precision):
    import rpba_b200 as rb
    blk = _arc() if scene == "arc" else _city(*scene)
    prec = rb.PREC_FP64 if precision == "fp64" else rb.PREC_MIXED
    for kw in (dict(solver=rb.SOLVER_PCG), dict(solver=rb.SOLVER_LEARNED, pcg_tolerance=1e-4)):
        with rb.Solver(blk, precision=prec, **kw) as S, rb.Solver(blk, precision=prec, **kw) as F:
            _runs_out(S, 1, S.solve)
            st, _ = S.solve()
            st_f, _ = F.solve()
            assert st == st_f == 0
            assert _same(S.state(), F.state())


def _arc_large():
    """More than 65,536 points and observations: the sums run on every SM."""
    from rpba_b200 import scenes
    return scenes.to_block(scenes.arc_scene(seed=5, n_cams=20, n_pts=66_000))


def test_exteval_sum_that_never_comes():
    import rpba_b200 as rb
    blk = _arc_large()
    assert blk.n_points > 65536
    with rb.Solver(blk, exteval=True) as S, rb.Solver(blk, exteval=True) as F:
        for _ in range(2):
            _runs_out(S, 2, S.exteval)
            res, rep = S.exteval()
            res_f, rep_f = F.exteval()
            assert np.array_equal(res, res_f, equal_nan=True)
            for key in ("exteval_sigma0", "exteval_nrobs", "exteval_redundancy"):
                assert rep[key] == rep_f[key], key


def test_solve_sum_that_never_comes():
    import rpba_b200 as rb
    blk = _arc_large()
    with rb.Solver(blk) as S, rb.Solver(blk) as F:
        _runs_out(S, 2, S.solve)
        st, _ = S.solve()
        st_f, _ = F.solve()
        assert st == st_f == 0
        assert _same(S.state(), F.state())


@pytest.mark.parametrize("which", [3, 4])
def test_direct_solve_wait(which):
    """The envelope solve's first row, and the factorisation's barrier."""
    import rpba_b200 as rb
    blk = _arc()
    with rb.Solver(blk, solver=rb.SOLVER_DIRECT) as S, rb.Solver(blk, solver=rb.SOLVER_DIRECT) as F:
        _runs_out(S, which, S.solve)
        st, _ = S.solve()
        st_f, _ = F.solve()
        assert st == st_f == 0
        assert _same(S.state(), F.state())
