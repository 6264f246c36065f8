"""One linear solve of every form of the PCG against the direct solve of the
same system, and the drop-in stop rule against the oracle's: no later LM step
can absorb a wrong operator, and no fallback stands in for the PCG.

Bars.  A step that stops at the relative preconditioned residual t has an
A-norm error of at most t sqrt(cond(M^-1 A)) of the step; the damping (1e-4 of
the diagonal) bounds an entry's error in the diagonal's units by 100 times
that.  sqrt(cond) is 60 or less here (660 iterations to 1e-10, 95 to 1e-6), so
FP64 at 1e-10 is within 1e-6, held to 1e-4 since the groups mix units; mixed at
1e-6 within 6e-3, its FP32 products (2e-7 over the damping) another 2e-3, held
to 2e-2.  A row's piece lost between groups is a percent of its row or more,
over the damping a multiple of the step.  The state comes back in floats: four
units of the last place on top."""
import functools

import numpy as np
import pytest

from tests.parity_util import COST_RTOL, PARAM_RTOL, param_errors

pytestmark = pytest.mark.gpu
FORMS = {"resident": 0, "streamed": 2, "gathered": 3}
GROUPS = ("pmat", "K", "distpara", "XX")
# (scene, size, points a camera) -> the library's form, FP64 and FP32
CASES = [("arc", 9, 150, "resident", "resident"), ("arc", 33, 150, "resident", "resident"),
         ("city", (4, 60), 120, "resident", "resident"), ("city", (6, 75), 120, "streamed", "resident"),
         ("city", (8, 100), 120, "streamed", "streamed")]


@functools.lru_cache(maxsize=1)
def _block(kind, size, per):
    from rpba_b200 import scenes
    if kind == "arc":
        return scenes.to_block(scenes.arc_scene(seed=5, n_cams=size, n_pts=per * size))
    return scenes.to_block(scenes.city_scene(seed=8, n_clusters=size[0], cams_per_cluster=size[1],
                                             n_pts=per * size[0] * size[1]))


def _step(blk, form=0, **kw):
    import rpba_b200 as rb
    with rb.Solver(blk, robust=False, max_lm_iterations=1, **kw) as S:
        S.debug_pcg_form(form)
        st, rep = S.solve()
        assert st == 0 and rep["linear_solves"] == 1
        return S.state(), rep, S.kernel_stats()["_rcs"]["pcg_form"]


@pytest.mark.parametrize("kind,size,per,fp64,fp32", CASES)
def test_one_solve_equals_direct(kind, size, per, fp64, fp32):
    import rpba_b200 as rb
    blk = _block(kind, size, per)
    for prec, chosen, tol, bar in ((rb.PREC_FP64, fp64, 1e-10, 1e-4), (rb.PREC_MIXED, fp32, 1e-6, 2e-2)):
        ref, _, _ = _step(blk, precision=prec, solver=rb.SOLVER_DIRECT)
        names = list(FORMS) if prec == rb.PREC_FP64 else ["resident", "streamed"]
        for name in names[names.index(chosen):]:
            for coarse in (-1, 0):
                out, rep, ran = _step(blk, FORMS[name] if name != chosen else 0, precision=prec,
                                      solver=rb.SOLVER_LEARNED, pcg_tolerance=tol, coarse_aggregates=coarse)
                assert ran == name and rep["pcg_fallbacks"] == 0 and rep["pcg_iterations"] > 0
                for g in GROUPS:
                    a, b, p = (np.asarray(getattr(x, g), np.float64) for x in (out, ref, blk))
                    step = np.abs(b - p).max()
                    assert step > 0
                    err = np.abs(a - b).max()
                    assert err <= bar * step + 4 * 2.0 ** -24 * np.abs(b).max(), (prec, name, coarse, g, err, step)


@pytest.mark.parametrize("cams", [9, 33])
def test_drop_in_solve_equals_oracle(oracle_mod, cams):
    """The reference's stop rule and set-up, in each FP64 form: the drop-in
    contract's bars on the arc scene."""
    import rpba_b200 as rb
    blk = _block("arc", cams, 150)
    st, ora, rep_o, _ = oracle_mod.calc_plsa(blk, rb.make_options(solver=rb.SOLVER_PCG, robust=False,
                                                                  max_lm_iterations=1))
    assert st == 0
    for name, form in FORMS.items():
        out, rep, ran = _step(blk, form, solver=rb.SOLVER_PCG)
        assert ran == name and rep["pcg_iterations"] > 0
        assert abs(rep["cost"] - rep_o["cost"]) <= COST_RTOL * rep_o["cost"]
        err = param_errors(out, ora)
        assert max(err.values()) <= PARAM_RTOL, (name, err)
