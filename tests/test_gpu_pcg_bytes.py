"""The algorithmic bytes that rpba_kernel_stats reports for the PCG are those
of the form that ran: blocks that stay in shared memory are counted once a
solve, streamed ones once an iteration, with the products that pass through
memory."""
import pytest

pytestmark = pytest.mark.gpu

# (scene, size, precision, form, blocks stay)
CASES = [("arc", 33, "fp64", "resident", True), ("city", (4, 75), "fp64", "streamed", True),
         ("city", (6, 75), "fp64", "streamed", False), ("city", (6, 75), "fp64", "gathered", False),
         ("arc", 33, "mixed", "resident", True), ("city", (8, 100), "mixed", "streamed", False)]


@pytest.mark.parametrize("kind,size,precision,form,stay", CASES)
def test_bytes_by_form(kind, size, precision, form, stay):
    import rpba_b200 as rb
    from rpba_b200 import scenes
    if kind == "arc":
        blk = scenes.to_block(scenes.arc_scene(seed=5, n_cams=size, n_pts=150 * size))
    else:
        blk = scenes.to_block(scenes.city_scene(seed=8, n_clusters=size[0], cams_per_cluster=size[1],
                                                n_pts=120 * size[0] * size[1]))
    fp64 = precision == "fp64"
    with rb.Solver(blk, robust=False, precision=rb.PREC_FP64 if fp64 else rb.PREC_MIXED, verbose=2,
                   max_lm_iterations=2) as S:
        if form == "gathered":
            S.debug_pcg_form(3)
        st, rep = S.solve()
        stats = S.kernel_stats()
    rcs, pcg = stats["_rcs"], stats["pcg"]
    assert st == 0 and rcs["pcg_form"] == form
    nc, nb, it, solves = rcs["rows"], rcs["offdiag_blocks"], rep["pcg_iterations"], pcg["launches"]
    assert solves >= 1 and it >= solves
    if form == "gathered":
        blocks, products = 656 * (nc + 2 * nb), 0
    elif fp64:
        blocks, products = 664 * (nc + nb), 144 * (nc + 2 * nb) if form == "streamed" else 0
    else:
        blocks, products = 340 * (nc + nb), 128 * nb
    want = blocks * (solves if stay else it) + it * (products + nc * (648 + 22 * 72))
    assert pcg["bytes"] == want
