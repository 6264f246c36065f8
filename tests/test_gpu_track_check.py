"""Track entries that name no observation are refused by the per-point
refinement and by an Exteval handle (checked on the device), wherever in the
tracks they stand; the same block without them is taken."""
import pytest

pytestmark = pytest.mark.gpu

BAD = [("image", -1), ("image", "n"), ("slot", -1), ("slot", "count")]


@pytest.mark.parametrize("field,value", BAD)
@pytest.mark.parametrize("where", ["first", "block edge", "last"])
def test_bad_track_entry(field, value, where):
    import rpba_b200 as rb
    from rpba_b200 import scenes
    blk = scenes.to_block(scenes.arc_scene(seed=5, n_cams=5, n_pts=120))
    nt = int(blk.pt_obs_off[-1])
    t = {"first": 0, "block edge": 256, "last": nt - 1}[where]
    assert 0 <= t < nt
    rb.triangulate(blk)
    with rb.Solver(blk, exteval=True) as S:
        S.exteval()
    im = int(blk.pt_obs_image[t])
    if field == "image":
        blk.pt_obs_image[t] = blk.n_images if value == "n" else value
    else:
        blk.pt_obs_slot[t] = blk.img_obs_off[im + 1] - blk.img_obs_off[im] if value == "count" else value
    for call in (lambda: rb.triangulate(blk), lambda: rb.Solver(blk, exteval=True)):
        with pytest.raises(rb.RpbaError) as e:
            call()
        assert e.value.status == 1  # RPBA_ERR_ARG
