"""Device memory of an FP64 solve: the PCG's streamed form, which keeps the
products of every block, takes no more than reading every block from both
sides did (490,421,399 bytes in the pool for this scene of 83,251 blocks,
measured before the form existed)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu
BEFORE = 490_421_399


def _pool_used():
    import torch
    torch.zeros(1, device="cuda")
    rt = C.CDLL("libcudart.so.12")
    pool, v = C.c_void_p(), C.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(v)) == 0  # cudaMemPoolAttrUsedMemCurrent
    return v.value


def test_fp64_pcg_memory():
    import rpba_b200 as rb
    from rpba_b200 import scenes
    blk = scenes.to_block(scenes.city_scene(seed=8, n_clusters=8, cams_per_cluster=100, n_pts=96_000))
    used = _pool_used()
    with rb.Solver(blk) as S:
        st, _ = S.solve()
        assert st == 0
        stats = S.kernel_stats()["_rcs"]
        assert stats["pcg_form"] == "streamed"
        assert _pool_used() - used <= BEFORE
