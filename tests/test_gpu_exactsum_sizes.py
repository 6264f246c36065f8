"""The exact float sum at the edges of its forms -- the sequential head, the
windows of one CTA, the first length the grid form takes and its chunk
remainders -- bit for bit against numpy's sequential float32 cumsum, from
16-byte aligned and unaligned addresses."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 511, 512, 513, 2559, 2560, 2561, 8193, 65535, 65536, 65537, 65541, 131073, 300_007]
KINDS = ["cost-like", "ties", "heavy tail", "subnormal start"]


def _values(kind, n):
    rng = np.random.default_rng(n)
    if kind == "cost-like":
        v = rng.normal(0, 0.5, n) ** 2
    elif kind == "ties":
        v = rng.integers(0, 4, n) * 0.5
    elif kind == "heavy tail":
        v = np.exp(rng.normal(0, 6, n))
    else:
        v = np.where(np.arange(n) > n // 2, rng.random(n), 1e-42 * rng.integers(0, 3, n))
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", KINDS)
def test_exact_sum_at_form_edges(kind):
    import torch
    import rpba_b200 as rb
    L = rb.load()
    for n in SIZES:
        v = _values(kind, n)
        ref = np.cumsum(v, dtype=np.float32)[-1]
        assert rb.float_sequential_sum(v).tobytes() == ref.tobytes(), (kind, n)
        for skip in (0, 1, 3):  # the device array's alignment
            dv = torch.zeros(n + skip, dtype=torch.float32, device="cuda")
            dv[skip:] = torch.from_numpy(v).cuda()
            out = torch.zeros(1, dtype=torch.float32, device="cuda")
            st = L.rpba_float_sequential_sum_noalloc(C.c_void_p(dv.data_ptr() + 4 * skip), n,
                                                     C.c_void_p(out.data_ptr()),
                                                     C.c_void_p(torch.cuda.current_stream().cuda_stream))
            torch.cuda.synchronize()
            assert st == 0 and out.cpu().numpy()[0].tobytes() == ref.tobytes(), (kind, n, skip)
