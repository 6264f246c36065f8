"""The status of a call on a device without room for it: a bad track entry is
RPBA_ERR_ARG there too, a good block RPBA_ERR_CUDA, and the calls work again
once there is room."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (a process of its own: the library's memory pool keeps what earlier handles
# used, which would leave room)
CODE = """
import numpy as np, torch
import rpba_b200 as rb
from rpba_b200 import scenes
from rpba_b200.block import Block

small = scenes.to_block(scenes.arc_scene(seed=5, n_cams=5, n_pts=120))
rb.triangulate(small)
n, nt = 4, 60_000_000  # one track of two slots' entries over and over: 480 MB here, over 1.4 GB there
big = Block(small.pmat[:n].copy(), small.K[:n].copy(), small.distpara[:n].copy(), small.XX[:1].copy(),
            np.arange(0, 2 * n + 1, 2, dtype=np.int32), np.zeros((2 * n, 2), np.float32), *(np.ones(2 * n, np.float32) for _ in range(3)),
            np.array([0, nt], np.int32), np.zeros(nt, np.int32), np.zeros(nt, np.int32))

def status(call):
    try:
        r = call()
        if hasattr(r, "close"):
            r.close()
        return 0
    except rb.RpbaError as e:
        return e.status

def both(b):
    return [status(lambda: rb.triangulate(b)), status(lambda: rb.Solver(b, exteval=True))]

free, _ = torch.cuda.mem_get_info()
hold = torch.empty(free - (600 << 20), dtype=torch.uint8, device="cuda")
assert both(big) == [2, 2], "good, no room"
big.pt_obs_slot[-1] = 2
assert both(big) == [1, 1], "bad, no room"
assert both(small) == [0, 0], "small, while the rest is held"
del hold
torch.cuda.empty_cache()
assert both(big) == [1, 1], "bad, room"
print("ok")
"""


def test_status_without_room():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
