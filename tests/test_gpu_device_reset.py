"""A program may reset its device context between simulations: a handle made
afterwards works as the first one did (what the library keeps per process must
not rest on state that the reset discards).  Runs in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes
import numpy as np
import sca2012_b200 as sph

def run(mode):
    cfg = sph.preset(sph.PRESET_DAM_3D2)
    cfg.max_particle, cfg.grid_every = 4000, 0
    pos = (np.random.default_rng(0).random((1000, 3)) * 0.2 + 0.1).astype(np.float32)
    s = sph.Solver(cfg)
    s.set_graph(mode == "graph")
    s.set_persistent(mode == "persistent")
    s.set_state(dict(pos=pos, vel=np.zeros_like(pos), level=np.ones(1000, np.uint32)))
    s.step(3)
    assert s.sync_status() == 0
    out = s.get_state()["pos"].tobytes()
    s.close()
    return out

for mode in ("launches", "graph", "persistent"):
    before = run(mode)
    assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0
    assert run(mode) == before
print("ok")
"""


def test_a_handle_after_a_device_reset(gpu):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
