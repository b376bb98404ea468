"""Steps as programmatic dependent launches against the same steps replayed
from graphs (ordinary edges) and run by the persistent kernel (no launches
between the stages), over enough steps and launches in a row that a kernel
reading before its predecessor's writes were visible would show: sizes of one
block per SM and below (every kernel a dependent) and above (the pair passes are
not), adaptive, and the same step recorded by the caller's own stream capture."""
import numpy as np
import pytest

import sca2012_b200 as sph
from sca2012_b200 import scenes

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "ev", "acc", "dens", "press", "energy", "surface", "level", "interior", "sibling")


def _setup(counts, ways):
    cfg = sph.preset(sph.PRESET_DAM_3D4 if ways == 4 else sph.PRESET_DAM_3D2)
    cfg.grid_every = 0
    cfg.merge_interior_steps = 5
    s = float(cfg.kernel[0]) / 2
    pos = scenes.lattice(counts, s, np.full(3, 2 * s), 5, jitter=0.1)
    cfg.max_particle = 4 * len(pos)
    vel = np.random.default_rng(5).normal(0.0, 0.2, pos.shape).astype(np.float32)
    return cfg, dict(pos=pos, vel=vel, ev=vel, level=np.ones(len(pos), np.uint32))


def _run(cfg, st, steps, mode):
    s = sph.Solver(cfg)
    s.set_graph(mode == "graph")
    s.set_persistent(mode == "persistent")
    s.set_state(st)
    s.step(steps)
    assert s.sync_status() == 0
    out = s.get_state()
    s.close()
    return out


@pytest.mark.parametrize("counts,ways", [((3, 3, 3), 2), ((16, 16, 16), 4), ((27, 26, 27), 2), ((40, 40, 32), 4)])
def test_dependent_launches_equal_graph_and_persistent(gpu, counts, ways):
    cfg, st = _setup(counts, ways)
    want = _run(cfg, st, 60, "graph")
    for mode in ("launches", "launches", "persistent"):
        got = _run(cfg, st, 60, mode)
        for f in STATE:
            assert got[f].tobytes() == want[f].tobytes(), (mode, f)


def test_step_recorded_by_the_caller(gpu):
    import torch
    cfg, st = _setup((20, 20, 20), 2)
    want = _run(cfg, st, 6, "launches")
    stream = torch.cuda.Stream()
    s = sph.Solver(cfg)
    s.set_stream(stream.cuda_stream)
    s.set_state(st)
    s.step(4)   # the launch shapes no longer change with the count's bound
    s.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        s.step(2)   # both buffers, so that a replay starts where the recording did
    g.replay()
    torch.cuda.synchronize()
    got = s.get_state()
    s.close()
    for f in STATE:
        assert got[f].tobytes() == want[f].tobytes(), f
