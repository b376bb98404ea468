"""The two forms of the rank scans of a step (one cluster, or two launches over
a full grid) are chosen by the live count the host last knew: by launches and by
a handle that replays captured steps, with the bits of the persistent step,
which has a scan of its own, in either form."""
import numpy as np
import pytest

import sca2012_b200 as sph
from sca2012_b200 import scenes

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "ev", "acc", "dens", "press", "energy", "surface", "level", "interior", "sibling")
LIMIT = 3 << 19           # live count up to which the ranks are scanned by a cluster
CLUSTER, LAUNCHES = 2, 4  # launches of the split and the removal ranks of a step


def _setup(counts, cap, ways=2):
    cfg = sph.preset(sph.PRESET_DAM_3D4 if ways == 4 else sph.PRESET_DAM_3D2)
    cfg.grid_every = 0
    cfg.merge_interior_steps = 2
    s = float(cfg.kernel[0]) / 2
    for a in range(3):   # a cell grid that holds the block and stays one cluster's scan
        cfg.ncell[a] = max(8, counts[a] // 2 + 4)
        cfg.world[a] = float(np.float32(cfg.ncell[a]) * np.float32(cfg.cell_size))
        cfg.ndens[a] = 0
    pos = scenes.lattice(counts, s, np.full(3, 2 * s), 3, jitter=0.1)
    cfg.max_particle = cap
    return cfg, dict(pos=pos, vel=np.zeros_like(pos), level=np.ones(len(pos), np.uint32))


def _plain_launches(cfg, st):
    """Launches of the same step without splits and merges, apart from the merge pass."""
    c = cfg.copy()
    c.use_split = c.use_merge = 0
    s = sph.Solver(c)
    s.set_state(st)
    s.step(1)
    s.step(1)   # hashed by the first
    n = s.last_launch_count()
    s.close()
    return n + 1


@pytest.mark.parametrize("mode", ["launches", "graph"])
def test_form_follows_the_count(gpu, mode):
    """One handle stepped from counts on both sides of the limit (its bound is
    beyond it after a step of either), and the persistent step beside it."""
    cfg, big = _setup((128, 128, 97), 2 * 128 * 128 * 97)
    n = 128 * 128 * 96
    assert n == LIMIT
    small = {k: v[:n] for k, v in big.items()}
    base = _plain_launches(cfg, small)
    s, p = sph.Solver(cfg), sph.Solver(cfg)
    s.set_graph(mode == "graph")
    p.set_persistent(True)
    for st, form in ((big, LAUNCHES), (small, CLUSTER), (big, LAUNCHES)):
        for h in (s, p):
            h.set_state(st)
            for k in range(3):
                h.step(1)
                if h is s and k:   # the first step also hashes the new state
                    assert h.last_launch_count() == base + form
            assert h.sync_status() == 0
        stats = s.last_step_stats()
        assert stats == p.last_step_stats() and stats["n_level2"] > 0
        a, b = s.get_state(), p.get_state()
        for f in STATE:
            assert a[f].tobytes() == b[f].tobytes(), f
    s.close()
    p.close()


@pytest.mark.parametrize("mode", ["launches", "graph"])
def test_form_keeps_to_the_count_as_the_bound_grows(gpu, mode):
    """The bound of a small count grows past the limit unseen: still one cluster."""
    cfg, st = _setup((20, 20, 10), 4 << 20, ways=4)
    base = _plain_launches(cfg, st)
    outs = []
    for m in (mode, "persistent"):
        s = sph.Solver(cfg)
        s.set_graph(m == "graph")
        s.set_persistent(m == "persistent")
        s.set_state(st)
        for k in range(8):
            s.step(1)
            if m != "persistent" and k:
                assert s.last_launch_count() == base + CLUSTER, k
        outs.append((s.last_step_stats(), s.get_state()))
        assert s.sync_status() == 0
        s.close()
    (sa, xa), (sb, xb) = outs
    assert sa == sb and sa["n_end"] > len(st["pos"])
    for f in STATE:
        assert xa[f].tobytes() == xb[f].tobytes(), f
