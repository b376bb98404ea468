"""The two forms of the rank scans of a step (one cluster, or two launches over
a full grid) are chosen by the live count the host last knew, with a limit on
the host's bound: on launches and on replayed graphs, and with the bits of the
persistent step, which has a scan of its own, in either form."""
import numpy as np
import pytest

import sca2012_b200 as sph
from sca2012_b200 import scenes

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "ev", "acc", "dens", "press", "energy", "surface", "level", "interior", "sibling")
LIMIT = 3 << 19           # live count up to which the ranks are scanned by a cluster
BOUND = 1 << 22           # and the largest bound at which they are
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


@pytest.mark.parametrize("counts,form", [((128, 128, 96), CLUSTER), ((128, 128, 97), LAUNCHES)])
def test_form_follows_the_count(gpu, counts, form):
    """Counts on both sides of the limit, bounds (twice the count after a step) beyond it."""
    n = int(np.prod(counts))
    assert (n <= LIMIT) == (form == CLUSTER)
    cfg, st = _setup(counts, 2 * n)
    base = _plain_launches(cfg, st)
    outs = []
    for persistent in (False, True):
        s = sph.Solver(cfg)
        s.set_persistent(persistent)
        s.set_state(st)
        for k in range(4):
            s.step(1)
            if not persistent and k:   # the first step also hashes the new state
                assert s.last_launch_count() == base + form
        stats = s.last_step_stats()
        assert s.sync_status() == 0
        outs.append((stats, s.get_state()))
        s.close()
    (sa, xa), (sb, xb) = outs
    assert sa == sb and sa["n_level2"] > 0
    for f in STATE:
        assert xa[f].tobytes() == xb[f].tobytes(), f


@pytest.mark.parametrize("mode", ["launches", "graph"])
def test_bound_limits_the_form(gpu, mode):
    """A small count whose bound grows past its limit unseen: the scans move to
    launches, in a captured step too, with the same bits."""
    cfg, st = _setup((20, 20, 10), BOUND + 1000, ways=4)
    base = _plain_launches(cfg, st)
    outs = []
    for m in (mode, "persistent"):
        s = sph.Solver(cfg)
        s.set_graph(m == "graph")
        s.set_persistent(m == "persistent")
        s.set_state(st)
        bound = len(st["pos"])
        for k in range(8):
            s.step(1)
            if m != "persistent" and k:
                assert s.last_launch_count() == base + (CLUSTER if bound <= BOUND else LAUNCHES), k
            bound = min(4 * bound, cfg.max_particle)
        stats = s.last_step_stats()
        assert bound > BOUND and s.sync_status() == 0
        outs.append((stats, s.get_state()))
        s.close()
    (sa, xa), (sb, xb) = outs
    assert sa == sb and sa["n_end"] > len(st["pos"])
    for f in STATE:
        assert xa[f].tobytes() == xb[f].tobytes(), f
