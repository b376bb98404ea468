"""The scans at the sizes where a segment, a warp row or a whole form of them
ends: cell grids from one cell to beyond the one-cluster limit (cell ranges and
sorted order bit-exact against the oracle), and split and removal ranks at
particle counts around the segment size (ordinary launches, which scan them as
one cluster, against the persistent step, which scans them with its whole
grid)."""
import numpy as np
import pytest

import sca2012_b200 as sph
from sca2012_b200 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "ev", "acc", "dens", "press", "energy", "surface", "level", "interior", "sibling")


@pytest.mark.parametrize("ncell", [(1, 1, 1), (3, 1, 1), (127, 1, 1), (43, 3, 1), (128, 32, 16), (257, 16, 16),
                                   (64, 64, 191), (64, 64, 192), (768, 32, 32), (787, 33, 31)])
def test_cell_scan_sizes(gpu, ncell):
    cfg = sph.preset(sph.PRESET_DAM_3D2)
    cfg.use_split = cfg.use_merge = 0
    n = 3000
    cfg.max_particle = n
    for a in range(3):
        cfg.ncell[a] = ncell[a]
        cfg.world[a] = float(np.float32(ncell[a]) * np.float32(cfg.cell_size))
        cfg.ndens[a] = 0
    r = np.random.default_rng(int(np.prod(ncell)))
    pos = (r.random((n, 3)) * np.array(ncell) * float(cfg.cell_size)).astype(np.float32)
    s = sph.Solver(cfg)
    s.set_state(dict(pos=pos, vel=np.zeros_like(pos), level=np.ones(n, np.uint32)))
    for _ in range(2):   # the second step starts from the counts the first one cleared
        before = s.get_state()["pos"]
        s.step(1)
        assert s.sync_status() == 0
        d = s.get_debug()
        key, idx, cs, ce = O.sort(cfg, before)
        assert np.array_equal(d["hash"], key) and np.array_equal(d["index"], idx)
        assert np.array_equal(d["cell_start"], cs) and np.array_equal(d["cell_end"], ce)
    s.close()


def _run(cfg, pos, level, persistent):
    s = sph.Solver(cfg)
    s.set_persistent(persistent)
    s.set_state(dict(pos=pos, vel=np.zeros_like(pos), level=level))
    out = []
    for _ in range(8):
        s.step(1)
        assert s.sync_status() == 0
        out.append((s.last_step_stats(), s.get_state()))
    s.close()
    return out


@pytest.mark.parametrize("preset", [sph.PRESET_DAM_3D2, sph.PRESET_DAM_3D4])
@pytest.mark.parametrize("counts", [(1, 1, 1), (5, 5, 5), (16, 16, 8), (17, 11, 11), (41, 40, 40)])
def test_rank_scan_sizes(gpu, preset, counts):
    cfg = sph.preset(preset)
    cfg.grid_every = 0
    cfg.merge_interior_steps = 2
    cfg.use_split = cfg.use_merge = 1
    s = float(cfg.kernel[0]) / 2
    pos = scenes.lattice(counts, s, np.full(3, 4 * s), 3, jitter=0.2)
    cfg.max_particle = 4 * len(pos)
    level = np.ones(len(pos), np.uint32)
    a, b = _run(cfg, pos, level, False), _run(cfg, pos, level, True)
    assert sum(st["n_split"] for st, _ in a) > 0
    for (sa, xa), (sb, xb) in zip(a, b):
        assert sa == sb
        for f in STATE:
            assert xa[f].tobytes() == xb[f].tobytes(), f
