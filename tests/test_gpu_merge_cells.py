"""The per-cell merge pass over cell populations around its list and warp
sizes: cells of 1 to 600 eligible members (the list holds 256), every few cells
empty, on grids of one cell, of a few and of more cells than the launch has
warps.  Bit-identical between the ordinary launches and the persistent step
(another grid, so another number of cells per warp), and the number of groups is
that of the rule: floor(eligible members / ways) per cell, a member being
eligible when its score (NaN without a neighbour) is below the criterion."""
import numpy as np
import pytest

import sca2012_b200 as sph
from oracle import oracle as O

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "ev", "acc", "dens", "press", "energy", "surface", "level")


@pytest.mark.parametrize("ways", [2, 4])
@pytest.mark.parametrize("ncell,members", [((1, 1, 1), [600]), ((3, 2, 1), [1, 3, 4, 33, 257, 0]),
                                           ((8, 8, 8), [14] * 512), ((8, 8, 8), [5, 0, 40, 1] * 128),
                                           ((90, 70, 60), [9, 0, 2] * 400)])
def test_merge_groups_per_cell(gpu, ncell, members, ways):
    cfg = sph.preset(sph.PRESET_REF_3D4 if ways == 4 else sph.PRESET_REF_3D2)
    cfg.use_split, cfg.use_merge = 0, 1
    cfg.merge_criteria = 1e30      # every level-2 particle is eligible
    cfg.grid_every = 0
    cells = np.arange(int(np.prod(ncell)))
    for a in range(3):
        cfg.ncell[a] = ncell[a]
        cfg.world[a] = float(np.float32(ncell[a]) * np.float32(cfg.cell_size))
        cfg.ndens[a] = 0
    r = np.random.default_rng(len(members))
    count = np.zeros(len(cells), np.int64)
    count[: len(members)] = members
    at = np.stack([cells % ncell[0], cells // ncell[0] % ncell[1], cells // (ncell[0] * ncell[1])], 1)
    pos = (np.repeat(at, count, 0) + 0.1 + 0.8 * r.random((count.sum(), 3))) * float(cfg.cell_size)
    pos = pos.astype(np.float32)
    order = r.permutation(len(pos))
    pos = pos[order]
    cfg.max_particle = len(pos)
    out = []
    for merge, persistent in ((0, False), (1, False), (1, True)):
        c = cfg.copy()
        c.use_merge = merge
        s = sph.Solver(c)
        s.set_persistent(persistent)
        s.set_state(dict(pos=pos, vel=np.zeros_like(pos), level=np.full(len(pos), 2, np.uint32)))
        s.step(1)
        s.sync_status()
        out.append((s.last_step_stats(), s.get_state()))
        s.close()
    plain = out[0][1]   # without merging: the same particles in the same order, with their scores
    score = plain["energy"] * float(cfg.co_energy) + plain["surface"] * float(cfg.co_surface)
    key, idx, _, _ = O.sort(cfg, pos)
    eligible = np.bincount(key[score[idx] < cfg.merge_criteria], minlength=len(cells))
    assert out[1][0]["n_removed"] == int((eligible // ways).sum()) * (ways - 1)
    assert out[1][0] == out[2][0]
    for f in STATE:
        assert out[1][1][f].tobytes() == out[2][1][f].tobytes(), f
