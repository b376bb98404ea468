"""The density walk at the sizes where its staging can go wrong: particle
counts around a warp's 32 slots and a block's 128, stencil rows longer than
the 64 staged slots, buffers that fill up inside a row, candidate lists that
overflow, both levels, and every launch shape.  Neighbour counts are exact and
densities within 1e-5 of the FP64 oracle; the force pass over the recorded
lists gives the bits of the force pass that walks the stencil itself."""
import numpy as np
import pytest

import sca2012_b200 as sph
from oracle import oracle as O
from tests._parity import check_close

pytestmark = pytest.mark.gpu


def _points(n, dim, spread, seed):
    """n points around the middle of the box, `spread` cells wide (dense when small)."""
    cfg = sph.preset(sph.PRESET_DAM_2D if dim == 2 else sph.PRESET_DAM_3D2)
    r = np.random.default_rng(seed)
    mid = np.array([float(cfg.world[a]) for a in range(dim)]) * 0.5
    pos = (mid + (r.random((n, dim)) - 0.5) * spread * float(cfg.cell_size)).astype(np.float32)
    return cfg, pos, r.integers(1, 3, n).astype(np.uint32)


def _step(cfg, pos, level, walk_only=0, shape=None):
    c = cfg.copy()
    c.use_split = c.use_merge = 0
    c.max_particle = len(pos)
    c.walk_only = walk_only
    s = sph.Solver(c)
    if shape:
        t = s.get_tuning()
        block, bpsm = list(t["block"]), list(t["blocks_per_sm"])
        block[3], bpsm[3] = shape
        s.set_tuning(block, bpsm)
    s.set_state(dict(pos=pos, vel=np.zeros_like(pos), level=level))
    s.step(1)
    assert s.sync_status() == 0
    out, dbg = s.get_state(), s.get_debug()
    s.close()
    return c, out, dbg


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,spread", [(1, 1.0), (2, 0.5), (31, 2.0), (32, 2.0), (33, 3.0), (65, 1.0), (127, 4.0),
                                      (129, 6.0), (700, 1.5), (2000, 3.0), (3001, 9.0)])
def test_density_walk_matches_oracle(gpu, dim, n, spread):
    cfg, pos, level = _points(n, dim, spread, seed=n + dim)
    c, out, dbg = _step(cfg, pos, level)
    key, idx, cs, ce = O.sort(c, pos)
    dens, _, nbr = O.density(c, pos, level, idx, cs, ce)
    assert np.array_equal(dbg["nbr_count"], nbr)
    check_close("density", out["dens"], dens)
    _, walked, _ = _step(cfg, pos, level, walk_only=1)
    for f in ("dens", "acc", "surface", "pos", "energy"):
        assert out[f].tobytes() == walked[f].tobytes(), f


@pytest.mark.parametrize("shape", [(128, 2), (256, 8), (512, 4), (512, 64)])
def test_density_walk_shapes_agree(gpu, shape):
    cfg, pos, level = _points(5003, 3, 12.0, seed=9)
    _, a, da = _step(cfg, pos, level)
    _, b, db = _step(cfg, pos, level, shape=shape)
    assert np.array_equal(da["nbr_count"], db["nbr_count"])
    for f in ("dens", "acc", "energy"):
        assert a[f].tobytes() == b[f].tobytes(), f
