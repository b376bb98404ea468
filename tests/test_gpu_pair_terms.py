"""The force and energy pair terms where their two forms meet: warps whose
particles share one level (the short form), warps of mixed levels, list lengths
around the rounds of four, pairs at the ends of the square root's range, and
close pairs.  Accelerations and |grad c| within 1e-5 of the FP64 oracle fed the
same FP32 state, and the list path bit-identical to the stencil walk (whose
pairs always take the general form)."""
import numpy as np
import pytest

import sca2012_b200 as sph
from oracle import oracle as O
from tests._parity import check_close

pytestmark = pytest.mark.gpu

PRESETS = {2: sph.PRESET_DAM_2D, 3: sph.PRESET_DAM_3D2}


def _cloud(dim, n, levels, spread, seed):
    cfg = sph.preset(PRESETS[dim])
    cfg.use_split = cfg.use_merge = 0
    cfg.max_particle = n
    r = np.random.default_rng(seed)
    mid = np.array([float(cfg.world[a]) for a in range(dim)]) * 0.5
    pos = (mid + (r.random((n, dim)) - 0.5) * spread * float(cfg.cell_size)).astype(np.float32)
    vel = r.normal(0.0, 0.1, (n, dim)).astype(np.float32)
    level = np.full(n, levels[0], np.uint32) if len(levels) == 1 else r.integers(1, 3, n).astype(np.uint32)
    return cfg, pos, vel, level


def _step(cfg, pos, vel, level, walk):
    c = cfg.copy()
    c.walk_only = walk
    s = sph.Solver(c)
    s.set_state(dict(pos=pos, vel=vel, ev=vel, level=level))
    s.step(1)
    assert s.sync_status() == 0
    out = s.get_state()
    s.close()
    return c, out


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("levels", [(1,), (2,), (1, 2)])
@pytest.mark.parametrize("n,spread", [(2, 0.3), (5, 0.8), (37, 2.0), (130, 2.5), (1000, 4.5)])
def test_pair_terms_match_oracle_and_walk(gpu, dim, levels, n, spread):
    cfg, pos, vel, level = _cloud(dim, n, levels, spread, seed=7 * n + dim)
    c, out = _step(cfg, pos, vel, level, 0)
    _, walked = _step(cfg, pos, vel, level, 1)
    for f in ("acc", "surface", "energy", "pos", "vel"):
        assert out[f].tobytes() == walked[f].tobytes(), f
    key, idx, cs, ce = O.sort(c, pos)
    dens, press, _ = O.density(c, pos, level, idx, cs, ce)
    got = O.force(c, pos, vel, level, dens, press, idx, cs, ce)
    check_close("force", out["acc"], np.asarray(got[0])[:, :dim])


@pytest.mark.parametrize("gap", [1e-9, 1e-6, 2.1e-5, 1e-3, 0.0159, 0.0199999])
def test_single_pair(gpu, gap):
    """Two particles `gap` apart along x, around close_r2 and both kernel lengths."""
    cfg = sph.preset(sph.PRESET_DAM_3D2)
    cfg.use_split = cfg.use_merge = 0
    cfg.max_particle = 2
    x = np.float32(0.25)
    pos = np.array([[x, 0.2, 0.2], [x + np.float32(gap), 0.2, 0.2]], np.float32)
    vel = np.array([[0.1, 0, 0], [-0.1, 0.05, 0]], np.float32)
    for level in ([1, 1], [1, 2], [2, 2]):
        level = np.array(level, np.uint32)
        c, out = _step(cfg, pos, vel, level, 0)
        _, walked = _step(cfg, pos, vel, level, 1)
        assert out["acc"].tobytes() == walked["acc"].tobytes()
        key, idx, cs, ce = O.sort(c, pos)
        dens, press, _ = O.density(c, pos, level, idx, cs, ce)
        got = O.force(c, pos, vel, level, dens, press, idx, cs, ce)
        check_close("force", out["acc"], np.asarray(got[0])[:, :3])


@pytest.mark.parametrize("levels", [(1,), (1, 2)])
def test_rejected_neighbour_with_nan_velocity_adds_nothing(gpu, levels):
    """A listed neighbour outside the pair test contributes nothing, whatever
    its velocity holds: the list path keeps the walk's bits."""
    cfg, pos, vel, level = _cloud(3, 400, levels, 3.5, seed=11)
    vel[::40] = np.nan
    outs = []
    for walk in (0, 1):
        c = cfg.copy()
        c.walk_only = walk
        s = sph.Solver(c)
        s.set_state(dict(pos=pos, vel=np.zeros_like(vel), ev=vel, level=level))
        s.step(1)
        outs.append(s.get_state())
        s.close()
    assert np.isnan(outs[0]["acc"]).any() and np.isfinite(outs[0]["acc"]).all(-1).any()
    for f in ("acc", "surface", "pos", "energy"):
        assert np.array_equal(outs[0][f], outs[1][f], equal_nan=True), f
