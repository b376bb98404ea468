"""States uploaded as the caller holds them and unpacked on the device: every
field comes back as it went in, absent ones as zeros, at sizes around a block,
on a fresh handle and over an earlier, larger state, and particles added after a
step leave the ones before them with their outputs."""
import numpy as np
import pytest

import sca2012_b200 as sph

pytestmark = pytest.mark.gpu

VEC = ("pos", "vel", "ev", "acc")
SCALAR = ("dens", "press", "energy", "surface")


def _solver(dim, cap):
    cfg = sph.preset(sph.PRESET_DAM_2D if dim == 2 else sph.PRESET_DAM_3D2)
    cfg.use_split = cfg.use_merge = 0
    cfg.max_particle = cap
    return sph.Solver(cfg)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [0, 1, 2, 255, 256, 257, 4096])
def test_state_round_trip(gpu, dim, n):
    r = np.random.default_rng(n + dim)
    s = _solver(dim, 5000)
    full = {k: r.random((5000, dim), np.float32) * 0.5 for k in VEC}
    full.update({k: r.random(5000, np.float32) for k in SCALAR})
    full.update(level=r.integers(1, 3, 5000).astype(np.uint32), interior=r.integers(0, 9, 5000).astype(np.uint32),
                sibling=r.integers(0, 5000, 5000).astype(np.uint32))
    s.set_state(full)
    for keys in (VEC + SCALAR + ("level", "interior", "sibling"), ("pos", "level"), ("pos", "vel", "level", "press")):
        part = {k: full[k][:n] for k in keys}
        s.set_state(part)
        assert s.num_particles() == n
        got = s.get_state()
        for k in VEC + SCALAR + ("level", "interior"):
            want = part[k] if k in keys else np.zeros_like(full[k][:n])
            assert got[k].tobytes() == want.tobytes(), (keys, k)
        want = part["sibling"] if "sibling" in keys else np.full(n, sph.NO_SIBLING, np.uint32)
        assert got["sibling"].tobytes() == want.tobytes()
    s.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_added_particles_keep_the_others(gpu, dim):
    r = np.random.default_rng(dim)
    s = _solver(dim, 1000)
    pos = (0.1 + 0.3 * r.random((600, dim))).astype(np.float32)
    s.add_particles(pos[:300], np.zeros((300, dim)), np.ones(300, np.uint32))
    s.step(1)
    before = s.get_state()
    s.step(0)
    vel = r.random((300, dim), np.float32)
    s.add_particles(pos[300:], vel, np.full(300, 2, np.uint32))
    after = s.get_state()
    for k in VEC + SCALAR + ("level",):
        assert after[k][:300].tobytes() == before[k].tobytes(), k
    assert after["pos"][300:].tobytes() == pos[300:].tobytes() and after["vel"][300:].tobytes() == vel.tobytes()
    assert not after["ev"][300:].any() and not after["dens"][300:].any() and (after["level"][300:] == 2).all()
    s.step(1)
    assert s.sync_status() == 0 and s.num_particles() == 600
    s.close()
