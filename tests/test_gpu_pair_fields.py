"""The colour-field gradient and the wavelet energy of clouds of one level and
of mixed levels against the FP64 oracle (their list and walk forms share the
code of the terms, so agreeing with each other shows nothing of it).

|grad c| by the tolerance of every parity check.  Energy, m/2 |T|^2 with T the
wavelet-weighted mean of at most n velocities over sqrt(h): numerator and
denominator are FP32 sums of n terms whose weights have one sign, each weight
within 24 roundings u = 2^-24, so |dT| <= (2 n + 48) u max|v| / sqrt(h) and
|de| <= m (|T| |dT| + |dT|^2)."""
import numpy as np
import pytest

import sca2012_b200 as sph
from oracle import oracle as O
from tests._parity import check_close

pytestmark = pytest.mark.gpu

PRESETS = {2: sph.PRESET_DAM_2D, 3: sph.PRESET_DAM_3D2}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("levels", [(1,), (2,), (1, 2)])
@pytest.mark.parametrize("n,spread", [(2, 0.3), (5, 0.8), (37, 2.0), (130, 2.5), (1000, 4.5)])
def test_surface_and_energy_match_oracle(gpu, dim, levels, n, spread):
    cfg = sph.preset(PRESETS[dim])
    cfg.use_split = cfg.use_merge = 0
    cfg.max_particle = n
    r = np.random.default_rng(3 * n + dim)
    mid = np.array([float(cfg.world[a]) for a in range(dim)]) * 0.5
    pos = (mid + (r.random((n, dim)) - 0.5) * spread * float(cfg.cell_size)).astype(np.float32)
    vel = r.normal(0.0, 0.1, (n, dim)).astype(np.float32)
    level = np.full(n, levels[0], np.uint32) if len(levels) == 1 else r.integers(1, 3, n).astype(np.uint32)
    s = sph.Solver(cfg)
    s.set_debug(True)
    s.set_state(dict(pos=pos, vel=vel, ev=vel, level=level))
    s.step(1)
    assert s.sync_status() == 0
    out, dbg = s.get_state(), s.get_debug()
    s.close()
    key, idx, cs, ce = O.sort(cfg, pos)
    dens, press, nbr = O.density(cfg, pos, level, idx, cs, ce)
    _, surf, _ = O.force(cfg, pos, vel, level, dens, press, idx, cs, ce)
    check_close("surface |grad c|", out["surface"], surf)
    e64, tv = O.energy(cfg, out["pos"], out["vel"], level, idx, cs, ce)
    assert np.array_equal(np.isnan(out["energy"]), np.isnan(e64))
    has = ~np.isnan(e64)
    mass = np.array([float(cfg.mass[0]), float(cfg.mass[1])])[level - 1] if cfg.energy_mass_weight else np.ones(n)
    h = min(float(cfg.kernel[0]), float(cfg.kernel[1]))
    dt = (2.0 * n + 48.0) * 2.0 ** -24 * np.abs(out["vel"].astype(np.float64)).max() / h ** 0.5
    bound = mass * (np.linalg.norm(tv, axis=1) * dt + dt * dt) + 4 * 2.0 ** -24 * np.abs(e64)
    assert (np.abs(out["energy"] - e64)[has] <= bound[has]).all()
    assert (np.abs(dbg["trans_vel"] - tv)[has] <= dt).all()
    assert has.any()
