"""Node grids of odd, even and ragged sizes: the density-grid splat against the
FP64 oracle, and marching cubes against the oracle's, cube order included.

Splat: 2 x 2 node groups (grids of an even multiple of the cells plus one node,
0.4M nodes and more) and x pairs (the others), whose nodes share a cell or do
not, and groups cut off at the upper faces.
Marching cubes: 32 x 32 tiles and 256-cube blocks with remainders, down to a
single cube; a random grid fills the blocks' triangle lists.
"""
import ctypes as C

import numpy as np
import pytest

import sca2012_b200 as sph
from oracle import mc as M
from oracle import oracle as O
from sca2012_b200 import scenes
from tests._parity import check_close

pytestmark = pytest.mark.gpu


def _cfg(dims):
    cfg = sph.preset(sph.PRESET_REF_3D2)
    cfg.use_split = cfg.use_merge = 0
    for a in range(3):
        cfg.ndens[a] = dims[a]
    cfg.max_particle = 40000
    return cfg


def _f(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


@pytest.mark.parametrize("dims", [(129, 65, 65), (64, 33, 20), (65, 34, 17), (130, 66, 9), (33, 17, 5), (2, 3, 2),
                                  (129, 65, 60), (193, 97, 65)])
def test_splat_matches_oracle(dims, gpu):
    cfg = _cfg(dims)
    cfg.grid_every = 1
    s = sph.Solver(cfg)
    s.set_state(dict(zip(("pos", "vel", "level"), scenes.ref_box_3d2(cfg))))
    s0 = s.get_state()
    s.step(1)
    assert s.sync_status() == 0
    dens = np.zeros(int(np.prod(dims)), np.float32)
    nrm = np.zeros((len(dens), 3), np.float32)
    assert s._lib.sph_density_grid(s._h, _f(dens), _f(nrm)) == 0
    st = s.get_state()
    s.close()
    key, idx, cs, ce = O.sort(cfg, s0["pos"])
    d64, _ = O.density_grid(cfg, st["pos"], s0["level"], idx, cs, ce)
    check_close(f"splat {dims}", dens, d64)


@pytest.mark.parametrize("dims", [(2, 2, 2), (33, 3, 34), (34, 35, 33), (65, 18, 32), (3, 40, 66), (97, 5, 2)])
@pytest.mark.parametrize("interpolate", [0, 1])
def test_marching_cubes_matches_oracle(dims, interpolate, gpu):
    cfg = _cfg(dims)
    cfg.mc_interpolate = interpolate
    G = int(np.prod(dims))
    cfg.max_triangles = 5 * G   # never reached
    rng = np.random.default_rng(sum(dims))
    dens = (float(cfg.iso_value) * rng.uniform(0.5, 1.5, G)).astype(np.float32)
    nrm = rng.uniform(-1, 1, (G, 3)).astype(np.float32)
    s = sph.Solver(cfg)
    bufs = [np.zeros((5 * G, 3), np.float32) for _ in range(6)]
    mv = sph.MeshView()
    mv.max_triangles = 5 * G
    for k, b in zip(("v0", "v1", "v2", "n0", "n1", "n2"), bufs):
        setattr(mv, k, _f(b))
    assert s._lib.sph_surface_from_grid(s._h, _f(dens), _f(nrm), C.byref(mv)) == 0
    s.close()
    tris, _ = M.marching_cubes(cfg, dens, nrm)
    n = int(mv.num_triangles)
    assert n == len(tris)
    ours = np.stack([b[:n] for b in bufs], 1)
    check_close(f"vertices {dims}", ours[:, :3].reshape(-1, 3), tris[:, :3].reshape(-1, 3))
    # a normal is the rounded sum of two FP32 numbers below 1 in size, halved
    np.testing.assert_allclose(ours[:, 3:], tris[:, 3:], rtol=0, atol=1e-6)
