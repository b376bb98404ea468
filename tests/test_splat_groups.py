"""The splat takes 2 x 2 nodes a thread where both nodes of every group
(2m - 1, 2m) of an axis lie in one cell: on the CPU, by the FP32 arithmetic of
the kernel's cell of a node, for the axes the rule accepts; and on the GPU at
numbers of node spacings per cell, equal and not, beyond the smallest."""
import ctypes as C

import numpy as np
import pytest

import sca2012_b200 as sph
from oracle import oracle as O
from sca2012_b200 import scenes
from tests._parity import check_close

F = np.float32


def _cells(nodes, ncell):
    """floor((v / nodes) * ncell), rounded to FP32 after each operation, clamped."""
    v = np.arange(nodes, dtype=np.int64).astype(F)
    return np.minimum(np.floor((v / F(nodes)) * F(ncell)), F(ncell - 1))


AXES = [(c, s) for s in (2, 4, 6, 10, 64) for c in list(range(1, 260)) + [511, 777, 1000, 1024, 2047, 4095, 4097, 10007]]
AXES += [((1 << 21) - 1, 2), (2097000, 2), (1398101, 2), ((1 << 20) - 1, 4), ((1 << 19) - 1, 8), (699050, 6),
         (1, (1 << 22) - 2), (3, 1398100)]


def test_groups_of_accepted_axes_lie_in_one_cell():
    for ncell, s in AXES:
        nodes = ncell * s + 1
        assert nodes <= 1 << 22 and nodes % 2 == 1
        q = _cells(nodes, ncell)
        assert np.array_equal(q[1::2], q[2::2]), (ncell, s)


def test_groups_of_other_axes_do_not():
    """What the rule refuses: an odd number of spacings per cell, and axes so
    long that rounding takes a cell's last node into the next."""
    for ncell, s in ((8, 1), (8, 3), (33, 5), ((1 << 23) - 1, 2)):
        q = _cells(ncell * s + 1, ncell)
        m = (ncell * s) // 2
        assert not np.array_equal(q[1::2][:m], q[2::2][:m])


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(257, 129, 17), (257, 129, 65), (385, 193, 9), (257, 65, 33), (129, 193, 20)])
def test_splat_groups_match_oracle(dims, gpu):
    cfg = sph.preset(sph.PRESET_REF_3D2)
    cfg.use_split = cfg.use_merge = 0
    for a in range(3):
        cfg.ndens[a] = dims[a]
    assert all((dims[a] - 1) % (2 * cfg.ncell[a]) == 0 for a in (0, 1)) and np.prod(dims) >= 4 * 5 * 128 * 148
    cfg.max_particle = 40000
    cfg.grid_every = 1
    s = sph.Solver(cfg)
    s.set_state(dict(zip(("pos", "vel", "level"), scenes.ref_box_3d2(cfg))))
    s0 = s.get_state()
    s.step(1)
    assert s.sync_status() == 0
    dens = np.zeros(int(np.prod(dims)), np.float32)
    nrm = np.zeros((len(dens), 3), np.float32)
    f = C.POINTER(C.c_float)
    assert s._lib.sph_density_grid(s._h, dens.ctypes.data_as(f), nrm.ctypes.data_as(f)) == 0
    st = s.get_state()
    s.close()
    key, idx, cs, ce = O.sort(cfg, s0["pos"])
    d64, _ = O.density_grid(cfg, st["pos"], s0["level"], idx, cs, ce)
    check_close(f"splat {dims}", dens, d64)
