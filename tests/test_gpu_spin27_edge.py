"""A spinning part on the D3Q27 lattice that sweeps the layer next to the
outermost one: its re-voxelizer reads whole states of face cells (one level)
or ghost cells (two), which those cells otherwise store only in part.  Against
the CPU oracle with the bounds of a part in the middle."""
import numpy as np
import pytest

from oracle import OracleMulti
from simlab_b200.lbm import SpinGeometry, Storage, voxelize_spin
from simlab_b200.mlattice import MultiLattice

from helpers import rel_l2
from test_gpu_spin import spin_steps
from test_gpu_spin27 import small_paddle, spin27_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP64])
def test_sweeping_the_layer_next_to_the_outermost(storage, levels):
    s, geo = spin27_case(storage, levels)
    s.center[1] = 7.2  # the blades (radius 6.3) pass y = 1
    v, t = small_paddle()
    c = s.center
    geo = SpinGeometry(vox=voxelize_spin(v, t, [0.0, 0.0, 1.0], 0.125), box_lo=[int(c[0]) - 8, 1, int(c[2]) - 4], box_n=[17, 14, 9])
    g, o = MultiLattice(s, geo), OracleMulti(s, geo, real64=storage == Storage.FP64)
    steps = spin_steps(60, 0.025, -2.3)
    # a cell at y = 1 is solid on the way and uncovered again
    solid = []
    hg, ho = [], []
    for k in range(0, 60, 6):
        hg.append(g.run(steps[k:k + 6]))
        ho.append(o.run(steps[k:k + 6]))
        m = g.macros(levels - 1)[:, 0].reshape(s.dims(levels - 1)[::-1])
        solid.append(int(np.isnan(m[geo.box_lo[2]:geo.box_lo[2] + 9, 1, geo.box_lo[0]:geo.box_lo[0] + 17]).sum()))
    assert max(solid) > 0 and solid[-1] < max(solid)
    hg, ho = np.concatenate(hg), np.concatenate(ho)
    rg, ro = g.records().reshape(-1, 24), o.records().reshape(-1, 24)
    assert np.array_equal(rg[:, :15], ro[:, :15])
    for l in range(levels):
        mg, mo = g.macros(l), o.macros(l)
        assert np.array_equal(np.isnan(mg[:, 0]), np.isnan(mo[:, 0])), l
        assert rel_l2(mg[:, 1:4], mo[:, 1:4]) <= (1e-5 if storage == Storage.FP32 else 1e-6), l
    assert np.max(np.abs(hg - ho)) <= (1e-5 if storage == Storage.FP32 else 1e-9) * np.max(np.abs(ho))
