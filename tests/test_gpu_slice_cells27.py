"""Slice pixels of a refined lattice: each takes its density and velocity from
the updated fluid cell of the finest level whose interior holds it, never from
a face, ghost or restricted cell (which store only the populations that are
read from them), and pixels outside every interior stay empty."""
import numpy as np
import pytest

from simlab_b200.lbm import FaceBc, Probes, SliceDef, Storage, steps_array, voxelize_static
from simlab_b200.mlattice import LevelBox, MultiLattice, MultiSetup
from simlab_b200.shapes import sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pixels_come_from_updated_cells(axis):
    F = FaceBc
    s = MultiSetup(dims0=[26, 20, 22], faces=[F.VELOCITY] + [F.OPEN] * 5, nu0=0.02, u_inf=[0.05, 0.004, -0.003], u_init=[0.05, 0.004, -0.003],
                   total_pressure_inlet=True, storage=Storage.FP32, debug_dump=True,
                   boxes=[LevelBox(lo=[5, 4, 4], n=[15, 12, 13]), LevelBox(lo=[6, 5, 6], n=[15, 12, 11])])
    org, scale = [np.zeros(3)], [4.0]
    for b in s.boxes:
        org.append(org[-1] + np.asarray(b.lo) * scale[-1])
        scale.append(scale[-1] / 2)
    s.center = [14.3, 11.4, 10.2]  # finest cells
    v, t = sphere(s.center, 4.3, 3)
    a, b = [(1, 2), (0, 2), (0, 1)][axis]
    ext = [4 * (d - 1) + 1 for d in s.dims0]  # the lattice in finest cells
    origin = [0, 0, 0]  # slices start at the coarsest level's corner, in finest cells
    origin[axis] = int(org[2][axis] + s.center[axis])  # through the part
    unit = np.eye(3, dtype=int)
    pr = Probes(slices=[SliceDef(origin=origin, u=list(unit[a]), v=list(unit[b]), nu=ext[a], nv=ext[b])])
    with MultiLattice(s, voxelize_static(v, t, list(s.dims(2)), 27), pr) as lat:
        st = steps_array(8)
        st["sample"][-1] = 1
        lat.run(st)
        got = lat.slice_means().reshape(ext[b], ext[a], 4)
        mac = [lat.macros(l).reshape(*s.dims(l)[::-1], 4) for l in range(3)]
    want = np.full(got.shape, np.nan, dtype=np.float32)
    for iv in range(ext[b]):
        for iu in range(ext[a]):
            pt = np.asarray(origin) + iu * unit[a] + iv * unit[b]
            for l in (2, 1, 0):
                x = np.floor((pt - org[l]) / scale[l] + 0.5).astype(int)
                q = 1 if l == 0 else 2
                if all(q <= x[k] <= s.dims(l)[k] - 1 - q for k in range(3)):
                    want[iv, iu] = mac[l][x[2], x[1], x[0]]
                    break
    assert np.isfinite(want).mean() > 0.5
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    m = np.isfinite(want)
    # one sample in FP32 against the same FP32 expression: a few roundings of values of order 1
    assert np.abs(got[m] - want[m]).max() <= 1e-6
