"""Force and moment of a batch longer than the wall kernel's kept partials
(16 MB: fewer steps the more records there are): the batch equals the same
steps in batches that fit, as does the batch after it."""
import numpy as np
import pytest

from simlab_b200.lbm import FaceBc, Lattice, LatticeSetup, SpinGeometry, Storage, voxelize_spin
from simlab_b200.mlattice import MultiLattice, MultiSetup

from test_gpu_spin import paddle, spin_steps

pytestmark = pytest.mark.gpu


def _spin(n):
    v, t = paddle()
    return SpinGeometry(vox=voxelize_spin(v, t, [0.0, 0.0, 1.0], 0.25), box_lo=[4] * 3, box_n=[n] * 3)


def _ring(records, block, most):
    return min((16 << 20) // (-(-records // block) * 64), most)


def _in_pieces(lat, steps, pieces):
    out, k = [], 0
    for n in pieces:
        out.append(lat.run(steps[k:k + n]))
        k += n
    assert k == len(steps)
    return np.concatenate(out)


def _check(make, total, ring):
    steps = spin_steps(total + 20, 0.01)
    half = ring // 2
    whole = _in_pieces(make(), steps, [total, 20])
    assert whole.tobytes() == _in_pieces(make(), steps, [half] * (total // half) + [total % half, 20]).tobytes()
    assert np.abs(whole).max(axis=1).min() > 0.0  # every step has a force


def test_d3q19():
    n = 46
    ring = _ring(n ** 3, 64, 512)
    assert 100 < ring < 200
    F = FaceBc
    st = LatticeSetup(dims=[n + 8] * 3, faces=[F.VELOCITY] + [F.OPEN] * 5, nu=0.02, u_inf=[0.03, 0, 0], u_init=[0.03, 0, 0],
                      storage=Storage.FP32, center=[26.3, 26.4, 26.1])
    # a batch of more steps than one readback (512), no multiple of the ring
    _check(lambda: Lattice(st, _spin(n)), 530, ring)


def test_d3q27():
    n = 52
    ring = _ring(n ** 3, 256, 1024)
    assert 400 < ring < 500
    F = FaceBc
    s = MultiSetup(dims0=[n + 8] * 3, faces=[F.VELOCITY] + [F.OPEN] * 5, nu0=0.02, u_inf=[0.03, 0, 0], u_init=[0.03, 0, 0],
                   total_pressure_inlet=True, storage=Storage.FP32)
    s.center = [29.3, 29.4, 29.1]
    _check(lambda: MultiLattice(s, _spin(n)), 1100, ring)


@pytest.mark.parametrize("mode", [1, 2])
def test_the_force_sums_are_counted_among_the_launches(mode):
    n = 46
    F = FaceBc
    st = LatticeSetup(dims=[n + 8] * 3, faces=[F.VELOCITY] + [F.OPEN] * 5, nu=0.02, u_inf=[0.03, 0, 0], u_init=[0.03, 0, 0],
                      storage=Storage.FP32, center=[26.3, 26.4, 26.1])
    with Lattice(st, _spin(n)) as lat:
        ring = _ring(n ** 3, 64, 512)
        lat.run(spin_steps(1, 0.01))
        lat.profile(mode)
        lat.run(spin_steps(ring + 3, 0.01))
        # per step: triangle scatter, re-voxelizer, faces, walls, bulk; one sum per ring begun
        assert lat.kernel_times()["launches"] == 5 * (ring + 3) + 2
