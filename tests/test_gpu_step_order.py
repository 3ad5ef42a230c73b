"""A step whose wall and face cells share a grid, or whose wall kernel runs on
a second stream beside the bulk, gives the bits of the step whose kernels run
one by one (as they do when they are timed one by one), over many steps."""
import numpy as np
import pytest

from simlab_b200.lbm import Collision, FaceBc, Lattice, LatticeSetup, Storage, voxelize_static
from simlab_b200.shapes import cuboid

from helpers import ball, momentum_setup

pytestmark = pytest.mark.gpu


def _same(setup, vox, steps=96):
    one, timed = Lattice(setup, vox), Lattice(setup, vox)
    timed.profile(1)
    for n in (1, steps, 7):
        a, b = one.run(n), timed.run(n)
        assert a.tobytes() == b.tobytes()
    assert one.macros().tobytes() == timed.macros().tobytes()
    assert one.records().tobytes() == timed.records().tobytes()
    return a


def _near(vox, dims):
    c = vox.walls["cell"].astype(np.int64)
    q = np.stack([c % dims[0], c // dims[0] % dims[1], c // (dims[0] * dims[1])])
    return int(min(q.min(), min((dims[k] - 1 - q[k]).min() for k in range(3))))


@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP16, Storage.BF16, Storage.FP64])
@pytest.mark.parametrize("collision", [Collision.REGULARIZED, Collision.BGK])
@pytest.mark.parametrize("dims,lo,near", [((64, 40, 36), 3.6, 3), ((64, 40, 36), 2.6, 2), ((61, 39, 37), 3.6, 3)])
def test_walls_and_faces_in_one_grid(storage, collision, dims, lo, near):
    # a block whose nearest wall cells are three cells from the y face (one
    # grid takes walls and faces) or two (wall kernel after the face kernel)
    F = FaceBc
    v, t = cuboid([20.3, lo, 10.4], [31.2, 15.7, 24.6])
    vox = voxelize_static(v, t, list(dims))
    assert _near(vox, dims) == near
    st = LatticeSetup(dims=list(dims), faces=[F.VELOCITY] + [F.OPEN] * 3 + [F.FREE_SLIP] * 2, nu=2e-3, collision=collision,
                      smagorinsky=0.17 if collision == Collision.REGULARIZED else 0.0, u_inf=[0.05, 0.004, -0.003],
                      u_init=[0.05, 0.004, -0.003], sponge=[4, 8, 0, 4, 4, 4], sponge_tau=1.0, sponge_sigma=0.1,
                      total_pressure_inlet=True, storage=storage, center=[25.0, 9.0, 17.0], debug_dump=True)
    assert np.abs(_same(st, vox)).max() > 0


@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP16, Storage.FP64])
def test_walls_beside_the_bulk_of_a_periodic_box(storage):
    st = momentum_setup(33, 0.02, 0.03, 1e-6, [FaceBc.PERIODIC] * 6, storage)
    assert np.abs(_same(st, ball(33, 7.0))).max() > 0
