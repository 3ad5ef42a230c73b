"""Rows that are no whole number of 16-byte units, over the forms that the
staged kernel's ragged variant takes or leaves to the direct kernel: the same
forces, fields and wall records, bit for bit, with the staged kernel allowed
and with SIMLAB_LBM_NO_TMA=1, which selects the direct one."""
import pytest

from simlab_b200.lbm import Collision, FaceBc, Lattice, LatticeSetup, Storage, voxelize_static
from simlab_b200.shapes import sphere

pytestmark = pytest.mark.gpu

F = FaceBc
OPEN = [F.VELOCITY] + [F.OPEN] * 5
FORMS = {
    "les_sponge": dict(smagorinsky=0.17, sponge=[4, 6, 3, 3, 4, 4], sponge_tau=1.0, sponge_sigma=0.1),
    "plain": dict(),
    "bgk": dict(collision=Collision.BGK, faces=[F.VELOCITY, F.OPEN] + [F.FREE_SLIP] * 4, total_pressure_inlet=False),
    "force": dict(body_force=[1e-5, 2e-6, 0.0]),
    "absorb_velocity": dict(smagorinsky=0.1, sponge=[4, 6, 3, 3, 4, 4], sponge_tau=1.0, sponge_sigma=0.1, absorb_velocity=True),
    "periodic_z": dict(smagorinsky=0.17, faces=[F.VELOCITY] + [F.OPEN] * 3 + [F.PERIODIC] * 2),
}


def _run(dims, storage, form):
    c = [dims[0] * 0.4 + 0.3, dims[1] * 0.5 + 0.1, dims[2] * 0.5 - 0.2]
    v, t = sphere(c, 5.3, 3)
    kw = dict(faces=OPEN, total_pressure_inlet=True)
    kw.update(FORMS[form])
    st = LatticeSetup(dims=list(dims), nu=2e-3, u_inf=[0.05, 0.004, -0.003], u_init=[0.05, 0.004, -0.003], storage=storage, center=c,
                      debug_dump=True, **kw)
    with Lattice(st, voxelize_static(v, t, list(dims))) as lat:
        return lat.run(21), lat.macros(), lat.records()


def _check(dims, storage, form, monkeypatch):
    monkeypatch.delenv("SIMLAB_LBM_NO_TMA", raising=False)
    allowed = _run(dims, storage, form)
    monkeypatch.setenv("SIMLAB_LBM_NO_TMA", "1")
    for a, b in zip(allowed, _run(dims, storage, form)):
        assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("form", sorted(FORMS))
def test_fp64(form, monkeypatch):
    _check((61, 43, 37), Storage.FP64, form, monkeypatch)


@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP16])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_every_form_above_the_size_of_the_staged_kernel(storage, form, monkeypatch):
    _check((163, 79, 80), storage, form, monkeypatch)


@pytest.mark.parametrize("storage", [Storage.FP16, Storage.BF16])
@pytest.mark.parametrize("nx", [164, 165, 166])  # 4, 5 and 6 of the 8 elements of a unit
@pytest.mark.parametrize("form", ["les_sponge", "plain"])
def test_two_byte_rows(storage, nx, form, monkeypatch):
    _check((nx, 66, 65), storage, form, monkeypatch)


@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP16, Storage.BF16])
@pytest.mark.parametrize("dims", [(125, 71, 57), (113, 67, 67), (1501, 19, 19)])  # about the smallest that are staged: 505,875, 507,257, 541,861 cells
@pytest.mark.parametrize("form", ["les_sponge", "plain"])
def test_smallest_staged(storage, dims, form, monkeypatch):
    _check(dims, storage, form, monkeypatch)
