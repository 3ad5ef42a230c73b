"""Two cells per thread give the bits of one cell per thread
(SIMLAB_LBM_ONE_CELL=1) on rows of whole 16-byte units: same forces, fields,
wall records and saved states, for both 2-byte storages, with and without LES
and sponges, with fused x faces (every tunnel), without any (a spinning part,
a state loaded anew), with a periodic z, and with a last tile that is nearly
empty or a single one."""
import pytest

from simlab_b200.lbm import FaceBc, Lattice, LatticeSetup, Storage, voxelize_static
from simlab_b200.shapes import sphere

from test_gpu_spin import spin_case, spin_steps

pytestmark = pytest.mark.gpu

F = FaceBc


def _tunnel(dims, storage, les, sponge, zper):
    c = [dims[0] * 0.4 + 0.3, dims[1] * 0.5 + 0.1, dims[2] * 0.5 - 0.2]
    v, t = sphere(c, 0.2 * min(dims), 3)
    st = LatticeSetup(dims=list(dims), faces=[F.VELOCITY] + [F.OPEN] * 3 + [F.PERIODIC if zper else F.OPEN] * 2, nu=1e-3,
                      smagorinsky=0.17 if les else 0.0, u_inf=[0.05, 0.004, -0.003], u_init=[0.05, 0.004, -0.003],
                      sponge=([4, 6, 3, 3] + ([0, 0] if zper else [4, 4])) if sponge else [0] * 6, sponge_tau=1.0, sponge_sigma=0.1,
                      total_pressure_inlet=True, storage=storage, center=c, debug_dump=True)
    vox = voxelize_static(v, t, list(dims))

    def go():
        with Lattice(st, vox) as lat:
            a = lat.run(41)
            blob = lat.save_state()
            lat.load_state(blob)
            return a, lat.run(8), lat.macros(), lat.records(), blob
    return go


def _spin(storage):
    st, geo = spin_case(storage)

    def go():
        with Lattice(st, geo) as lat:
            return lat.run(spin_steps(40, 0.02)), lat.macros(), lat.records()
    return go


def _check(go, monkeypatch):
    monkeypatch.delenv("SIMLAB_LBM_ONE_CELL", raising=False)
    two = go()
    monkeypatch.setenv("SIMLAB_LBM_ONE_CELL", "1")
    for a, b in zip(two, go()):
        assert (a if isinstance(a, bytes) else a.tobytes()) == (b if isinstance(b, bytes) else b.tobytes())


@pytest.mark.parametrize("storage", [Storage.FP16, Storage.BF16])
@pytest.mark.parametrize("les", [True, False])
@pytest.mark.parametrize("sponge", [True, False])
# 26 tiles of 2560 cells and 40 cells; a single tile; 15 tiles
@pytest.mark.parametrize("dims,zper", [((72, 37, 25), False), ((16, 11, 13), False), ((40, 33, 29), True)])
def test_tunnels(storage, les, sponge, dims, zper, monkeypatch):
    _check(_tunnel(dims, storage, les, sponge, zper), monkeypatch)


@pytest.mark.parametrize("storage", [Storage.FP16, Storage.BF16])
def test_large_tunnel(storage, monkeypatch):
    _check(_tunnel((256, 96, 80), storage, True, True, False), monkeypatch)


@pytest.mark.parametrize("storage", [Storage.FP16, Storage.BF16])
def test_spinning_part(storage, monkeypatch):
    _check(_spin(storage), monkeypatch)
