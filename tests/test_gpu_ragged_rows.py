"""The staged D3Q19 bulk kernel on rows that are no whole number of 16-byte
units gives the direct kernel's bits: same forces, fields and wall records,
for every storage with stochastic rounding or none, at row lengths of every
kind of misalignment, with a last tile that is nearly empty.
SIMLAB_LBM_NO_TMA=1 selects the direct kernel."""
import numpy as np
import pytest

from simlab_b200.lbm import FaceBc, Lattice, LatticeSetup, Storage, voxelize_static
from simlab_b200.shapes import sphere

pytestmark = pytest.mark.gpu


def _run(dims, storage, les):
    F = FaceBc
    c = [dims[0] * 0.3 + 0.2, dims[1] * 0.5 - 0.1, dims[2] * 0.5 + 0.3]
    v, t = sphere(c, 7.4, 3)
    st = LatticeSetup(dims=list(dims), faces=[F.VELOCITY] + [F.OPEN] * 5, nu=1e-3, smagorinsky=0.17 if les else 0.0, u_inf=[0.05, 0.004, -0.003],
                      u_init=[0.05, 0.004, -0.003], sponge=[4, 8, 4, 4, 4, 4], sponge_tau=1.0, sponge_sigma=0.1, total_pressure_inlet=True,
                      storage=storage, center=c, debug_dump=True)
    with Lattice(st, voxelize_static(v, t, list(dims))) as lat:
        f = lat.run(7)
        return f, lat.macros(), lat.records()


@pytest.mark.parametrize("storage", [Storage.FP32, Storage.FP16, Storage.BF16, Storage.FP64])
@pytest.mark.parametrize("dims,les", [((161, 81, 79), True), ((162, 80, 81), False), ((163, 78, 80), True), ((167, 77, 79), True)])
def test_ragged_rows_match_the_direct_kernel(storage, dims, les, monkeypatch):
    monkeypatch.delenv("SIMLAB_LBM_NO_TMA", raising=False)
    staged = _run(dims, storage, les)
    monkeypatch.setenv("SIMLAB_LBM_NO_TMA", "1")
    direct = _run(dims, storage, les)
    if storage == Storage.FP64:
        assert np.abs(staged[0] - direct[0]).max() <= 1e-12 * np.abs(direct[0]).max()
        m = np.isfinite(direct[1])
        assert (np.isfinite(staged[1]) == m).all()
        assert np.abs(staged[1][m] - direct[1][m]).max() <= 2.5e-7  # float32 fields of order 1
        return
    for a, b in zip(staged, direct):
        assert a.tobytes() == b.tobytes()
