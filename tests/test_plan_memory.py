"""The plan's device memory counts what a spinning part's re-voxelizer keeps,
so that a part planned within a memory budget fits it."""
import numpy as np
import pytest

from simlab_b200 import lbm
from simlab_b200 import tunnel as T

from test_tunnel import rotating_sphere_case


@pytest.mark.parametrize("cells", [16, 48])
def test_spinning_part_counts_its_box(cells):
    cfg, m = rotating_sphere_case(1.0, cells, 6.0)
    p = T.plan(cfg, m, 1e-3, T.SolverOptions())
    assert p.spin
    box = int(np.prod(p.box_n))
    n = int(np.prod(p.dims))
    d = p.dims
    # FP32 populations and flags, faces, and the fixed part
    rest = n * (19 * 4 + 4) + 88 * (d[0] * d[1] + d[1] * d[2] + d[0] * d[2]) + (64 << 20)
    # per box cell: a record of 40 words, two sets of 9 links x 3 words; the solid bytes of box and halo
    want = box * (160 + 216) + int(np.prod([k + 2 for k in p.box_n]))
    assert p.storage == int(lbm.Storage.FP32) and p.memory == rest + want
    # a budget that holds everything but the scratch does not take FP32
    assert T.plan(cfg, m, 1e-3, T.SolverOptions(memory_budget=p.memory)).storage == int(lbm.Storage.FP32)
    assert T.plan(cfg, m, 1e-3, T.SolverOptions(memory_budget=p.memory - 1)).storage == int(lbm.Storage.FP16)
