"""The tile kernel at the edges of its tiles in the shapes that run it (asserted),
FP16 lattices of 8000 nodes and more and partially saturated obstacles among
them: the bits of one step per launch."""
import numpy as np
import pytest

import harness as H
from test_gpu_parity import make_gpu
from test_gpu_stream import advance, same
from test_gpu_tile import PLAN, box

pytestmark = pytest.mark.gpu


def in_tiles(lists, p, storage):
    with make_gpu(lists, p, storage=storage) as g:
        return g.run_kernel(50)[0] == 16


# tiles store up to 22, 56 or 120 rows and 26 columns
SHAPES = [(3, 3, 0), (700, 3, 0), (20, 40, 0), (26, 27, 0), (113, 290, 0), (1492, 43, 0),
          (3, 3, 1), (700, 3, 1), (57, 33, 1), (181, 97, 1), (113, 290, 1), (50, 3700, 1),
          (2800, 3, 2), (4001, 5, 2), (1700, 7, 2), (112, 73, 2), (113, 72, 2), (121, 70, 2), (240, 36, 2), (241, 290, 2),
          (7, 3800, 2), (121, 1900, 2), (480, 800, 2)]


@pytest.mark.parametrize("rows,cols,storage", SHAPES)
def test_edges(rows, cols, storage):
    lists = H.classify(box(rows, cols))
    p = H.Params.trt_magic(0.7)
    assert in_tiles(lists, p, storage)
    table = H.open_values(lists, "lidramp:0.1:0.05", "const:0:0", 1 + sum(k for k, _ in PLAN))
    act = H.active_mask(lists)
    same(advance(lists, p, table, storage, None, PLAN), advance(lists, p, table, storage, -1, PLAN), act)


@pytest.mark.parametrize("rows,cols", [(118, 130), (120, 160), (97, 300)])
def test_obstacles_and_side_openings_in_fp16(rows, cols):
    lists = H.classify(H.porous_types(rows, cols, fraction=0.25, rmin=2, rmax=5, seed=3))
    p = H.Params(tau=0.8, outlet_bc=H.BC_ZH_PRESSURE)
    with make_gpu(lists, p, storage=2) as g:
        assert g.run_kernel(8)[0] == 16
    table = H.open_values(lists, "const:0.02:0.005", "pressure", 1)
    act = H.active_mask(lists)
    same(advance(lists, p, table, 2, None, PLAN), advance(lists, p, table, 2, -1, PLAN), act)


@pytest.mark.parametrize("rows,cols", [(60, 65), (53, 230), (120, 230)])
def test_partially_saturated(rows, cols):
    lists = H.classify(H.porous_types(rows, cols, fraction=0.25, rmin=2, rmax=6, seed=8))
    b = np.random.default_rng(3).uniform(0.0, 1.0, len(lists.obstacle))
    p = H.Params.trt_magic(0.6, outlet_bc=H.BC_ZH_PRESSURE, obstacle_bc=1, ps_tau=0.7, obstacle_b=b)
    assert in_tiles(lists, p, 0)
    table = H.open_values(lists, "const:0.03:0", "pressure", 1)
    act = H.active_mask(lists)
    a = advance(lists, p, table, 0, None, PLAN)
    same(a, advance(lists, p, table, 0, -1, PLAN), act)
    ref = H.run_oracle(lists, p, a[0], table)
    np.testing.assert_array_equal(a[2][:, act], ref["post"][:, act])
