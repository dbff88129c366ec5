"""Several steps per launch over register-resident tiles: the default of lattices
that fit L2, at the edges of its tiles.  The default pipeline equals the
one-thread-per-node kernel bit for bit in every storage form (FP64 against the
oracle: test_gpu_parity.py and test_gpu_partial.py run on it too)."""
import numpy as np
import pytest

import harness as H
from test_gpu_stream import advance, same

pytestmark = pytest.mark.gpu

# launches of 1 to 8 steps, remainders, output steps alone and after a run
PLAN = [(1, True), (2, False), (3, True), (7, False), (8, True), (29, False), (1, False), (16, True)]


def box(rows, cols):
    t = np.full((rows, cols), H.FLUID, dtype=np.uint8)
    t[0, :] = t[-1, :] = t[:, 0] = t[:, -1] = H.BOUNDARY
    t[0, 1:-1] = H.INLET
    return t


@pytest.mark.parametrize("rows,cols", [(3, 3), (3, 700), (700, 3), (19, 21), (20, 40), (21, 64), (26, 27), (53, 33), (129, 64),
                                       (181, 97), (113, 290)])
@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32s", "f16s"])
def test_tile_edges(rows, cols, storage):
    lists = H.classify(box(rows, cols))
    p = H.Params(tau=0.8)
    table = H.open_values(lists, "lidramp:0.1:0.05", "const:0:0", 1 + sum(k for k, _ in PLAN))
    act = H.active_mask(lists)
    same(advance(lists, p, table, storage, None, PLAN), advance(lists, p, table, storage, -1, PLAN), act)


@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32s", "f16s"])
def test_obstacles_dead_nodes_and_open_corners(storage):
    t = H.porous_types(131, 190, fraction=0.25, rmin=2, rmax=5, seed=3)
    t[:, 0] = H.INLET
    t[60, 90] = t[61, 90] = H.SOLID
    lists = H.classify(t)
    p = H.Params.trt_magic(0.7, outlet_bc=H.BC_ZH_PRESSURE)
    table = H.open_values(lists, "const:0.02:0.005", "pressure", 1)
    act = H.active_mask(lists)
    same(advance(lists, p, table, storage, None, PLAN), advance(lists, p, table, storage, -1, PLAN), act)


def test_partially_saturated_tiles():
    """Obstacles with weights across tile borders, columns and strips."""
    t = H.porous_types(150, 260, fraction=0.25, rmin=2, rmax=6, seed=8)
    lists = H.classify(t)
    b = np.random.default_rng(3).uniform(0.0, 1.0, len(lists.obstacle))
    p = H.Params.trt_magic(0.6, outlet_bc=H.BC_ZH_PRESSURE, obstacle_bc=1, ps_tau=0.7, obstacle_b=b)
    table = H.open_values(lists, "const:0.03:0", "pressure", 1)
    act = H.active_mask(lists)
    a = advance(lists, p, table, 0, None, PLAN)
    same(a, advance(lists, p, table, 0, -1, PLAN), act)
    ref = H.run_oracle(lists, p, a[0], table)
    np.testing.assert_array_equal(a[2][:, act], ref["post"][:, act])


def test_tuner_keeps_the_default_mode_or_a_kernel():
    """Tuning a small lattice times its default way of stepping too; the run
    stays the run of that many ordinary steps."""
    lists = H.classify(box(80, 90))
    p = H.Params(tau=0.7)
    table = H.open_values(lists, "const:0.05:0", "const:0:0", 1)
    from test_gpu_parity import make_gpu

    outs = []
    for tune in (True, False):
        with make_gpu(lists, p, pipeline=None if tune else -1) as g:
            g.set_open_values(table, 0)
            g.init()
            if tune:
                g.tune_pipeline(16)
                steps = g.t + 30
            g.step(steps - g.t, macro=True)
            outs.append((g.t, g.post_collision(), g.macro()))
    assert outs[0][0] == outs[1][0]
    act = H.active_mask(lists)
    np.testing.assert_array_equal(outs[0][1][:, act], outs[1][1][:, act])
    np.testing.assert_array_equal(outs[0][2][1], outs[1][2][1])
