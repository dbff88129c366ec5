"""The streaming two-step kernel (pipelines 3, 4 and 5, and the longer runs of
large lattices on their default pipeline) at the edges of its strips and chunks.

FP64 equals the oracle bit for bit; the shifted forms equal the
one-thread-per-node kernel bit for bit."""
import numpy as np
import pytest

import harness as H
from test_gpu_parity import make_gpu, pressure_table

pytestmark = pytest.mark.gpu


def advance(lists, p, table, storage, pipeline, plan):
    with make_gpu(lists, p, storage=storage, table_rows=table.shape[0], pipeline=pipeline) as g:
        g.set_open_values(pressure_table(table, lists, p), 0)
        g.init()
        for k, macro in plan:
            g.step(k, macro=macro)
        g.check_numerics()
        return g.t, g.populations(), g.post_collision(), g.macro()


def same(a, b, act):
    assert a[0] == b[0]
    np.testing.assert_array_equal(a[1][:, act], b[1][:, act])
    np.testing.assert_array_equal(a[2][:, act], b[2][:, act])
    for x, y in zip(a[3], b[3]):
        np.testing.assert_array_equal(x, y)


# a strip stores 28 / 60 rows in FP64, 56 / 120 in FP32, 112 / 240 in FP16;
# narrow lattices have fewer columns than a chunk plus its halo
@pytest.mark.parametrize("rows,cols", [(3, 3), (4, 9), (27, 5), (28, 33), (29, 40), (57, 64), (61, 7), (113, 70), (241, 36)])
@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32s", "f16s"])
def test_strip_edges(rows, cols, storage):
    t = H.cavity_types(max(rows, cols))[:rows, :cols].copy()
    t[-1, :] = t[:, -1] = H.BOUNDARY
    lists = H.classify(t)
    p = H.Params.trt_magic(0.6)
    plan = [(1, False), (2, False), (7, True), (33, False), (40, True)]
    steps = 1 + sum(k for k, _ in plan)
    table = H.open_values(lists, "lidramp:0.1:0.05", "const:0:0", steps)
    act = H.active_mask(lists)
    ref = advance(lists, p, table, storage, -1, plan)
    for pipeline in (3, 4, 5):
        same(advance(lists, p, table, storage, pipeline, plan), ref, act)
    if storage == 0:
        o = H.run_oracle(lists, p, steps, table)
        np.testing.assert_array_equal(ref[2][:, act], o["post"][:, act])


@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32s", "f16s"])
def test_general_columns(storage):
    """Every column on the long path: obstacles, dead nodes beside fluid, corner
    open nodes, an open outlet, on ragged strips."""
    t = H.porous_types(131, 190, fraction=0.25, rmin=2, rmax=5, seed=3)
    t[1:-1, 0] = H.BOUNDARY
    t[:, 0] = H.INLET
    t[60, 90] = t[61, 90] = H.SOLID
    lists = H.classify(t)
    p = H.Params(tau=0.8, outlet_bc=H.BC_OPEN)
    plan = [(5, False), (64, False), (2, True)]
    table = H.open_values(lists, "const:0.02:0.005", "const:0.01:0", 1)
    act = H.active_mask(lists)
    ref = advance(lists, p, table, storage, -1, plan)
    for pipeline in (3, 4, 5):
        same(advance(lists, p, table, storage, pipeline, plan), ref, act)
    if storage == 0:
        o = H.run_oracle(lists, p, 1 + sum(k for k, _ in plan), table)
        np.testing.assert_array_equal(ref[2][:, act], o["post"][:, act])


@pytest.mark.parametrize("kind,rows,cols,storage,default", [
    ("cavity", 700, 940, 0, -1), ("cavity", 1001, 1049, 1, -1), ("cavity", 977, 953, 2, -1),
    ("porous", 1440, 1460, 1, -3)], ids=["f64", "f32s", "f16s", "porous_f32s"])
def test_longer_runs_of_large_lattices(kind, rows, cols, storage, default):
    """The smallest lattices whose longer runs stream by default: lone steps,
    short and long runs, output steps and graph replays in turn equal the
    one-thread-per-node kernel; the reported pipeline is unchanged."""
    import llalbm_cuda as L

    if kind == "cavity":
        t = np.full((rows, cols), H.FLUID, dtype=np.uint8)
        t[0, :] = t[-1, :] = t[:, 0] = t[:, -1] = H.BOUNDARY
        t[0, 1:-1] = H.INLET
    else:
        t = H.porous_types(rows, cols, seed=6)
    n = L.classify(t)
    outs = []
    for pipeline in (None, -1):
        with L.from_types(t, storage=storage, tau=0.8, outlet_bc=2) as g:
            assert g.pipeline == default
            if pipeline is not None:
                g.set_pipeline(pipeline)
            v = np.zeros((1, g.n_open, 2))
            v[0, :, 0] = 0.05
            v[0, len(n["inlet"]):, 0] = 1.0
            g.set_open_values(v)
            g.init()
            for k, macro in [(1, False), (2, False), (37, True), (1, True), (65, False), (3, False), (34, True)]:
                g.step(k, macro=macro)
            g.check_numerics()
            outs.append((g.t, g.post_collision(), g.macro()))
    assert outs[0][0] == outs[1][0]
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
    for x, y in zip(outs[0][2], outs[1][2]):
        np.testing.assert_array_equal(x, y)
