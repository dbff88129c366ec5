"""The streaming kernel's split of a lattice into tasks: one wave of them, several
waves, the sizes on both sides of the line between, and a width that leaves a
narrow last task.  The same bits as one step per launch."""
import numpy as np
import pytest

import harness as H

pytestmark = pytest.mark.gpu


# rows, columns: in FP64 about 15, 39, 41, 60 and 41 columns per resident warp
# (148 SMs), in FP32 half of that, in FP16 a third
@pytest.mark.parametrize("shape", [(1000, 997), (1601, 1566), (1601, 1650), (2000, 1930), (57, 24301)],
                         ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f64", "f32s", "f16s"])
def test_tasks_cover_the_lattice_once(storage, shape):
    import llalbm_cuda as L

    types = np.full(shape, H.FLUID, dtype=np.uint8)
    types[0, :] = types[-1, :] = types[:, 0] = types[:, -1] = H.BOUNDARY
    types[0, 1:-1] = H.INLET
    types[shape[0] // 3:shape[0] // 3 + 9, shape[1] // 2:shape[1] // 2 + 14] = H.OBSTACLE
    n = L.classify(types)
    v = np.zeros((1, len(n["inlet"]) + len(n["outlet"]), 2))
    v[0, :, 1] = np.linspace(0.0, 0.05, v.shape[1])
    out = []
    for pipeline in (3, -1):
        with L.from_types(types, storage=storage, collision=1, tau_even=0.6, tau_odd=1.1) as g:
            g.set_pipeline(pipeline)
            g.set_open_values(v)
            g.init()
            g.step(11)
            g.check_numerics()
            out.append(g.post_collision())
    np.testing.assert_array_equal(out[0], out[1])


# A lattice whose pipeline was never set, on both sides of the sizes from which
# its longer runs are streamed, either operator: the bits of one step per launch.
@pytest.mark.parametrize("storage,rows,cols", [(0, 800, 819), (0, 800, 820), (0, 885, 888), (0, 885, 889),
                                               (1, 885, 888), (1, 885, 889), (2, 800, 819), (2, 800, 820)])
@pytest.mark.parametrize("coll", [0, 1], ids=["bgk", "trt"])
def test_default_of_open_flow(storage, rows, cols, coll):
    import llalbm_cuda as L

    types = np.full((rows, cols), H.FLUID, dtype=np.uint8)
    types[0, :] = types[-1, :] = types[:, 0] = types[:, -1] = H.BOUNDARY
    types[0, 1:-1] = H.INLET
    v = np.full((1, cols - 2, 2), 0.03)
    par = dict(collision=0, tau=0.7) if coll == 0 else dict(collision=1, tau_even=0.6, tau_odd=1.1)
    out = []
    for default in (True, False):
        with L.from_types(types, storage=storage, **par) as g:
            if not default:
                g.set_pipeline(-1)
            g.set_open_values(v)
            g.init()
            g.step(40)
            out.append(g.post_collision())
    np.testing.assert_array_equal(out[0], out[1])


# Porous lattices around the sizes from which runs of 32 steps leave the compacted
# planes (FP64 with TRT never does).
@pytest.mark.parametrize("storage,shape", [(0, (1773, 1774)), (0, (1774, 1780)), (2, (1915, 1915)), (2, (1916, 1920))])
@pytest.mark.parametrize("coll", [0, 1], ids=["bgk", "trt"])
def test_default_of_porous_media(storage, shape, coll):
    import llalbm_cuda as L

    types = H.porous_types(*shape, seed=5)
    n = L.classify(types)
    v = np.zeros((1, len(n["inlet"]) + len(n["outlet"]), 2))
    v[0, :len(n["inlet"]), 1] = 0.02
    v[0, len(n["inlet"]):, 0] = 1.0
    par = dict(collision=0, tau=0.8) if coll == 0 else dict(collision=1, tau_even=0.6, tau_odd=1.1)
    out = []
    for default in (True, False):
        with L.from_types(types, storage=storage, outlet_bc=2, **par) as g:
            if not default:
                g.set_pipeline(-1)
            g.set_open_values(v)
            g.init()
            g.step(34)
            g.step(5)
            out.append(g.post_collision())
    np.testing.assert_array_equal(out[0], out[1])
