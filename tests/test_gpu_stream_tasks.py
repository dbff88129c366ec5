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
