"""Which lattices stream their longer runs by default, on both sides of every line:
the sizes, the operator, the rows streamed for nothing on lattices of few rows,
and lattices of few columns."""
import numpy as np
import pytest

import harness as H
from test_gpu_run_kernel import box, kernel, lattice

pytestmark = pytest.mark.gpu

BGK, TRT = dict(collision=0, tau=0.8), dict(collision=1, tau_even=0.8, tau_odd=1.1)
F64, F32, F16 = 0, 1, 2


# rows, columns, form, operator, longer runs stream
OPEN_FLOW = [(800, 819, F64, BGK, False), (800, 820, F64, BGK, True), (885, 888, F64, TRT, False),
             (885, 889, F64, TRT, True), (885, 888, F32, BGK, False), (885, 889, F32, TRT, True),
             (830, 789, F16, TRT, False), (830, 790, F16, BGK, True), (800, 820, F16, BGK, False),
             (100, 9000, F32, BGK, True), (400, 2100, F32, BGK, False), (128, 8192, F32, BGK, False), (64, 14000, F32, TRT, False),
             (128, 8192, F16, BGK, False), (440, 2100, F16, BGK, True), (128, 8192, F64, BGK, True),
             (64, 14000, F64, TRT, False), (470, 6000, F16, BGK, True), (260, 5000, F16, TRT, False), (260, 16000, F16, BGK, True),
             (128, 16000, F32, BGK, False),
             (25000, 31, F64, BGK, False), (90000, 10, F32, BGK, False), (3, 60000, F16, BGK, False)]


@pytest.mark.parametrize("rows,cols,form,coll,streams", OPEN_FLOW)
def test_open_flow(rows, cols, form, coll, streams):
    with lattice(box(rows, cols), storage=form, **coll) as g:
        assert (kernel(g, 200) == 3) == streams
        if streams:
            assert g.run_kernel(2) == (3, 2) and kernel(g, 1) == g.pipeline
            assert g.run_kernel(1, macro=True) == (-1, 1)


POROUS = [(1773, 1774, F64, BGK, False), (1774, 1780, F64, BGK, True), (1774, 1780, F64, TRT, False),
          (1448, 1448, F32, BGK, False), (1449, 1449, F32, TRT, True), (1915, 1915, F16, BGK, False),
          (1916, 1920, F16, TRT, True), (148, 22317, F64, BGK, False), (171, 12877, F32, BGK, False),
          (341, 11300, F16, BGK, False)]


@pytest.mark.parametrize("rows,cols,form,coll,streams", POROUS)
def test_porous_media(rows, cols, form, coll, streams):
    """Only runs of 32 steps or more leave the compacted planes."""
    with lattice(H.porous_types(rows, cols, seed=5), storage=form, **coll) as g:
        assert g.pipeline == -3 and kernel(g, 31) == -3
        assert (kernel(g, 32) == 3) == streams
        assert (kernel(g, 33, macro=True) == 3) == streams and kernel(g, 32, macro=True) == -3


def test_thin_lattice_steps_the_same_on_its_line():
    """100 x 9000 streams, 128 x 8192 does not; either gives the one-thread bits."""
    for rows, cols in ((100, 9000), (128, 8192)):
        posts = []
        for default in (True, False):
            with lattice(box(rows, cols), storage=F32) as g:
                if not default:
                    g.set_pipeline(-1)
                g.step(37)
                g.step(8, macro=True)
                posts.append(g.post_collision())
        np.testing.assert_array_equal(*posts)
