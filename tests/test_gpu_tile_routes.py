"""Which lattices step in tiles: those with no more tiles than SMs, and not a few
rows that the cluster kernel holds.  The numbers of tiles are for 148 SMs."""
import numpy as np
import pytest

import harness as H
from test_gpu_run_kernel import box, kernel, lattice

pytestmark = pytest.mark.gpu
TILES = 16


def sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


# rows, columns, form (3: partially saturated obstacles in FP64), steps in tiles
SHAPES = [(129, 129, 0, True), (181, 333, 0, True), (1492, 43, 0, True), (24, 3800, 0, True), (1000, 3, 0, True),
          (256, 380, 0, False), (256, 400, 0, False), (300, 380, 0, False), (3, 30000, 0, False), (20000, 5, 0, False),
          (3, 3900, 0, False), (3, 2000, 0, False), (3, 1000, 0, True),
          (256, 400, 1, True), (440, 450, 1, True), (400, 490, 1, False), (16, 12000, 1, False), (60000, 3, 1, False),
          (3, 3900, 1, False), (50, 3800, 1, True),
          (129, 129, 2, True), (680, 578, 2, True), (630, 630, 2, False), (7, 13053, 2, False), (130, 3000, 2, False),
          (3, 2800, 2, False), (100, 3800, 2, True), (80, 90, 2, False),
          (100, 250, 3, True), (200, 249, 3, False), (115, 292, 3, False)]


@pytest.mark.parametrize("rows,cols,form,tiles", SHAPES)
def test_lattices_that_step_in_tiles(rows, cols, form, tiles):
    if sms() != 148:
        pytest.skip("tiles per SM counted for 148 SMs")
    if form == 3:
        t = H.channel_types(rows, cols, discs=[(rows // 2, cols // 4, rows // 8)])
        kw = dict(obstacle_bc=1, ps_tau=0.8)
    else:
        t, kw = box(rows, cols), dict(storage=form)
    with lattice(t, **kw) as g:
        assert (kernel(g, 200) == TILES) == tiles
        if tiles:
            assert 3 <= g.run_kernel(200)[1] <= 8
            g.set_pipeline(g.pipeline)
            assert kernel(g, 200) == g.pipeline


# lattice, form, and the kernel of a run of so many steps (with output: o): T tiles,
# G one thread per node, C the cluster
RUNS = [("cavity 129 x 129", 0, dict(zip((1, 2, 3, 50, "1o", "2o", "3o"), "GTTTGTT"))),
        ("cavity 181 x 333", 0, dict(zip((1, 2, 3, 50, "1o", "2o", "3o"), "GGTTGGT"))),
        ("cavity 40 x 50", 1, dict(zip((1, 2, 3, 50, "1o", "2o", "3o"), "GTTTGTT"))),
        ("cavity 256 x 1024", 2, dict(zip((1, 2, 3, 50, "1o", "2o", "3o", "4o"), "GGTTGGGT"))),
        ("cavity 181 x 333", 2, dict(zip((1, 2, 3, 50, "1o", "2o", "3o"), "GTTTGTT"))),
        ("cavity 90 x 92", 2, dict(zip((1, 2, 8, 9, 200, "1o", "2o"), "GTTTTGT"))),
        ("channel 90 x 95", 2, dict(zip((1, 2, 8, 9, 200, "1o", "8o", "9o"), "GTTCCGTC"))),
        ("channel 150 x 165", 2, dict(zip((1, 2, 8, 9, 200, "1o", "9o"), "GTTTTGT")))]


@pytest.mark.parametrize("name,form,runs", RUNS, ids=[f"{r[0]} {r[1]}".replace(" ", "_") for r in RUNS])
def test_short_runs(name, form, runs):
    """Launches of one step, of two with two columns a warp, and long runs of small
    FP16 channels stay on the one-step kernels; the bits are theirs."""
    if sms() != 148:
        pytest.skip("tiles per SM counted for 148 SMs")
    kind, rows, _, cols = name.split()
    rows, cols = int(rows), int(cols)
    t = box(rows, cols) if kind == "cavity" else H.channel_types(rows, cols, discs=[(rows // 2, cols // 3, rows // 8)])
    posts = []
    for default in (True, False):
        with lattice(t, storage=form) as g:
            if not default:
                g.set_pipeline(-1)
            for run, k in runs.items():
                n, out = (int(run[:-1]), True) if isinstance(run, str) else (run, False)
                if default:
                    assert kernel(g, n, out) == {"T": TILES, "G": -1, "C": -4}[k], run
                g.step(n, macro=out)
                if out:
                    posts.append(g.macro()[1])
            for n in (4, 5, 7, 10, 11):  # remainders
                g.step(n, macro=n % 2 == 1)
            assert g.t == 1 + 37 + sum(int(str(r).rstrip("o")) for r in runs)
            posts += [g.post_collision(), g.macro()[0]]
    half = len(posts) // 2
    for a, b in zip(posts[:half], posts[half:]):
        np.testing.assert_array_equal(a, b)
