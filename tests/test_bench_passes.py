"""bench.py counts a run's passes over the lattice and its launches by the kernel
that runs, not by the configuration the lattice reports for a lone step."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


class Lattice:
    """A lattice of the given default: runs of `from_steps` steps or more take
    another kernel than shorter ones."""

    def __init__(self, pipeline, kernel, per, from_steps):
        self.pipeline, self.kernel, self.per, self.from_steps = pipeline, kernel, per, from_steps

    def run_kernel(self, n, macro=False):
        return (self.kernel, self.per) if n >= self.from_steps else (self.pipeline, 1)


# reported pipeline, run's kernel and its steps per launch, from so many steps; warm-up, steps;
# the run's kernel, steps per pass and launches
@pytest.mark.parametrize("lattice,warmup,steps,want", [
    ((-3, 3, 2, 32), 10, 1000, (3, 2, 501)),   # leaves the compacted planes: one copy
    ((-3, 3, 2, 32), 64, 1001, (3, 2, 501)),   # left them in the warm-up; a lone step at the end
    ((-3, 3, 2, 32), 10, 20, (-3, 1, 20)),
    ((0, 3, 2, 2), 10, 100, (3, 2, 50)),
    ((-1, -1, 1, 1), 10, 100, (-1, 1, 100)),
    ((-1, 16, 5, 3), 10, 2000, (16, 5, 400))])
def test_passes_of_a_run(lattice, warmup, steps, want):
    assert bench.run_launches(Lattice(*lattice), warmup, steps) == want


def test_a_streamed_run_moves_half_the_bytes():
    n = 4096 * 4096
    assert bench.bytes_per_step(8, n, n, 2) == (18 * 8 + 1) * n // 2
