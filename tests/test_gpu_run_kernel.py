"""How a lattice steps can be seen, left and gone back to (llb_run_kernel,
llb_set_pipeline, llb_reset_pipeline, llb_tune_pipeline)."""
import numpy as np
import pytest

import harness as H

pytestmark = pytest.mark.gpu

STREAM, COMPACT, GRID = 3, -3, -1


def box(rows, cols):
    t = np.full((rows, cols), H.FLUID, dtype=np.uint8)
    t[0, :] = t[-1, :] = t[:, 0] = t[:, -1] = H.BOUNDARY
    t[0, 1:-1] = H.INLET
    return t


def lattice(types, **kw):
    import llalbm_cuda as L

    n = L.classify(types)
    g = L.from_types(types, outlet_bc=2, **{"tau": 0.8, **kw})
    v = np.zeros((1, g.n_open, 2))
    v[0, :, 0] = 0.02
    v[0, len(n["inlet"]):, 0] = 1.0
    g.set_open_values(v)
    g.init()
    return g


def kernel(g, n, macro=False):
    return g.run_kernel(n, macro)[0]


# kernel of a long run by default
LATTICES = [("small", lambda: box(129, 129), 0, 16), ("large", lambda: box(900, 900), 0, STREAM),
            ("porous", lambda: H.porous_types(1500, 1460, seed=6), 1, STREAM)]


@pytest.mark.parametrize("name,types,storage,default", LATTICES, ids=[x[0] for x in LATTICES])
def test_reset_goes_back_to_the_default(name, types, storage, default):
    """Setting the reported configuration makes every step run on it; reset brings
    the default back, also where graphs of the same configuration exist, and
    the run is the run without either."""
    t = types()
    outs = []
    for switch in (True, False):
        with lattice(t, storage=storage) as g:
            assert kernel(g, 200) == default
            g.step(70)
            if switch:
                g.set_pipeline(g.pipeline)
                assert kernel(g, 200) == g.pipeline and g.run_kernel(200)[1] == 1
            g.step(66)
            if switch:
                g.reset_pipeline()
                assert kernel(g, 200) == default
            g.step(67, macro=True)
            if switch:
                g.reset_pipeline()  # nothing to do
            g.step(64)
            g.check_numerics()
            outs.append((g.t, g.post_collision(), g.macro()))
    assert outs[0][0] == outs[1][0]
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
    np.testing.assert_array_equal(outs[0][2][1], outs[1][2][1])


def test_run_kernel_of_every_configuration():
    import llalbm_cuda as L

    with lattice(box(129, 129)) as g:
        for cfg in (-4, -3, -2, -1, 0, 1, 2, 3, 4, 5, 6):
            g.set_pipeline(cfg)
            k, per = g.run_kernel(10)
            assert k == cfg and per == (10 if cfg == -4 else 2 if cfg in (3, 4, 5) else 1)
            assert g.run_kernel(1)[0] == (GRID if cfg in (3, 4, 5) else cfg)
            assert g.run_kernel(1, macro=True) == (GRID, 1)
        with pytest.raises(L.LLBError) as e:
            g.run_kernel(0)
        assert e.value.code == -1


def test_tuner_of_a_lattice_that_steps_in_tiles():
    """It tries the tiles and the one-thread kernel; the tiles are about twice as
    fast here and stay, and the steps advanced are those of every configuration."""
    with lattice(box(129, 129)) as g:
        configs = 0
        for cfg in (-4, -3, -2, -1, 0, 1, 2, 3, 4, 5, 6):
            g.set_pipeline(cfg)
            configs += 1
        best, ms = g.tune_pipeline(400)
        assert g.t == 1 + 2 * 400 * configs
        assert best == g.pipeline and kernel(g, 200) == 16 and 0.0 < ms < 0.003
        g.set_pipeline(best)
        assert kernel(g, 200) == best


def test_tuner_of_a_large_lattice():
    """The streaming kernel wins as configuration 3, which any lattice can be given."""
    with lattice(box(2000, 2000), storage=1) as g:
        best, ms = g.tune_pipeline(64)
        assert best == g.pipeline and kernel(g, 64) == best and best in (3, 4, 5)
