"""Results reach the caller's arrays whole on every route (small, direct and
large copies), also from several threads at once."""
import threading

import numpy as np
import pytest

import harness as H

pytestmark = pytest.mark.gpu


def fields(n_rows, n_cols, steps):
    import llalbm_cuda as L

    t = np.full((n_rows, n_cols), H.FLUID, dtype=np.uint8)
    t[0, :] = t[-1, :] = t[:, 0] = t[:, -1] = H.BOUNDARY
    t[0, 1:-1] = H.INLET
    g = L.from_types(t, storage=L.STORE_F32S, tau=0.8)
    v = np.zeros((1, g.n_open, 2))
    v[0, :, 0] = np.linspace(0.02, 0.1, g.n_open)
    g.set_open_values(v)
    g.init()
    g.step(steps, macro=True)
    return g


# rho and u: 3 x 8 bytes a node; 512 KB and 32 MB are the borders of the routes
@pytest.mark.parametrize("rows,cols", [(3, 3), (146, 149), (147, 149), (300, 300), (1181, 1183), (1183, 1183), (1700, 1001)])
def test_fields_and_populations(rows, cols):
    """rho and u after an output step equal those computed from the
    post-collision state of the step before, in numpy."""
    with fields(rows, cols, 7) as g:
        post = g.post_collision()
        g.step(1, macro=True)
        rho, u = g.macro()
        rho2, u2 = g.macro()
        np.testing.assert_array_equal(rho, rho2)
        np.testing.assert_array_equal(u, u2)
        # interior fluid nodes two away from the walls pull from fluid nodes
        sl = lambda k: post[k, 2 - H.DJ[k]:cols - 2 - H.DJ[k], 2 - H.DI[k]:rows - 2 - H.DI[k]]
        if rows > 5 and cols > 5:
            s = np.stack([sl(k) for k in range(9)])
            r = s.sum(axis=0)
            ux = (s[1] + s[5] + s[8] - s[3] - s[6] - s[7]) / r
            # FP32 moments of order-one populations: 9 roundings of 2^-24 each way
            assert np.abs(rho[2:-2, 2:-2] - r).max() <= 16 * 2.0**-24
            assert np.abs(u[0, 2:-2, 2:-2] - ux).max() <= 32 * 2.0**-24


def test_concurrent_copies():
    """Two threads read large and small fields of two lattices over and over:
    the calls share the staging memory or copy directly, the data is whole."""
    with fields(1300, 1200, 3) as a, fields(60, 50, 3) as b:
        want = {id(a): a.macro(), id(b): b.macro()}
        bad = []

        def read(g, n):
            for _ in range(n):
                r, u = g.macro()
                if not (np.array_equal(r, want[id(g)][0]) and np.array_equal(u, want[id(g)][1])):
                    bad.append(g)

        ts = [threading.Thread(target=read, args=(a, 12)), threading.Thread(target=read, args=(b, 200))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not bad
