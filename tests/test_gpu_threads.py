"""Lattices driven from several host threads: distinct handles are independent."""
import threading
import time

import numpy as np
import pytest

import harness as H
from test_gpu_parity import make_gpu

pytestmark = pytest.mark.gpu


def saturated(rows, cols):
    t = H.channel_types(rows, cols, discs=[(rows // 2, cols // 3, 8)])
    lists = H.classify(t)
    p = H.Params(tau=0.8, outlet_bc=H.BC_ZH_PRESSURE, obstacle_bc=1, ps_tau=0.8)
    g = make_gpu(lists, p)
    v = np.zeros((1, g.n_open, 2))
    v[0, :len(lists.inlet), 0] = 0.02
    v[0, len(lists.inlet):, 0] = 1.0
    g.set_open_values(v)
    g.init()
    return g


def test_partially_saturated_tiles_of_different_sizes_from_two_threads():
    """Two lattices whose launches need different amounts of shared memory step
    at the same time; every call succeeds and both end in the state of a run on
    one thread."""
    shapes, calls, per = [(98, 280), (60, 65)], 6000, [3, 5]
    with saturated(*shapes[0]) as a, saturated(*shapes[1]) as b:
        errors = []

        def run(g, k):
            try:
                for _ in range(calls):
                    g.step(k)
                g.synchronize()
            except Exception as e:  # noqa: BLE001
                errors.append(e)

        ts = [threading.Thread(target=run, args=x) for x in zip((a, b), per)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not errors, errors
        got = [g.post_collision() for g in (a, b)]
    for shape, k, post in zip(shapes, per, got):
        with saturated(*shape) as g:
            for _ in range(calls):
                g.step(k)
            np.testing.assert_array_equal(g.post_collision(), post)


def cavity(n):
    import llalbm_cuda as L

    t = np.full((n, n), H.FLUID, dtype=np.uint8)
    t[0, :] = t[-1, :] = t[:, 0] = t[:, -1] = H.BOUNDARY
    t[0, 1:-1] = H.INLET
    g = L.from_types(t, tau=0.8)
    v = np.zeros((1, g.n_open, 2))
    v[0, :, 0] = 0.05
    g.set_open_values(v)
    g.init()
    return g


def test_lattices_come_and_go_while_another_thread_waits_for_results():
    """One thread waits for the fields of a lattice with seconds of steps queued;
    another creates and destroys lattices meanwhile, and is not held up until
    the results are there."""
    with cavity(2048) as g:
        g.step(64, macro=True)
        g.macro()
        with cavity(64):
            pass
        g.step(20000, macro=True)  # about 1.2 s on the device
        ready = threading.Event()

        def read():
            g.macro()
            ready.set()

        t = threading.Thread(target=read)
        t.start()
        time.sleep(0.05)
        made = 0
        while made < 3 and not ready.is_set():
            with cavity(64):
                pass
            made += not ready.is_set()
        t.join()
        assert made == 3


def test_waiting_for_results_takes_one_processor():
    """While a call waits for the steps queued before its results, only the calling
    thread is busy (it polls an event); the threads that will move the results
    touch the destination's pages and then sleep."""
    with cavity(2048) as g:
        g.step(64, macro=True)
        g.macro()
        g.step(20000, macro=True)  # about 1.2 s on the device
        wall, cpu = time.perf_counter(), time.process_time()
        g.macro()
        wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    # the copy itself, 100 MB with 9 threads, takes some 5 ms
    assert wall > 0.3 and cpu < 2.0 * wall
