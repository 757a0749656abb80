"""GPU: resident loops of several handles at once, each from its own host thread on
its own stream, give the bits of each handle alone: systems that share the SMs and
systems that have to wait for one another, of both particle types together."""
import threading

import numpy as np
import pytest

import test_barrier_limit_gpu as make

pytestmark = pytest.mark.gpu


def work(s, dpg):
    for _ in range(3):
        s.nveSteps(5e-3, 120)
        if isinstance(s, dpg.Disk):
            dpg.minimizeFire(s, 0.1, 1e-2, 0.0, 0.0, 60)
        else:
            s.minimizeFire(0.1, 1e-2, 0.0, 0.0, 60)


def state(s, dpg):
    return s.getState() if isinstance(s, dpg.Disk) else s.getBodies()


@pytest.mark.parametrize("kinds", [
    [("disks", 64)] * 4, [("disks", 1000)] * 3, [("disks", 16384)] * 2, [("disks", 40000)] * 2,
    [("bodies", 33)] * 2, [("bodies", 301)] * 3, [("bodies", 1500)] * 2,
    [("disks", 300), ("disks", 2000), ("bodies", 301), ("bodies", 1500)],
])
def test_handles_at_once(kinds):
    import dpcuda_gb300 as dpg

    def build(q):
        return make.disks(dpg, q[1]) if q[0] == "disks" else make.bodies(dpg, q[1])

    want = {}
    for q in set(kinds):
        s = build(q)
        work(s, dpg)
        want[q] = state(s, dpg)
        s.close()
    handles = [build(q) for q in kinds]
    errors = []

    def go(s):
        try:
            work(s, dpg)
        except Exception as e:  # reported below, not in the thread
            errors.append(e)

    threads = [threading.Thread(target=go, args=(s,)) for s in handles]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for q, s in zip(kinds, handles):
        got = state(s, dpg)
        for k in got:
            np.testing.assert_array_equal(got[k], want[q][k], err_msg=f"{q} {k}")
        s.close()
