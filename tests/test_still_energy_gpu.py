"""GPU: a minimisation that moves nothing ends at its first iteration by the
energy-change test, in every form of the loop: the energy before it and the energy
after it are sums of the same numbers, and have to be the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [None, "cond", "stream"])
@pytest.mark.parametrize("n", [3, 64, 113, 513, 2000, 16385, 30001])
def test_disks_that_stay(monkeypatch, n, mode):
    import dpcuda_gb300 as dpg
    from oracle.oracle import disk_packing
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    st = disk_packing(n, 0.9, 3)
    s = dpg.Disk(n, st["box"])
    s.setState(st["x"], st["y"], None, None, st["r"], st["m"])
    s.setupNeighbors("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)
    r = dpg.minimizeFire(s, 0.1, 1e-14, 0.0, 1e-16, 20)  # forces of at most ~10 move a disk by 1e-27
    assert (r["steps"], r["converged"]) == (0, 1)
    s.close()


@pytest.mark.parametrize("mode", [None, "cond"])
@pytest.mark.parametrize("n", [5, 301, 1500])
def test_bodies_that_stay(monkeypatch, n, mode):
    import dpcuda_gb300 as dpg
    from oracle.oracle import bumpy_packing
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    st = bumpy_packing(n, 0.9, 3, n_small=12)
    b = dpg.RigidBumpy(n, st["nv"], st["box"], st["e_c"], 2.0, st["rv"], st["seg"], True)
    b.setBodies(st["x"], st["y"], st["th"], st["r"], st["nvb"])
    b.setMass(1.0)
    b.setupNeighbors("cell", 1.5, 0.2, 8.0, 0.5)
    r = b.minimizeFire(0.1, 1e-14, 0.0, 1e-16, 20)
    assert (r["steps"], r["converged"]) == (0, 1)
    b.close()
