"""GPU: a minimisation stops as soon as its mean energy is below the energy target,
also where energies are negative (e_c < 0) and the target is zero or below: disks
and rigid bodies as the oracle does, the resident batched form as the grid form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 1000, 20000])
@pytest.mark.parametrize("target", [0.0, -1e-3, -1e9])
@pytest.mark.parametrize("mode", [None, "cond", "stream"])
def test_disks_stop_below_the_target(monkeypatch, n, target, mode):
    import dpcuda_gb300 as dpg
    from oracle.oracle import DiskOracle, disk_packing
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    st = disk_packing(n, 0.86, 3)
    o = DiskOracle(n, st["box"], -1.0, 2.0)
    o.set_arrays(x=st["x"], y=st["y"], r=st["r"], m=st["m"])
    o.setup_neighbors(0, 1.7 / 1.4, 0.2, 8.0, 0.5)
    steps, _ = o.minimize_fire(0.1, 1e-3, target, 0.0, 5, 0.0)
    s = dpg.Disk(n, st["box"], -1.0, 2.0)
    s.setState(st["x"], st["y"], None, None, st["r"], st["m"])
    s.setupNeighbors("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)
    r = dpg.minimizeFire(s, 0.1, 1e-3, target, 0.0, 5)
    assert r["steps"] == steps == (0 if target > -1e9 else 5)
    a, b = s.getState(), o.get_arrays()
    for k in ("x", "y", "fx", "fy", "pe"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    s.close()


@pytest.mark.parametrize("mode", [None, "cond"])
def test_bodies_stop_below_the_target(monkeypatch, mode):
    import dpcuda_gb300 as dpg
    from oracle.oracle import bumpy_packing
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    st = bumpy_packing(65, 0.9, 5, n_small=20)
    b = dpg.RigidBumpy(65, st["nv"], st["box"], -st["e_c"], 2.0, st["rv"], st["seg"], True)
    b.setBodies(st["x"], st["y"], st["th"], st["r"], st["nvb"])
    b.setMass(1.0)
    b.setupNeighbors("cell", 1.5, 0.2, 8.0, 0.5)
    r = b.minimizeFire(0.1, 1e-3, 0.0, 0.0, 5)
    assert r["steps"] == 0
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [64, 300, 3000, 5000])
def test_batches_stop_below_the_target(n, precision):
    import dpcuda_gb300 as dpg
    from dpcuda_gb300.ensemble import FORM_GRID, FORM_RESIDENT
    from oracle.oracle import disk_packing
    sts = [disk_packing(n, 0.86, 3 + k) for k in range(2)]
    got = []
    for form in (FORM_RESIDENT, FORM_GRID):
        e = dpg.Ensemble([n] * 2, [q["box"] for q in sts], 1.7, 0.3, -1.0, 2.0, precision=precision)
        e.setForm(form)
        e.setState(*[np.concatenate([q[c] for q in sts]) for c in ("x", "y", "r", "m")])
        res = e.minimizeFire(0.1, 1e-3, 0.0, 0.0, 5, fmax_target=1e-13)
        got.append([(r["fire_steps"], r["converged"]) for r in res])
        e.close()
    # the resident form counts the FP64 pass that measures a mixed minimum, too
    assert got[0] == [(steps + precision, done) for steps, done in got[1]]
