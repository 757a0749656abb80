"""GPU: a mixed system whose switch threshold is zero goes over to FP64 when every
force is zero (max|F| <= 0), and the FP64 iteration after that passes the force
test: a minimisation of particles that do not touch ends at step 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [None, "cond", "stream"])
@pytest.mark.parametrize("switch", [0.0, 1e-6])
@pytest.mark.parametrize("n", [16, 900])
def test_disks_apart(monkeypatch, n, switch, mode):
    import dpcuda_gb300 as dpg
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    k = int(np.ceil(np.sqrt(n)))
    g = np.arange(n)
    s = dpg.Disk(n, 2.0 * k, precision=dpg.MIXED)
    s.setState(2.0 * (g % k) + 1.0, 2.0 * (g // k) + 1.0, None, None, np.full(n, 0.5), np.ones(n))
    s.setupNeighbors("verlet", 1.5, 0.2, 8.0, 0.5)
    s.setMixedSwitch(switch)
    r = dpg.minimizeFire(s, 0.1, 1e-2, 0.0, 0.0, 50, fmax_target=1e-12)
    assert (r["steps"], r["converged"]) == (1, 1)
    s.close()


@pytest.mark.parametrize("mode", [None, "cond"])
@pytest.mark.parametrize("switch", [0.0, 1e-6])
def test_bodies_apart(monkeypatch, switch, mode):
    import dpcuda_gb300 as dpg
    from oracle.oracle import bumpy_packing
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    n = 16
    st = bumpy_packing(n, 0.1, 5, n_small=12)
    g = np.arange(n)
    b = dpg.RigidBumpy(n, st["nv"], 12.0, st["e_c"], 2.0, st["rv"], st["seg"], True, precision=dpg.MIXED)
    b.setBodies(3.0 * (g % 4) + 1.5, 3.0 * (g // 4) + 1.5, st["th"], st["r"], st["nvb"])
    b.setMass(1.0)
    b.setupNeighbors("verlet", 1.5, 0.2, 8.0, 0.5)
    b.setMixedSwitch(switch)
    r = b.minimizeFire(0.1, 1e-2, 0.0, 0.0, 50, fmax_target=1e-12, tmax_target=1e-12)
    assert (r["steps"], r["converged"]) == (1, 1)
    b.close()
