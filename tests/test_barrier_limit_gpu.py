"""GPU: a grid barrier of the resident loops that runs out of looks is reported
as such, and leaves a handle that refuses to go on until its lists are set up
again.  The limit is set to one look, which no barrier of 152 blocks keeps; every
wait ends by itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMEOUT, STATE = 6, 5


def disks(dpg, n=2000, precision=0):
    from oracle.oracle import disk_packing
    st = disk_packing(n, 0.84, 7)
    v = np.random.default_rng(n).normal(0, 0.05, (2, n))
    s = dpg.Disk(n, st["box"], precision=precision)
    s.setState(st["x"], st["y"], v[0], v[1], st["r"], st["m"])
    s.setupNeighbors("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)
    return s


def bodies(dpg, n=609):
    from oracle.oracle import bumpy_packing
    st = bumpy_packing(n, 0.8, 3, n_small=20)
    v = np.random.default_rng(n).normal(0, 0.05, (3, n))
    b = dpg.RigidBumpy(n, st["nv"], st["box"], st["e_c"], 2.0, st["rv"], st["seg"], True)
    b.setBodies(st["x"], st["y"], st["th"], st["r"], st["nvb"], v[0], v[1], v[2])
    b.setMass(1.0)
    b.setupNeighbors("cell", 1.5, 0.2, 8.0, 0.5)
    return b


@pytest.mark.parametrize("make", [disks, lambda dpg: disks(dpg, 30000), lambda dpg: disks(dpg, 2000, 1), bodies])
@pytest.mark.parametrize("kind", ["nve", "fire"])
def test_a_barrier_that_runs_out_is_an_error(monkeypatch, make, kind):
    import dpcuda_gb300 as dpg

    def run(s):
        if kind == "nve":
            s.nveSteps(1e-2, 200)
        elif isinstance(s, dpg.Disk):
            dpg.minimizeFire(s, 0.1, 1e-2, 0.0, 0.0, 200)
        else:
            s.minimizeFire(0.1, 1e-2, 0.0, 0.0, 200)

    monkeypatch.setenv("DPG_LOOP_POLLS", "1")
    s = make(dpg)
    with pytest.raises(dpg.DpgError) as e:
        run(s)
    assert e.value.code == TIMEOUT
    with pytest.raises(dpg.DpgError) as e:  # the lists are gone
        run(s)
    assert e.value.code == STATE
    s.close()
    monkeypatch.delenv("DPG_LOOP_POLLS")
    s = make(dpg)  # the GPU is none the worse
    run(s)
    s.close()
