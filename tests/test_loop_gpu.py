"""GPU: the loops as one resident grid give the bits of the loops as separate
launches (DPG_LOOP_MODE=stream), at the sizes where its blocks change: one
particle, fewer than a block, one more than fills a block or the last SM, more
than a block's registers hold, rows longer than its caches, and a list that
outgrows its capacity on the way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vx", "vy", "fx", "fy", "pe")


def system(dpg, monkeypatch, mode, n, phi, precision, method="cell"):
    from oracle.oracle import disk_packing
    if mode:
        monkeypatch.setenv("DPG_LOOP_MODE", mode)
    else:
        monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
    st = disk_packing(n, phi, 7)
    g = np.random.default_rng(n)
    v = g.normal(0, 0.05, (2, n))
    s = dpg.Disk(n, st["box"], precision=precision)
    s.setState(st["x"], st["y"], v[0], v[1], st["r"], g.uniform(0.5, 2.0, n))
    s.setupNeighbors(method, 1.7 / 1.4, 0.2, 8.0, 0.5)
    return s


def run(dpg, s, kind):
    if kind == "nve":
        s.nveSteps(1e-2, 1)
        s.nveSteps(1e-2, 61)
    elif kind == "damped":
        s.dampedNveSteps(2e-2, 0.3, 40)
    elif kind == "walls":
        s.nveWallSteps(1e-2, 40)
    else:
        r = dpg.minimizeFire(s, 0.1, 1e-2, 1e-16, 1e-16, 120)
        return s.getState(), s.neighborInfo(), (r["steps"], r["converged"], r["alpha"], r["dt"])
    return s.getState(), s.neighborInfo(), ()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["nve", "damped", "walls", "fire"])
@pytest.mark.parametrize("n,phi,method", [
    (1, 0.5, "cell"), (5, 0.8, "cell"), (33, 0.8, "all"), (63, 0.84, "verlet"), (609, 0.84, "cell"),
    (1217, 0.9, "cell"), (5000, 0.84, "cell"), (19457, 0.84, "cell"), (300, 4.0, "cell"),
])
def test_resident_grid_matches_separate_launches(monkeypatch, n, phi, method, kind, precision):
    import dpcuda_gb300 as dpg
    a = system(dpg, monkeypatch, "stream", n, phi, precision, method)
    b = system(dpg, monkeypatch, None, n, phi, precision, method)
    (sa, ia, ra), (sb, ib, rb) = run(dpg, a, kind), run(dpg, b, kind)
    for k in KEYS:
        np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
    assert ia == ib and ra == rb
    assert a.checkForNeighborUpdate() == b.checkForNeighborUpdate()
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["nve", "damped", "walls", "fire"])
@pytest.mark.parametrize("n,phi,n_small,rotation", [
    (1, 0.5, 20, True), (33, 0.8, 7, True), (301, 0.85, 20, False), (609, 0.85, 40, True), (5100, 0.8, 12, True),
])
def test_resident_grid_matches_separate_launches_bumpy(monkeypatch, n, phi, n_small, rotation, kind, precision):
    import dpcuda_gb300 as dpg
    from oracle.oracle import bumpy_packing
    st = bumpy_packing(n, phi, 3, n_small=n_small)
    g = np.random.default_rng(n)
    vel = g.normal(0, 0.05, (3, n))
    got = []
    for mode in ("stream", None):
        if mode:
            monkeypatch.setenv("DPG_LOOP_MODE", mode)
        else:
            monkeypatch.delenv("DPG_LOOP_MODE", raising=False)
        b = dpg.RigidBumpy(n, st["nv"], st["box"], st["e_c"], 2.0, st["rv"], st["seg"], rotation, precision=precision)
        b.setBodies(st["x"], st["y"], st["th"], st["r"], st["nvb"], vel[0], vel[1], vel[2])
        b.setMass(1.3)
        b.setupNeighbors("cell", 1.5, 0.2, 8.0, 0.5)
        r = ()
        if kind == "nve":
            b.nveSteps(5e-3, 1)
            b.nveSteps(5e-3, 40)
        elif kind == "damped":
            b.dampedNveSteps(5e-3, 0.3, 30)
        elif kind == "walls":
            b.nveWallSteps(5e-3, 30)
        else:
            q = b.minimizeFire(0.1, 1e-2, 1e-16, 1e-16, 60)
            r = (q["steps"], q["converged"])
        got.append((b.getBodies(), b.getVertexPositions(), b.neighborInfo(), r, b.checkForNeighborUpdate()))
        b.close()
    for k in got[0][0]:
        np.testing.assert_array_equal(got[0][0][k], got[1][0][k], err_msg=k)
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][2:] == got[1][2:]
