"""GPU: the disk contact's root and quotients against the oracle's IEEE ones, bit
for bit: contact constants inside and outside the range in which the quick forms
run, overlaps from nothing to complete, pairs at a distance of their radius sum
and one rounding step to either side, length scales at which the forces are
tiny or large, and a general exponent (CUDA's pow and the host's may differ in
the last bits, two rounding errors of ~1e-16 each: 1e-14 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dpg():
    import dpcuda_gb300
    dpcuda_gb300.load_library()
    return dpcuda_gb300


def pairs(scale):
    """64 separate pairs in a row: distance d / (r_i + r_j) from 1e-9 to 1 + 2 ulp."""
    g = np.random.default_rng(5)
    k = 64
    ri, rj = g.uniform(0.4, 0.7, k), g.uniform(0.4, 0.7, k)
    q = np.concatenate([10.0 ** g.uniform(-9, -1, 16), g.uniform(0.1, 1.0, 32), 1.0 - 10.0 ** g.uniform(-16, -8, 10),
                        1.0 + np.arange(-3, 3) * 2.0 ** -53])
    x0 = np.zeros(k)
    y0 = 4.0 * np.arange(k) + 2.0
    a = g.uniform(0, 2 * np.pi, k)
    a[-6:] = 0.0  # the last ones along x from 0: their distance is exact
    d = q * (ri + rj)
    x = np.stack([x0, d * np.cos(a)], 1).ravel()
    y = np.stack([y0, y0 + d * np.sin(a)], 1).ravel()
    return x * scale, y * scale, np.stack([ri, rj], 1).ravel() * scale, 4.0 * k * scale


@pytest.mark.parametrize("e_c,n_c", [(1.0, 2.0), (0.37, 2.0), (1e-70, 2.0), (1e70, 2.0), (1.0, 2.5)])
@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e6])
def test_contacts_are_the_oracles(dpg, e_c, n_c, scale):
    from oracle.oracle import DiskOracle
    x, y, r, box = pairs(scale)
    n = len(x)
    o = DiskOracle(n, box, e_c, n_c)
    o.set_arrays(x=x, y=y, r=r, m=np.ones(n))
    o.setup_neighbors(2, 1.5, 0.2, 8.0, 0.5)
    s = dpg.Disk(n, box, e_c, n_c)
    s.setState(x, y, None, None, r, np.ones(n))
    s.setupNeighbors("all", 1.5, 0.2, 8.0, 0.5)
    s.zeroForceAndPotentialEnergy()
    s.calculateForces()
    o.zero_force_and_pe()
    o.calculate_forces()
    got, want = s.getState(), o.get_arrays()
    assert np.count_nonzero(want["fx"]) > n // 2
    for k in ("fx", "fy", "pe"):
        if n_c == 2.0:
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
        else:
            np.testing.assert_allclose(got[k], want[k], rtol=1e-14, atol=0, err_msg=k)
    s.close()
    o.close()


@pytest.mark.parametrize("n", [1, 33, 700])
@pytest.mark.parametrize("mass", ["unit", "random", "power", "tiny"])
def test_kicks_are_the_oracles(dpg, n, mass):
    """dt / m by unit masses, by the quick quotient and beyond its range (1e-70)."""
    from oracle.oracle import DiskOracle, disk_packing, fill_normal
    st = disk_packing(n, 0.5 if n > 1 else 0.1, 40 + n)
    g = np.random.default_rng(n)
    m = {"unit": np.ones(n), "random": g.uniform(0.3, 3.0, n), "power": 2.0 ** g.integers(-3, 4, n),
         "tiny": np.full(n, 1e-70)}[mass]
    vx, vy = fill_normal(n, 0.0, 1e-2, 1, n), fill_normal(n, 0.0, 1e-2, 1 + n, n)
    if mass == "tiny":  # no overlaps: a kick of anything but zero would leave the box
        st = dict(st, r=st["r"] * 1e-3)
    o = DiskOracle(n, st["box"])
    o.set_arrays(x=st["x"], y=st["y"], vx=vx, vy=vy, r=st["r"], m=m)
    o.setup_neighbors(0, 1.7 / 1.4, 0.2, 8.0, 0.5)
    s = dpg.Disk(n, st["box"])
    s.setState(st["x"], st["y"], vx, vy, st["r"], m)
    s.setupNeighbors("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)
    s.nveSteps(1e-2, 20)
    o.nve_steps(1e-2, 20)
    got, want = s.getState(), o.get_arrays()
    for k in ("x", "y", "vx", "vy", "fx", "fy", "pe"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    s.close()
    o.close()


@pytest.mark.parametrize("e_c", [2.0 ** -24, 2.0 ** 24])
@pytest.mark.parametrize("n,phi", [(2, 0.3), (31, 0.84), (700, 0.84), (700, 1.2), (5000, 0.84)])
def test_quick_fp32_contacts_are_the_general_ones(dpg, e_c, n, phi):
    """A contact constant of 2^-24 or 2^24 lies outside the quick FP32 operations'
    range and scales every term exactly: with 1 the forces must be the same bits."""
    from oracle.oracle import disk_packing
    st = disk_packing(n, phi, 60 + n)
    out = []
    for c in (1.0, e_c):
        s = dpg.Disk(n, st["box"], c, 2.0, precision=dpg.MIXED)
        s.setState(st["x"], st["y"], None, None, st["r"], st["m"])
        s.setupNeighbors("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)
        s.zeroForceAndPotentialEnergy()
        s.calculateForces()
        out.append(s.getState())
        s.close()
    for k in ("fx", "fy", "pe"):
        np.testing.assert_array_equal(out[1][k], e_c * out[0][k], err_msg=k)
