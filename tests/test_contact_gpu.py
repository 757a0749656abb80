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
