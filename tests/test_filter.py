"""The fixed-point filter in front of the FP64 pair tests.

CPU: the filter's arithmetic restated in numpy never rules out a pair that the
FP64 test accepts, nor accepts one that it rejects, over boxes, units and
unwrapped positions up to its limit.  GPU: lists, forces, contacts and pressure
stay those of the oracle where the filter's cases change (the sizes around a
warp, unwrapped and far positions, units that switch it off, lists longer than
a slot chunk and queues longer than a window)."""
import numpy as np
import pytest

TOL = 4.0 / 4294967296.0


def fixed(x, L):
    return (np.floor(x * (4294967296.0 / L)).astype(np.int64) & 0xFFFFFFFF).astype(np.uint32)


def d2_fixed(x, y, i, j, L):
    f = np.float32
    s = f(L / 4294967296.0)
    ux, uy = fixed(x, L), fixed(y, L)
    dx = (ux[i] - ux[j]).view(np.int32).astype(f) * s
    dy = (uy[i] - uy[j]).view(np.int32).astype(f) * s
    return dx * dx + dy * dy


@pytest.mark.parametrize("L", [1e-11, 2.4, 9.7, 148.8, 907.3, 3.1e4, 1e11])
@pytest.mark.parametrize("images", [0, 3, 4000])
def test_filter_bounds_the_exact_distance(L, images):
    g = np.random.default_rng(int(L * 7) % 1000 + images)
    n, m = 4000, 400_000
    x = g.uniform(0, L, n) + L * g.integers(-images, images + 1, n)
    y = g.uniform(0, L, n) + L * g.integers(-images, images + 1, n)
    i, j = g.integers(0, n, m), g.integers(0, n, m)
    dx, dy = x[i] - x[j], y[i] - y[j]
    dx, dy = dx - L * np.round(dx / L), dy - L * np.round(dy / L)
    d2, f2 = dx * dx + dy * dy, d2_fixed(x, y, i, j, L)
    for c in np.sqrt(d2[:200]) * g.uniform(0.999999, 1.000001, 200):  # limits at the pairs' own distances
        t = np.float32(np.float32(c) * np.float32(1.00001) + np.float32(L * TOL))
        assert not np.any((f2 > t * t) & (d2 < c * c))
        lo = np.float32(np.float32(c) * np.float32(0.99999) - np.float32(L * TOL))
        if lo > 0:
            assert not np.any((f2 < lo * lo) & (d2 >= c * c))


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("n,phi,images,unit", [
    (4, 0.8, 0, 1.0), (31, 0.84, 0, 1.0), (33, 0.84, 2, 1.0), (257, 0.86, 0, 1.0), (1025, 0.86, 3, 1.0),
    (300, 0.86, 6000, 1.0),      # beyond 4096 boxes: every pair tested in FP64
    (300, 0.86, 1, 1e-14),       # units that switch the filter off
    (500, 4.0, 0, 1.0),          # some 30 contacts a disk
])
def test_lists_and_sums_match_the_oracle(n, phi, images, unit, lanes):
    import dpcuda_gb300 as dpg
    from oracle.oracle import DiskOracle, disk_packing
    st = disk_packing(n, phi, 11)
    g = np.random.default_rng(n)
    L = st["box"] * unit
    x = st["x"] * unit + L * g.integers(-images, images + 1, n)
    y = st["y"] * unit + L * g.integers(-images, images + 1, n)
    r = st["r"] * unit
    o = DiskOracle(n, L)
    o.set_arrays(x=x, y=y, r=r, m=st["m"])
    o.setup_neighbors(0, 1.7 / 1.4, 0.2, 8.0, 0.5)
    s = dpg.Disk(n, L)
    s.setForceGroup(lanes)
    s.setState(x, y, None, None, r, st["m"])
    s.setupNeighbors("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)
    a, b = s.getState(), o.get_arrays()
    for k in ("x", "y", "fx", "fy", "pe"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert s.getContactCount() == o.contact_count()
    np.testing.assert_allclose(s.getPressure(), o.pressure(), rtol=1e-12)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,phi,n_small", [(1, 0.5, 20), (33, 0.8, 3), (100, 0.9, 20), (65, 0.9, 33), (40, 1.5, 70)])
def test_vertex_lists_and_sums_match_the_oracle(n, phi, n_small):
    import dpcuda_gb300 as dpg
    from oracle.oracle import BumpyOracle, bumpy_packing
    st = bumpy_packing(n, phi, 5, n_small=n_small)
    o = BumpyOracle(n, st["nv"], st["box"], st["e_c"], 2.0, st["rv"], st["seg"], True)
    o.set_bodies(st["x"], st["y"], st["th"], st["r"], st["nvb"])
    o.init_vertices()
    o.set_mass(1.0)
    o.setup_neighbors(0, 1.5, 0.2, 8.0, 0.5)
    px, py = o.vertices()
    b = dpg.RigidBumpy(n, st["nv"], st["box"], st["e_c"], 2.0, st["rv"], st["seg"], True)
    b.setBodies(st["x"], st["y"], st["th"], st["r"], st["nvb"])
    b.setVertexPositions(px, py)
    b.setMass(1.0)
    b.setupNeighbors("cell", 1.5, 0.2, 8.0, 0.5)
    g, r = b.getBodies(), o.bodies()
    for k in ("fx", "fy", "tq", "pe"):
        np.testing.assert_array_equal(g[k], r[k], err_msg=k)
    assert b.getVertexNeighborSets() == o.vertex_neighbor_sets()
    b.close()
