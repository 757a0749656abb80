"""GPU: the shapes of the resident batched form at the edges of their ranges.

* A system's result does not depend on the shape that runs it: alone it takes
  the wide table (lanes per particle, clusters), in a batch that outgrows the
  SMs the dense one; after 200 FIRE iterations both states are the same bits.
* The forces reported there are the oracle's at those positions.  A pair force
  e_c (1 - d / s) / (s d) r carries a few rounding errors of ~1e-16 from the
  Newton reciprocals on terms of at most 1 / 0.5, a particle has at most ~10
  overlapping neighbours: 1e-12 absolute is far above the sum of them and far
  below an FP32 error.
* Lists longer than the rows kept on chip take the loads from memory; the
  minimum still passes the oracle.
* The cell grids that fit stay accepted: 168 cells a side at 64 disks (and 169
  refused), 127 at 16384.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CUT = 1.7
EDGES = [1, 2, 3, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049,
         4095, 4096, 4097]


@pytest.fixture(scope="module")
def dpg():
    import dpcuda_gb300
    dpcuda_gb300.load_library()
    return dpcuda_gb300


def packing(n, seed):
    from oracle.oracle import disk_packing
    return disk_packing(n, 0.1 if n < 4 else 0.86, seed)


def run(dpg, sts, steps, cut=CUT, skin=0.3, fmax=1e-13):
    from dpcuda_gb300.ensemble import FORM_RESIDENT
    e = dpg.Ensemble([len(s["r"]) for s in sts], [s["box"] for s in sts], cut, skin, precision=dpg.MIXED)
    e.setForm(FORM_RESIDENT)
    e.setState(*[np.concatenate([s[c] for s in sts]) for c in ("x", "y", "r", "m")])
    res = e.minimizeFire(0.1, 1e-2, 0.0, 0.0, steps, fmax_target=fmax)
    out = e.getState()
    e.close()
    return out, res


def oracle_forces(st, x, y):
    from oracle.oracle import DiskOracle
    o = DiskOracle(len(st["r"]), st["box"])
    o.set_arrays(x=x, y=y, r=st["r"], m=st["m"])
    o.setup_neighbors(0, CUT / 1.4, 0.2, 8.0, 0.5)
    o.zero_force_and_pe()
    o.calculate_forces()
    a = o.get_arrays()
    o.close()
    return a["fx"], a["fy"]


@pytest.fixture(scope="module")
def dense(dpg):
    """Every size at once, with fillers: more blocks than SMs."""
    sts = [packing(n, 500 + n) for n in EDGES] + [packing(600, 900 + k) for k in range(17)]
    out, _ = run(dpg, sts, 200)
    off = np.concatenate([[0], np.cumsum([len(s["r"]) for s in sts])])
    return {n: (sts[k], {c: out[c][off[k]:off[k + 1]] for c in out}) for k, n in enumerate(EDGES)}


@pytest.mark.parametrize("n", EDGES)
def test_results_do_not_depend_on_the_shape(dpg, dense, n):
    st, got = dense[n]
    alone, _ = run(dpg, [st], 200)
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(alone[c], got[c], err_msg=c)
    if n >= 4:  # smaller boxes hold fewer than three cells a side of the oracle's list
        fx, fy = oracle_forces(st, alone["x"], alone["y"])
        np.testing.assert_allclose(alone["fx"], fx, rtol=0, atol=1e-12)
        np.testing.assert_allclose(alone["fy"], fy, rtol=0, atol=1e-12)


@pytest.mark.parametrize("n", [200, 2500])
def test_long_lists_reach_the_minimum(dpg, n):
    st = packing(n, 700 + n)
    out, res = run(dpg, [st], 1_000_000, cut=4.4, skin=3.0)
    assert res[0]["converged"] == 1 and res[0]["max_force"] <= 1e-13
    fx, fy = oracle_forces(st, out["x"], out["y"])
    assert np.sqrt(fx ** 2 + fy ** 2).max() <= 1.01e-13


@pytest.mark.parametrize("n,side,fits", [(64, 168, True), (64, 169, False), (16384, 127, True)])
def test_cell_grids_that_fit(dpg, n, side, fits):
    from dpcuda_gb300.ensemble import FORM_RESIDENT
    box = side * 1.1 * CUT * 1.0001  # a cell is 1.1 cutoffs wide
    e = dpg.Ensemble([n], [box], CUT, 0.3, precision=dpg.MIXED)
    if fits:
        e.setForm(FORM_RESIDENT)
    else:
        with pytest.raises(Exception):
            e.setForm(FORM_RESIDENT)
    e.close()


@pytest.mark.parametrize("n,copies", [(100, 140), (100, 290), (100, 500), (250, 140), (250, 290), (400, 140), (400, 200)])
def test_every_table_gives_the_same_bits(dpg, n, copies):
    """Batches of equal systems that fill half an SM, a third or a quarter each,
    or more than there is: every copy is the system alone."""
    st = packing(n, 500 + n)
    alone, _ = run(dpg, [st], 100)
    batch, _ = run(dpg, [st] * copies, 100)
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(batch[c].reshape(copies, n), np.tile(alone[c], (copies, 1)), err_msg=c)
