"""GPU: nothing that the batched resident form reports depends on the shape that
runs a system: positions, forces, energy, pressure, contacts and max|F| are the
same bits for a system alone (the wide table) and in batches that take the other
tables, in FP64 throughout, and in the mixed form past its switch to double words
with the FP64 pass that measures every minimum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EDGES = [2, 63, 64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097]
REPORTED = ("avg_pe", "pressure", "contacts", "max_force", "fire_steps", "dw_steps", "fp64_steps", "converged")


@pytest.fixture(scope="module")
def dpg():
    import dpcuda_gb300
    dpcuda_gb300.load_library()
    return dpcuda_gb300


def packing(n, phi=None):
    from oracle.oracle import disk_packing
    return disk_packing(n, phi or (0.1 if n < 4 else 0.86), 500 + n)


def run(dpg, sts, mixed, steps):
    from dpcuda_gb300.ensemble import FORM_RESIDENT
    e = dpg.Ensemble([len(s["r"]) for s in sts], [s["box"] for s in sts], 1.7, 0.3,
                     precision=dpg.MIXED if mixed else dpg.FP64)
    e.setForm(FORM_RESIDENT)
    e.setState(*[np.concatenate([s[c] for s in sts]) for c in ("x", "y", "r", "m")])
    res = e.minimizeFire(0.1, 1e-2, 0.0, 0.0, steps, fmax_target=1e-13)
    out = e.getState()
    e.close()
    return out, res


STEPS = {False: 150, True: 2500}


@pytest.fixture(scope="module")
def dense(dpg):
    sts = [packing(n) for n in EDGES] + [packing(601 + k) for k in range(20)]
    off = np.concatenate([[0], np.cumsum([len(s["r"]) for s in sts])])
    got = {}
    for mixed in (False, True):
        out, res = run(dpg, sts, mixed, STEPS[mixed])
        got[mixed] = {n: ({c: out[c][off[k]:off[k + 1]] for c in out}, res[k]) for k, n in enumerate(EDGES)}
    return got


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", EDGES)
def test_reports_do_not_depend_on_the_shape(dpg, dense, n, mixed):
    out, res = run(dpg, [packing(n)], mixed, STEPS[mixed])
    want, rep = dense[mixed][n]
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(out[c], want[c], err_msg=c)
    assert {k: res[0][k] for k in REPORTED} == {k: rep[k] for k in REPORTED}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,copies", [(100, 140), (100, 290), (100, 500), (250, 140), (250, 290), (400, 200),
                                      (900, 60), (1800, 30)])
def test_every_table_reports_the_same(dpg, n, copies, mixed):
    st = packing(n)
    steps = STEPS[mixed] if copies < 200 else 150
    alone, one = run(dpg, [st], mixed, steps)
    batch, all_ = run(dpg, [st] * copies, mixed, steps)
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(batch[c].reshape(copies, n), np.tile(alone[c], (copies, 1)), err_msg=c)
    for r in all_:
        assert {k: r[k] for k in REPORTED} == {k: one[0][k] for k in REPORTED}


@pytest.mark.parametrize("n,side", [(64, 168), (100, 168), (200, 166), (300, 160)])
def test_fp64_systems_keep_the_widest_grids(dpg, n, side):
    """The shapes that FP64 systems prefer leave less room for the cells; where they
    do not fit, the wide table's run the system."""
    st = packing(n)
    st = dict(st, box=side * 1.1 * 1.7 * 1.0001)
    out, res = run(dpg, [st], False, 40)
    assert res[0]["fire_steps"] > 0
    for c in ("x", "y", "fx", "fy"):
        assert np.all(np.isfinite(out[c]))
