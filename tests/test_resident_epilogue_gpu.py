"""GPU: the batched resident form's short end of an iteration (no FP64 tests where
none can fire) does what the general one does, with and without energy targets: a
force target of 1e-30 takes the general one always, and until a target is near
the states are the same bits.  With energy targets, too, no shape changes a bit."""
import numpy as np
import pytest

from test_resident_totals_gpu import REPORTED, packing

pytestmark = pytest.mark.gpu
TARGETS = [(0.0, 0.0), (1e-16, 0.0), (1e-16, 1e-16), (0.0, 1e-9)]


def run(sts, switch, targets, steps, fmax):
    import dpcuda_gb300 as dpg
    from dpcuda_gb300.ensemble import FORM_RESIDENT
    e = dpg.Ensemble([len(s["r"]) for s in sts], [s["box"] for s in sts], 1.7, 0.3, precision=dpg.MIXED,
                     switch_fmax=switch)
    e.setForm(FORM_RESIDENT)
    e.setState(*[np.concatenate([s[c] for s in sts]) for c in ("x", "y", "r", "m")])
    res = e.minimizeFire(0.1, 1e-2, *targets, steps, fmax_target=fmax)
    out = e.getState()
    e.close()
    return out, res


@pytest.mark.parametrize("targets", TARGETS)
@pytest.mark.parametrize("switch", [1e-12, 1e3])  # FP32, and double words from the start
@pytest.mark.parametrize("n", [30, 100, 300, 1000, 3000, 5000])
def test_short_and_general_end(n, switch, targets):
    st = packing(n)
    a, ra = run([st], switch, targets, 500, 1e-13)
    b, rb = run([st], switch, targets, 500, 1e-30)
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(a[c], b[c], err_msg=c)
    for k in REPORTED:
        assert ra[0][k] == rb[0][k], k


@pytest.mark.parametrize("targets", TARGETS[1:])
@pytest.mark.parametrize("n,copies", [(64, 140), (100, 290), (250, 140), (400, 200), (900, 60), (1800, 30)])
def test_energy_targets_in_every_table(n, copies, targets):
    st = packing(n)
    alone, one = run([st], 1e-6, targets, 1500, 1e-13)
    batch, res = run([st] * copies, 1e-6, targets, 1500, 1e-13)
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(batch[c].reshape(copies, n), np.tile(alone[c], (copies, 1)), err_msg=c)
    for r in res:
        assert {k: r[k] for k in REPORTED} == {k: one[0][k] for k in REPORTED}
