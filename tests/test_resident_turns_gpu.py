"""GPU: systems that take turns go on however short a turn is: a launch whose time
is up before it begins (a GPU shared with other processes may take it away between
the two) still runs its systems a little further, and where launches end changes no
result."""
import numpy as np
import pytest

from test_resident_totals_gpu import REPORTED, packing, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,copies", [(100, 700), (600, 200)])
@pytest.mark.parametrize("mixed", [False, True])
def test_turns_that_are_over_at_once(monkeypatch, n, copies, mixed):
    import dpcuda_gb300 as dpg
    st = packing(n)
    alone, one = run(dpg, [st], mixed, 200)
    monkeypatch.setenv("DPG_TURN_NS", "1")
    batch, res = run(dpg, [st] * copies, mixed, 200)
    for c in ("x", "y", "fx", "fy"):
        np.testing.assert_array_equal(batch[c].reshape(copies, n), np.tile(alone[c], (copies, 1)), err_msg=c)
    for r in res:
        assert {k: r[k] for k in REPORTED} == {k: one[0][k] for k in REPORTED}
