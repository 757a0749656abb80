"""GPU: batches of the resident form in which shapes that share a kernel need
different amounts of shared memory: dilute systems, whose cell lists are large,
beside dense ones.  Each system's state is that of the system run alone, bit for
bit.  And the widest cell grids that are accepted run."""
import numpy as np
import pytest

from test_resident_shapes_gpu import CUT, run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dpg():
    import dpcuda_gb300
    dpcuda_gb300.load_library()
    return dpcuda_gb300


def system(n, phi):
    from oracle.oracle import disk_packing
    return disk_packing(n, phi, 40 + n)


@pytest.mark.parametrize("parts", [
    [(256, 0.02, 1), (600, 0.86, 1)],     # few systems: both on clusters of 8-particle warps
    [(4096, 0.25, 8), (1000, 0.86, 12)],  # more: clusters of 32-particle warps
    [(500, 0.03, 30), (900, 0.86, 90), (2000, 0.86, 20)],
])
def test_shapes_that_share_a_kernel(dpg, parts):
    sts = [system(n, phi) for n, phi, k in parts for _ in range(k)]
    out, _ = run(dpg, sts, 60)
    at = 0
    for n, phi, k in parts:
        alone, _ = run(dpg, [system(n, phi)], 60)
        for c in ("x", "y", "fx", "fy"):
            got = out[c][at:at + n * k].reshape(k, n)
            np.testing.assert_array_equal(got, np.tile(alone[c], (k, 1)), err_msg=f"{n} {c}")
        at += n * k


@pytest.mark.parametrize("n,side", [(64, 168), (16384, 127)])
def test_widest_cell_grids_run(dpg, n, side):
    st = system(n, 0.86)
    st = dict(st, box=side * 1.1 * CUT * 1.0001)
    out, res = run(dpg, [st], 40)
    assert res[0]["fire_steps"] > 0
    for c in ("x", "y", "fx", "fy"):
        assert np.all(np.isfinite(out[c]))
