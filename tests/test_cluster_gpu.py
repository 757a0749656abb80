"""GPU: the disk loops on one thread-block cluster (up to 512 particles) give the
bits of the loops as separate launches, at the sizes where its blocks change:
two blocks, one particle in the last, sixteen blocks, more than four a block,
the largest, and one beyond."""
import numpy as np
import pytest

from test_loop_gpu import KEYS, run, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["nve", "fire"])
@pytest.mark.parametrize("n", [4, 8, 9, 64, 65, 300, 511, 512, 513])
def test_cluster_matches_separate_launches(monkeypatch, n, kind, precision):
    import dpcuda_gb300 as dpg
    a = system(dpg, monkeypatch, "stream", n, 0.84, precision)
    b = system(dpg, monkeypatch, None, n, 0.84, precision)
    (sa, ia, ra), (sb, ib, rb) = run(dpg, a, kind), run(dpg, b, kind)
    for k in KEYS:
        np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
    assert ia == ib and ra == rb
    a.close()
    b.close()
