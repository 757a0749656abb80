"""GPU: where the cooperative (or cluster) launch of a resident loop is refused, the
loop runs as a graph and gives the bits of the separate launches.  The refusal
comes from a fake of the two launch calls, loaded ahead of the CUDA runtime in a
child process; from the first call on, or after a resident call has succeeded."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdlib.h>
int refused_launches, seen_launches;
static int refuse(void) {
    const char *a = getenv("REFUSE_AFTER");
    const int no = seen_launches++ >= (a ? atoi(a) : 0);
    refused_launches += no;
    return no;
}
typedef struct { unsigned x, y, z; } dim;
static void *real(const char *name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name); }
int cudaLaunchCooperativeKernel(const void *f, dim g, dim b, void **a, size_t m, void *s) {
    if (refuse()) return 720; /* cudaErrorCooperativeLaunchTooLarge */
    return ((int (*)(const void *, dim, dim, void **, size_t, void *))real("cudaLaunchCooperativeKernel"))(f, g, b, a, m, s);
}
int cudaLaunchKernelExC(const void *c, const void *f, void **a) {
    if (refuse()) return 720;
    return ((int (*)(const void *, const void *, void **))real("cudaLaunchKernelExC"))(c, f, a);
}
"""

CHILD = r"""
import ctypes, os, sys
for p in (sys.argv[1], sys.argv[1] + "/dpcuda-v2_gb300", sys.argv[1] + "/tests"):
    sys.path.insert(0, p)
import numpy as np
import dpcuda_gb300 as dpg
import test_barrier_limit_gpu as make
fake = ctypes.CDLL(None)
count = lambda: ctypes.c_int.in_dll(fake, "refused_launches").value
n, kind, prec = sys.argv[2], sys.argv[3], int(sys.argv[4])
got = []
for mode in ("stream", None):
    os.environ.pop("DPG_LOOP_MODE", None)
    if mode:
        os.environ["DPG_LOOP_MODE"] = mode
    s = make.bodies(dpg, 33) if n == "bodies" else make.disks(dpg, int(n), prec)
    for steps in (30, 40):
        if kind == "nve":
            s.nveSteps(1e-2, steps)
        elif n == "bodies":
            s.minimizeFire(0.1, 1e-2, 0.0, 0.0, steps)
        else:
            dpg.minimizeFire(s, 0.1, 1e-2, 0.0, 0.0, steps)
    got.append(s.getBodies() if n == "bodies" else s.getState())
    assert (count() > 0) == (mode is None), (mode, count())
    s.close()
for k in got[0]:
    np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("needs a host compiler")
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.c").write_text(FAKE)
    subprocess.run([cc, "-shared", "-fPIC", "-o", str(d / "fake.so"), str(d / "fake.c"), "-ldl"], check=True)
    return d / "fake.so"


@pytest.mark.parametrize("after", [0, 1])
@pytest.mark.parametrize("kind", ["nve", "fire"])
@pytest.mark.parametrize("n,prec", [("64", 0), ("2000", 0), ("2000", 1), ("30000", 0), ("bodies", 0)])
def test_a_refused_launch_runs_as_a_graph(fake, n, prec, kind, after):
    env = dict(os.environ, LD_PRELOAD=str(fake), REFUSE_AFTER=str(after))
    r = subprocess.run([sys.executable, "-c", CHILD, str(ROOT), n, kind, str(prec)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
