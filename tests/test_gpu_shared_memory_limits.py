"""Kernels whose dynamic shared memory exceeds the default limit raise it at every launch: the limit
belongs to the device, and a thread may use contexts on several.  Counted by a library loaded ahead
of the CUDA runtime, on one device with two contexts."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int n;
int cudaFuncSetAttribute(const void *f, int a, int v) {
    static int (*real)(const void *, int, int);
    if (!real) {  /* the runtime this process has loaded by now */
        void *rt = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
        real = rt ? (int (*)(const void *, int, int))dlsym(rt, "cudaFuncSetAttribute") : 0;
    }
    ++n;
    return real ? real(f, a, v) : 999;
}
int counted(void) { return n; }
"""

_CHILD = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
counted = ctypes.CDLL(sys.argv[2]).counted
import numpy as np, sfhgpu
rng = np.random.default_rng(1)
M = np.asfortranarray(rng.random((1000, 120)))
r, G, c = rng.random(120), np.empty(120), np.empty(1000)
d = rng.poisson(M @ r).astype(float)
x, s, e = rng.random(1200), np.full(1200, 0.3), np.linspace(0, 1, 101)

def work():
    ctx = sfhgpu.Context(0)
    H = sfhgpu.Models(M, storage="f64", ctx=ctx)
    for name, call in (
            ("fg!", lambda: sfhgpu.fg_(True, G, r, H, d, c)),
            ("stamp tiles", lambda: sfhgpu.bin_cmd_smooth(x, x, s, s, 1, edges=(e, e), ctx=ctx)),
            ("narrow stars", lambda: sfhgpu.bin_cmd_smooth(
                x, x, s / 3e3, s, 0, edges=(np.linspace(0, 1, 3101), e[::25]), ctx=ctx))):
        before = counted()
        call()
        yield name, counted() - before

first, second = dict(work()), dict(work())
print(first, second)
assert all(v > 0 for v in first.values()) and first == second
"""


def test_limits_are_raised_for_every_context(sfh, tmp_path):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("no C compiler")
    src, lib = tmp_path / "count.c", tmp_path / "count.so"
    src.write_text(_COUNT)
    subprocess.run([cc, "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    pkg = os.path.dirname(os.path.dirname(os.path.abspath(sfh.__file__)))
    p = subprocess.run([sys.executable, "-c", _CHILD, pkg, str(lib)], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, LD_PRELOAD=str(lib)))
    assert p.returncode == 0, p.stdout[-500:] + p.stderr[-1500:]
