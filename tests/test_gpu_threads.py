"""Host copies on several threads, where the system has none to give: the calls do the work themselves."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
int threads_left = -1, refused = 0;   /* -1: no limit */
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    static int (*real)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    if (!real) *(void**)&real = dlsym(RTLD_NEXT, "pthread_create");
    if (threads_left == 0) { ++refused; return EAGAIN; }
    if (threads_left > 0) --threads_left;
    return real(t, a, f, x);
}
"""

PROGRAM = r"""
import ctypes, sys
import numpy as np
import rawphys
from rawphys import scenes as S
shim = ctypes.CDLL(sys.argv[1])
left, refused = (ctypes.c_int.in_dll(shim, k) for k in ("threads_left", "refused"))
w = rawphys.World(0, "fp32")
w.load_batch(S.tower_batch(400, 64, seed=1, substeps=2))   # 26000 bodies: thirteen chunks of hulls, three of records
w.step(1)
hulls, state = w.transformed_hulls(), w.get_state()
for n in (0, 3):
    left.value, refused.value = n, 0
    v, nrm = w.transformed_hulls()
    w.set_state(state)
    got = w.get_state()
    left.value = -1
    assert refused.value > 0, n
    assert np.array_equal(v, hulls[0]) and np.array_equal(nrm, hulls[1]) and np.array_equal(got, state), n
print("same")
"""


def test_hulls_and_records_without_threads(ext_built, tmp_path):
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(lib), "-ldl"], check=True)
    pkg = os.path.dirname(os.path.dirname(ext_built.__file__))
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=pkg)
    run = subprocess.run([sys.executable, "-c", PROGRAM, str(lib)], env=env, capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.strip() == "same", run.stderr[-2000:]
