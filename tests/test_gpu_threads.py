"""Creating a context and reading labels where the host has no thread to spare: the work is done by
the threads there are, with the same labels.  A preloaded pthread_create refuses the threads that
std::thread asks for, beyond a given number."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdatomic.h>
#include <string.h>
static atomic_int left = 1 << 30, refused = 0;
void shim_allow(int k) { left = k; refused = 0; }
int shim_refused(void) { return refused; }
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x)
{
    static int (*real)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    Dl_info who;
    if (!real) *(void **)&real = dlsym(RTLD_NEXT, "pthread_create");
    if (dladdr(__builtin_return_address(0), &who) && who.dli_fname && strstr(who.dli_fname, "libstdc++") &&
        atomic_fetch_sub(&left, 1) <= 0) {
        ++refused;
        return EAGAIN;
    }
    return real(t, a, f, x);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
import galp_gb300, oracle
shim = ctypes.CDLL(None)
# planned on several threads (a quarter of a million vertices) and read by several (a million)
for n, policy in ((300_000, 0), (1_100_000, 0), (300_000, 1)):
    deg = 3
    off = np.arange(n + 1, dtype=np.int64) * deg
    nbr = np.random.default_rng(n).integers(0, n, n * deg).astype(np.int32)
    nbr[:50] = 7
    g = galp_gb300.Graph(off, nbr)
    with galp_gb300.Propagator(g, policy=policy, early_exit=0) as p:  # CUDA starts its own threads
        p.run(2)
        want = p.get_labels()
    if not policy:
        assert np.array_equal(want, oracle.run_par(off, nbr, 2, early_exit=False)[1])
    for allowed in (0, 1, 2, 5):
        shim.shim_allow(allowed)
        with galp_gb300.Propagator(g, policy=policy, early_exit=0) as p:
            planned = shim.shim_refused()
            p.run(2)
            got = p.get_labels()
        shim.shim_allow(1 << 30)
        assert planned or allowed, "no thread was refused"
        assert np.array_equal(got, want), (n, policy, allowed)
print("exact")
"""


def test_no_threads_to_be_had(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run([cc, "-shared", "-fPIC", "-O1", str(src), "-o", str(lib), "-ldl", "-lpthread"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.split()[-1:] == ["exact"], p.stderr[-2000:]
