"""Calls that have another way when the driver refuses a launch or an
allocation: the refusal is an error code from a stand-in for the driver's entry
point (preloaded in a child process), which launches and allocates nothing."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(shutil.which("gcc") is None, reason="no gcc")]

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static void *next_dlsym(void *h, const char *name) {
  static void *(*next)(void *, const char *);
  if (!next) next = dlvsym(RTLD_NEXT, "dlsym", "GLIBC_2.34");
  if (!next) next = dlvsym(RTLD_NEXT, "dlsym", "GLIBC_2.2.5");
  return next(h, name);
}

static int refuse_coop(void) {
  if (getenv("REFUSE_COOPERATIVE")) fprintf(stderr, "refused a cooperative launch\n");
  return getenv("REFUSE_COOPERATIVE") != NULL;
}
static int (*coop)(void *, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, void *,
                   void **);
static int my_coop(void *f, unsigned gx, unsigned gy, unsigned gz, unsigned bx, unsigned by, unsigned bz,
                   unsigned sm, void *s, void **args) {
  return refuse_coop() ? 720 : coop(f, gx, gy, gz, bx, by, bz, sm, s, args);
}

static int (*alloc)(unsigned long long *, size_t);
static int my_alloc(unsigned long long *p, size_t n) {
  const char *bytes = getenv("REFUSE_BYTES");
  if (bytes && n == strtoull(bytes, NULL, 10)) {
    fprintf(stderr, "refused %zu bytes\n", n);
    return 2;
  }
  return alloc(p, n);
}

static int my_proc(const char *, void **, int, unsigned long long, void *);
static int (*proc)(const char *, void **, int, unsigned long long, void *);

static void *stand_in(const char *name, void *real) {
  if (!real) return real;
  if (!strncmp(name, "cuGetProcAddress", 16)) {
    *(void **)&proc = real;
    return (void *)my_proc;
  }
  if (!strcmp(name, "cuLaunchCooperativeKernel")) {
    *(void **)&coop = real;
    return (void *)my_coop;
  }
  if (!strcmp(name, "cuMemAlloc") || !strcmp(name, "cuMemAlloc_v2")) {
    *(void **)&alloc = real;
    return (void *)my_alloc;
  }
  return real;
}

static int my_proc(const char *name, void **p, int version, unsigned long long flags, void *status) {
  const int rc = proc(name, p, version, flags, status);
  if (!rc && p) *p = stand_in(name, *p);
  return rc;
}

void *dlsym(void *h, const char *name) {
  return stand_in(name, next_dlsym(h, name));
}
"""


def child(tmp_path, code, **env):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                       timeout=200, env=dict(os.environ, LD_PRELOAD=str(so), **env))
    assert r.returncode == 0, (r.stdout, r.stderr)
    return r


PLAIN = """
import numpy as np
import madmax_b200 as mb
from oracle import oracle as O
d = mb.rve_desc(6, 0.2, (1e9, 2e10), (0.3, 0.2))
eps = np.random.default_rng(1).normal(0, 1e-3, (6, 6))
_, st, _, info = mb.Rve(d).homogenize(eps, rtol=1e-10)
m = O.cube_mesh(6)
ref = O.homogenize(m, O.fiber_types(m, [1, 1], d.radius), tuple(d.E), tuple(d.nu), eps, rtol=1e-12,
                   lin_rtol=1e-13)[1]
assert info.status == 0 and info.pad > 3 * info.inner_its, (info.status, info.pad, info.inner_its)
assert np.abs(st - ref).max() <= 1e-8 * np.abs(ref).max()
"""


def test_plain_solve_without_cooperative_launches(tmp_path):
    """The graph of small kernels (three launches an iteration) solves it."""
    r = child(tmp_path, PLAIN, REFUSE_COOPERATIVE="1")
    assert "refused a cooperative launch" in r.stderr


SPMV = """
import ctypes as C
import numpy as np
import madmax_b200 as mb
from oracle import oracle as O
A = O.assemble(O.cube_mesh(13), np.zeros(13 ** 3, np.uint8), (1e9, 1e9), (0.3, 0.3))
n, w = A.cols.shape
B = mb.EllMatrix(n, n, w)
B.cols[:], B.vals[:] = A.cols, A.vals
h = mb._vp()
mb.check(mb.lib().sp_ell_upload(C.byref(B.m), C.byref(h)), "sp_ell_upload")
x = np.random.default_rng(2).standard_normal(n)
y = np.zeros(n)
mb.check(mb.lib().sp_ell_dev_mvp_host(h, mb.ptr(x), mb.ptr(y)), "sp_ell_dev_mvp_host")
ref = A.mvp(x)
assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()
"""


def test_upload_without_room_for_the_neighbour_lists(tmp_path):
    """n = 13: 14^3 nodes with 28 neighbours of 4 bytes.  The row kernel takes
    the matrix."""
    n = 14 ** 3 * 28 * 4
    r = child(tmp_path, SPMV, REFUSE_BYTES=str(n))
    assert "refused %d bytes" % n in r.stderr
