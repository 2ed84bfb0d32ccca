"""The workers that pack large batches: with all of them, and in a process that may start no thread (or only some)."""
import os
import pathlib
import subprocess
import sys

import pytest

from conftest import load_package

CHILD = """
import ctypes, sys
fn = ctypes.CDLL(sys.argv[1]).cubbs_bbs_gpu_pack_pool_for_test_v2
fn.argtypes, fn.restype = [ctypes.c_size_t, ctypes.c_void_p], ctypes.c_int32
for n in (0, 1, 16, 1000):
    s = ctypes.c_uint64(1)
    assert fn(n, ctypes.byref(s)) == 0 and s.value == n * (n + 1) // 2, n
print("packed")
"""
REFUSE = """
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
  static int left = ALLOWED;
  if (left-- <= 0) return EAGAIN;
  int (*real)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *) = dlsym(RTLD_NEXT, "pthread_create");
  return real(t, a, f, x);
}
"""


@pytest.mark.parametrize("allowed", [None, 0, 2])
def test_packing_without_threads(tmp_path, allowed):
    env = dict(os.environ)
    if allowed is not None:
        src, lib = tmp_path / "refuse.c", tmp_path / "refuse.so"
        src.write_text(REFUSE)
        subprocess.run(["gcc", "-shared", "-fPIC", "-DALLOWED=%d" % allowed, str(src), "-o", str(lib), "-ldl"], check=True)
        env["LD_PRELOAD"] = str(lib)
    path = pathlib.Path(load_package().build())
    out = subprocess.run([sys.executable, "-c", CHILD, str(path)], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "packed", (out.returncode, out.stderr[-1000:])
