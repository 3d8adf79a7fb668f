"""po_device_error allocates nothing (include/po_gb300.h), on any thread: the
CUDA runtime's allocating calls are counted by a preloaded stand-in that
passes them on. Without a GPU the calls fail, and are counted all the same."""
import os
import pathlib
import shutil
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int allocations = 0;
static void *real(const char *name)
{
    void *h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    return h ? dlsym(h, name) : NULL;
}
#define COUNTED(name, params, args)                                  \
    int name params                                                  \
    {                                                                \
        __atomic_add_fetch(&allocations, 1, __ATOMIC_SEQ_CST);       \
        int (*call) params = (int (*) params)real(#name);            \
        return call ? call args : 2;                                 \
    }
COUNTED(cudaMalloc, (void **p, size_t n), (p, n))
COUNTED(cudaMallocHost, (void **p, size_t n), (p, n))
COUNTED(cudaHostAlloc, (void **p, size_t n, unsigned f), (p, n, f))
COUNTED(cudaMallocAsync, (void **p, size_t n, void *s), (p, n, s))
COUNTED(cudaMallocFromPoolAsync, (void **p, size_t n, void *q, void *s), (p, n, q, s))
"""

RUN = r"""
import ctypes, sys, threading
from pypo_gb300 import _lib
lib = _lib.load()
count = ctypes.c_int.in_dll(ctypes.CDLL(sys.argv[1]), "allocations")
def call():
    code = ctypes.c_int(-1)
    lib.po_device_error(None, ctypes.byref(code))
for _ in range(3):
    t = threading.Thread(target=call)
    t.start()
    t.join()
print("allocations", count.value)
"""


@pytest.mark.parametrize("where", ["cpu", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_allocates_nothing(lib, tmp_path, where):
    cc = shutil.which("gcc")
    if not cc:
        pytest.skip("no gcc")
    (tmp_path / "count.c").write_text(COUNT)
    so = tmp_path / "count.so"
    subprocess.run([cc, "-shared", "-fPIC", "-o", so, tmp_path / "count.c", "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", RUN, str(so)], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == ["allocations", "0"]
