"""More fits at the same time than there are page-locked result boxes (16):
the same parameters as one after the other, and no box is made and freed for
one fit (freeing page-locked memory waits for the device); a fit without one
copies its results."""
import os
import pathlib
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent

COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int boxes = 0, frees = 0;
static void *real(const char *name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaHostAlloc(void **p, size_t n, unsigned f)
{
    if (n <= 4096) __atomic_add_fetch(&boxes, 1, __ATOMIC_SEQ_CST);
    return ((int (*)(void **, size_t, unsigned))real("cudaHostAlloc"))(p, n, f);
}
int cudaFreeHost(void *p)
{
    __atomic_add_fetch(&frees, 1, __ATOMIC_SEQ_CST);
    return ((int (*)(void *))real("cudaFreeHost"))(p);
}
"""

RUN = r"""
import ctypes, sys, threading
import numpy as np, torch
from pypo_gb300 import fitgauss as FG
shim = ctypes.CDLL(sys.argv[1])
n, N = 41, 28
ax = np.linspace(-0.5, 0.5, n)
x, y = (v.ravel() for v in np.meshgrid(ax, ax, indexing="ij"))
g7 = torch.zeros((7, n * n), dtype=torch.float64)
g7[0], g7[1] = torch.from_numpy(x), torch.from_numpy(y)
g7 = g7.cuda()
amps = [torch.from_numpy(np.exp(-(x**2 + (1 + 0.02 * k) * y**2) / (2 * 0.1**2))).cuda() for k in range(N)]
streams = [torch.cuda.Stream() for _ in range(N)]
fit = lambda k: FG.fit_gauss_abs_dev(g7, n, n, amps[k], None, -11.0, "LIN", None)
want = [fit(k) for k in range(N)]
torch.cuda.synchronize()
start, bad = threading.Barrier(N), []
def work(k):
    start.wait()
    with torch.cuda.stream(streams[k]):
        for _ in range(6):
            if not np.array_equal(fit(k), want[k]):
                bad.append(k)
threads = [threading.Thread(target=work, args=(k,)) for k in range(N)]
for t in threads: t.start()
for t in threads: t.join()
print(len(bad), ctypes.c_int.in_dll(shim, "boxes").value, ctypes.c_int.in_dll(shim, "frees").value)
"""


def test_more_fits_than_boxes(cuda, lib, tmp_path):
    cc = shutil.which("gcc")
    if not cc:
        pytest.skip("no gcc")
    (tmp_path / "count.c").write_text(COUNT)
    so = tmp_path / "count.so"
    subprocess.run([cc, "-shared", "-fPIC", "-o", so, tmp_path / "count.c", "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", RUN, str(so)], env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    bad, boxes, frees = (int(v) for v in r.stdout.split())
    assert bad == 0 and 1 <= boxes <= 16 and frees == 0, r.stdout
