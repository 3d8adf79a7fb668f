"""The drop-in calls (callKernelf_*) past their page-locked staging, where the
caller's rows are copied one by one and the device checks for M = 0, and on
several threads at once."""
import ctypes
import os
import pathlib
import shutil
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent


def _call(lib, mode, src, tgt, vals, k):
    from pypo_gb300 import Structs as S, marshal as M
    f = ctypes.c_float
    csp, _k1 = M.fill_reflparams(src, f)
    ctp, _k2 = M.fill_reflparams(tgt, f)
    cs, sblock = M.alloc_container(int(np.prod(src["gridsize"])), f)
    ct, tblock = M.alloc_container(int(np.prod(tgt["gridsize"])), f)
    cin = M.bundle(S.arrC1f if mode == "scalar" else S.c2Bundlef, vals, f)
    out = np.zeros((S.N_OUT[mode], tblock.shape[1]), dtype=np.float32)
    res = M.bundle(S.BUNDLE_F[mode], out, f)
    rc = getattr(lib, f"callKernelf_{mode}")(ctypes.byref(res), csp, ctp, ctypes.byref(cs), ctypes.byref(ct),
                                             ctypes.byref(cin), f(k), f(1.0), f(-1.0), 1, 256)
    assert rc == 0, lib.po_last_error()
    return out, sblock, tblock


@pytest.mark.parametrize("mode,m_zero", [("EH", True), ("JM", False), ("scalar", True)])
@pytest.mark.parametrize("ns,nt", [((13, 11), (421, 419)), ((421, 419), (9, 8)), ((421, 421), (421, 420)), ((13, 11), (9, 8))])
def test_rows_and_grids_past_the_staging(cuda, lib, mode, m_zero, ns, nt):
    """12 rows of 421 x 419 floats are 8.5 MB, past the 8 MiB block (the
    scalar mode's with both grids as well, in the third pair). The call is the
    device entries' on the same grids, narrowed to float: the same bits."""
    import torch
    from pypo_gb300 import engine, surfaces
    rng = np.random.default_rng(1)
    src = surfaces.plane(ns, gmode=0, lims_a=[-16.0, 16.0])
    tgt = surfaces.translate(surfaces.plane(nt, gmode=0, lims_a=[-8.0, 8.0]), dz=64.0)
    k = float(np.float32(2.0 * np.pi / 3.0))
    vals = rng.standard_normal((2 if mode == "scalar" else 12, ns[0] * ns[1])).astype(np.float32)
    if m_zero and mode != "scalar":
        vals[6:] = 0.0
    out, sblock, tblock = _call(lib, mode, src, tgt, vals, k)
    s7, t7 = engine.generate_grid_dev(src), engine.generate_grid_dev(tgt)
    want = engine.propagate_dev(mode, s7, torch.from_numpy(vals).double().cuda(), 0, *ns, t7, k,
                                m_zero=m_zero and mode != "scalar")
    np.testing.assert_array_equal(out, want.float().cpu().numpy())
    np.testing.assert_array_equal(sblock, s7.float().cpu().numpy())
    np.testing.assert_array_equal(tblock, t7.float().cpu().numpy())


COUNT = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int blocks = 0, frees = 0;
static void *real(const char *name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), name); }
int cudaHostAlloc(void **p, size_t n, unsigned f)
{
    if (n >= (1u << 20)) __atomic_add_fetch(&blocks, 1, __ATOMIC_SEQ_CST);
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
import numpy as np
from pypo_gb300 import BindGPU, PyPOTypes, surfaces
shim = ctypes.CDLL(sys.argv[1])
src = surfaces.plane([61, 61], gmode=0, lims_a=[-16.0, 16.0])
tgt = surfaces.translate(surfaces.plane([101, 101], gmode=0, lims_a=[-8.0, 8.0]), dz=64.0)
def job(seed):
    g = np.random.default_rng(seed)
    cur = PyPOTypes.currents(*[g.standard_normal((61, 61)) + 1j * g.standard_normal((61, 61)) for _ in range(6)])
    e = BindGPU.PyPO_GPUf(src, tgt, dict(mode="EH", k=2.0, s_current=cur))
    return np.stack([e[i] for i in range(6)])
want = [job(i) for i in range(8)]
bad = []
start = threading.Barrier(8)
def work(i):
    start.wait()
    for _ in range(12):
        if not np.array_equal(job(i), want[i]):
            bad.append(i)
threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
for t in threads: t.start()
for t in threads: t.join()
print(len(bad), ctypes.c_int.in_dll(shim, "blocks").value, ctypes.c_int.in_dll(shim, "frees").value)
"""


def test_eight_threads(cuda, lib, tmp_path):
    """The same results as one after the other, and a bounded set of staging
    blocks: at most four are made, and none is freed (which waits for the
    device) while calls run. A call that finds none copies its rows directly."""
    cc = shutil.which("gcc")
    if not cc:
        pytest.skip("no gcc")
    (tmp_path / "count.c").write_text(COUNT)
    so = tmp_path / "count.so"
    subprocess.run([cc, "-shared", "-fPIC", "-o", so, tmp_path / "count.c", "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", RUN, str(so)], env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    bad, blocks, frees = (int(v) for v in r.stdout.split())
    assert bad == 0 and 1 <= blocks <= 4 and frees == 0, r.stdout
