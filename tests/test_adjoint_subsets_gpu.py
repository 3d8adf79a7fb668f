"""The adjoint's kernels leave out the accumulators of gradients that are not
asked for: every subset of the gradients, mixed and FP64, against the FP64
oracle, at counts around the tiles (128 sources, 64 target pairs), with a
coplanar part whose pairs are tangent (the mixed path's FP64 fix-up adds to
the same rows). The bar is each path's own."""
import itertools

import numpy as np
import pytest

from tests.common import REL_L2_TOL, rel_l2

pytestmark = pytest.mark.gpu
NAMES = ("cur", "ds", "dt")


def _case(ns, nt, n_cur, seed):
    rng = np.random.default_rng(seed)
    s7, t7 = np.zeros((7, ns)), np.zeros((7, nt))
    s7[0:2] = rng.uniform(-2, 2, (2, ns))
    n = np.stack([0.2 * s7[0], 0.2 * s7[1], np.ones(ns)])
    n[:2, ::5] = 0.0
    s7[3:6] = n / np.linalg.norm(n, axis=0)
    s7[6] = 1.0 / ns
    t7[0:2], t7[2] = rng.uniform(-2, 2, (2, nt)), rng.uniform(3, 6, nt)
    t7[0, 3::9], t7[2, 3::9] = 5.0 + t7[0, 3::9], 0.0   # in the plane of the sources, beside them
    t7[5] = -1.0
    t7[6] = 1.0
    return rng, s7, t7, rng.standard_normal((n_cur, ns))


@pytest.mark.parametrize("precision,tol", [("mixed", REL_L2_TOL), ("fp64", 1e-9)])
@pytest.mark.parametrize("mode,m_zero", [("EH", True), ("JM", False), ("JMEH", False), ("scalar", True)])
@pytest.mark.parametrize("ns,nt", [(1, 1), (127, 129), (300, 40), (129, 1001)])
def test_subsets_against_oracle(cuda, lib, oracle_mod, mode, m_zero, ns, nt, precision, tol):
    from pypo_gb300 import engine
    rng, s7, t7, cur = _case(ns, nt, 2 if mode == "scalar" else 12, 7 * ns + nt)
    if m_zero and mode != "scalar":
        cur[6:] = 0.0
    k = 2 * np.pi
    cot = rng.standard_normal((engine.n_out(mode), nt))
    want = oracle_mod.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot)
    for r in (1, 2, 3):
        for names in itertools.combinations(NAMES, r):
            got = engine.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, precision=precision, want=names)
            for name in names:
                assert rel_l2(got[name], want[name]) <= tol, (names, name)
