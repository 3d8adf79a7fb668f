"""The set-up and epilogue kernels of the mixed forward (po_prep.cu, the
chunk groups of po_epilogue_kernel) against the oracle at the counts where
they can go wrong: sources around the tile of 128 and the frame cluster's
stride (16 x 512), and few targets with chunk counts around 8, 32 and 64,
where the epilogue changes the threads that share a target. The bar is the
mixed path's."""
import numpy as np
import pytest

from tests.common import PHASE_TOL, REL_L2_TOL, errors

pytestmark = pytest.mark.gpu


def _case(ns, nt, seed):
    rng = np.random.default_rng(seed)
    s7 = np.zeros((7, ns))
    s7[0:2] = rng.uniform(-1, 1, (2, ns))
    s7[2] = 0.1 * (s7[0] ** 2 + s7[1] ** 2)
    n = np.stack([-0.2 * s7[0], -0.2 * s7[1], np.ones(ns)])
    s7[3:6] = n / np.linalg.norm(n, axis=0)
    s7[6] = 1.0 / ns
    t7 = np.zeros((7, nt))
    t7[0:2] = rng.uniform(-1, 1, (2, nt))
    t7[2] = 3.0
    t7[5] = -1.0
    t7[6] = 1.0
    return s7, t7, rng.standard_normal((12, ns))


@pytest.mark.parametrize("ns,nt", [(1, 1), (127, 3), (128, 255), (129, 257), (7 * 128 + 1, 31), (31 * 128, 32),
                                   (32 * 128 + 1, 33), (63 * 128, 5), (8191, 8), (8192, 609), (8193, 1217),
                                   (64 * 128 + 127, 4)])
@pytest.mark.parametrize("mode,m_zero", [("EH", True), ("JM", False), ("scalar", True)])
def test_counts_against_oracle(cuda, lib, oracle_mod, ns, nt, mode, m_zero):
    from pypo_gb300 import engine
    s7, t7, cur = _case(ns, nt, ns + nt)
    if mode == "scalar":
        cur = cur[:2]
    elif m_zero:
        cur[6:] = 0.0
    got = engine.propagate(mode, s7, cur, -1, 0, 0, t7, 20.0)
    e, p = errors(got, oracle_mod.run(mode, s7, cur, -1, 0, 0, t7, 20.0), mode)
    assert e <= REL_L2_TOL and p <= PHASE_TOL, (e, p)


@pytest.mark.parametrize("shift", [0.0, 1e4, -3e-7])
def test_frame_matches_the_points_box(cuda, lib, shift):
    """The frame's half-extent: half the largest side of the points' box, in
    wavelengths, exactly (minima and maxima of coordinates of either sign)."""
    from pypo_gb300 import engine
    s7, t7, cur = _case(5000, 77, 3)
    s7[0:3] += shift
    t7[0:3] += shift
    engine.propagate("EH", s7, cur, -1, 0, 0, t7, 20.0)
    pts = np.concatenate([s7[0:3], t7[0:3]], axis=1)
    lo, hi = pts.min(axis=1), pts.max(axis=1)
    o = 0.5 * (lo + hi)
    want = max(np.abs(hi - o).max(), np.abs(lo - o).max()) * (20.0 / (2.0 * np.pi))
    assert engine.last_extent() == pytest.approx(want, rel=1e-14)


@pytest.mark.parametrize("ns,nt", [(1, 1), (1, 700), (31, 513), (33, 575), (32, 1025), (129, 2000), (2000, 3)])
@pytest.mark.parametrize("mode,m_zero", [("EH", True), ("JMEH", False), ("scalar", True)])
def test_adjoint_counts_against_oracle(cuda, lib, oracle_mod, ns, nt, mode, m_zero):
    """Few sources with chunk counts around 8, where the adjoint's epilogue
    changes the threads that share a source; odd target counts (a padded pair)."""
    from pypo_gb300 import engine
    s7, t7, cur = _case(ns, nt, 7 * ns + nt)
    if mode == "scalar":
        cur = cur[:2]
    elif m_zero:
        cur[6:] = 0.0
    cot = np.random.default_rng(nt).standard_normal((engine.n_out(mode), nt))
    want = oracle_mod.adjoint(mode, s7, cur, -1, 0, 0, t7, 20.0, cot)
    got = engine.adjoint(mode, s7, cur, -1, 0, 0, t7, 20.0, cot)
    for name, v in want.items():
        assert np.linalg.norm(got[name] - v) <= REL_L2_TOL * np.linalg.norm(v), name
