"""The far-field adjoint kernel (po_ff_adjoint.cu) against the FP64 oracle at
the counts where its stages and tiles can go wrong: directions around a stage
(64) and an odd one left over, sources around a tile (128) and an odd one,
several chunks of stages, with and without magnetic currents, a subset of the
gradients, and sources facing away from part of the directions. The bar is the
mixed path's."""
import numpy as np
import pytest

from tests.common import REL_L2_TOL, rel_l2

pytestmark = pytest.mark.gpu


def _case(ns, nt, seed, spread):
    rng = np.random.default_rng(seed)
    s7 = np.zeros((7, ns))
    s7[0:2] = rng.uniform(-spread, spread, (2, ns))
    s7[2] = 0.1 * (s7[0] ** 2 + s7[1] ** 2) / spread
    n = np.stack([-0.4 * s7[0] / spread, -0.4 * s7[1] / spread, np.ones(ns)])
    s7[3:6] = n / np.linalg.norm(n, axis=0)
    s7[6] = 1.0 / ns
    t7 = np.zeros((7, nt))
    t7[0], t7[1] = rng.uniform(0, 0.1, nt), rng.uniform(-3, 3, nt)
    t7[0, ::7] += np.pi / 2 + 0.3   # beyond the horizon of most sources
    return rng, s7, t7, rng.standard_normal((12, ns))


@pytest.mark.parametrize("ns,nt", [(1, 1), (2, 63), (127, 64), (128, 65), (129, 127), (255, 128), (1300, 129),
                                   (40, 3001)])
@pytest.mark.parametrize("m_zero,t,spread", [(True, -1.0, 1.0), (False, 1.0, 1.0), (True, 1.0, 300.0)])
def test_against_oracle_adjoint(cuda, lib, oracle_mod, ns, nt, m_zero, t, spread):
    """spread 300 mm at lambda 1 mm: tiles past 64 turns take the split phase."""
    from pypo_gb300 import engine
    rng, s7, t7, cur = _case(ns, nt, 10 * ns + nt, spread)
    if m_zero:
        cur[6:] = 0.0
    k = 2 * np.pi
    cot = rng.standard_normal((12, nt))
    want = oracle_mod.adjoint("FF", s7, cur, -1, 0, 0, t7, k, cot, 1.0, t)
    got = engine.adjoint("FF", s7, cur, -1, 0, 0, t7, k, cot, 1.0, t)
    for name in ("cur", "ds"):
        assert rel_l2(got[name], want[name]) <= REL_L2_TOL, name
    for name in ("cur", "ds"):
        part = engine.adjoint("FF", s7, cur, -1, 0, 0, t7, k, cot, 1.0, t, want=(name,))
        assert rel_l2(part[name], want[name]) <= REL_L2_TOL, name
