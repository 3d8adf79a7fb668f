"""The near-field and scalar forward kernel (po_kernels.cu) against the FP64
oracle at the counts where its halves can go wrong: tiles with one source
more in the even half, a tile of one source (an empty odd half), targets
around the half block of 64 (a thread's second lane idle), and tangent pairs
in either half and lane (the FP64 fixup's list). The bar is the mixed path's."""
import numpy as np
import pytest

from tests.common import PHASE_TOL, REL_L2_TOL, errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nt", [(1, 64), (2, 65), (3, 63), (129, 128), (130, 127), (255, 192), (257, 64),
                                   (1023, 193)])
@pytest.mark.parametrize("mode,m_zero,tangent", [("EH", True, False), ("EH", True, True), ("JMEH", False, True),
                                                 ("scalar", True, False)])
def test_halves_against_oracle(cuda, lib, oracle_mod, ns, nt, mode, m_zero, tangent):
    from pypo_gb300 import engine
    rng = np.random.default_rng(1000 * ns + nt)
    s7, t7 = np.zeros((7, ns)), np.zeros((7, nt))
    s7[0:2], s7[5], s7[6] = rng.uniform(-3, 3, (2, ns)), 1.0, 1.0 / ns
    t7[0:2], t7[2], t7[5], t7[6] = rng.uniform(-3, 3, (2, nt)), rng.uniform(4, 6, nt), -1.0, 1.0
    if tangent:
        t7[0, ::3], t7[2, ::3] = t7[0, ::3] + 7.0, 0.0   # in the sources' plane, beside them
    cur = rng.standard_normal((2 if mode == "scalar" else 12, ns))
    if m_zero and mode != "scalar":
        cur[6:] = 0.0
    got = engine.propagate(mode, s7, cur, -1, 0, 0, t7, 2 * np.pi)
    if tangent:
        assert engine.last_band_pairs() == ns * len(range(0, nt, 3))
    e, p = errors(got, oracle_mod.run(mode, s7, cur, -1, 0, 0, t7, 2 * np.pi), mode)
    assert e <= REL_L2_TOL and p <= PHASE_TOL, (e, p)
