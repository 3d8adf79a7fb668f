"""The near-field forward's variant for grids of at most two CTAs an SM: 2,432
sources (19 tiles) and 2,048 targets (16 blocks) are 304 CTAs, the last such
grid of 152 SMs; one target more takes the general kernel. The tiles' sums are
added in the same order, so the shared targets' fields are the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,m_zero,t", [("EH", True, -1.0), ("EH", True, 1.0), ("JMEH", False, -1.0),
                                           ("JMEH", False, 1.0)])
def test_equals_the_general_kernel(cuda, lib, mode, m_zero, t):
    from pypo_gb300 import engine
    rng = np.random.default_rng(2)
    ns, nt = 2432, 2049
    s7, t7 = np.zeros((7, ns)), np.zeros((7, nt))
    s7[0:2], s7[5], s7[6] = rng.uniform(-30, 30, (2, ns)), 1.0, 1.0 / ns
    t7[0:2], t7[2], t7[5], t7[6] = rng.uniform(-20, 20, (2, nt)), rng.uniform(40, 60, nt), -1.0, 1.0
    t7[0, ::50], t7[2, ::50] = 35.0, 0.0     # tangent pairs
    t7[0:3, -1] = [0.0, 0.0, 50.0]           # inside the others' box: the same frame
    cur = rng.standard_normal((12, ns))
    if m_zero:
        cur[6:] = 0.0
    k = 2 * np.pi
    many = engine.propagate(mode, s7, cur, -1, 0, 0, t7, k, 1.0, t)
    few = engine.propagate(mode, s7, cur, -1, 0, 0, np.ascontiguousarray(t7[:, :-1]), k, 1.0, t)
    tangent = np.zeros(nt - 1, bool)
    tangent[::50] = True                     # their FP64 terms are added in no fixed order
    np.testing.assert_array_equal(few[:, ~tangent], many[:, :-1][:, ~tangent])
    np.testing.assert_allclose(few[:, tangent], many[:, :-1][:, tangent], rtol=1e-12,
                               atol=1e-13 * np.abs(few).max())
