"""The far-field forward's variant for grids of at most two CTAs an SM: 2,432
sources (19 tiles) and 4,096 directions (16 blocks of 256) are 304 CTAs, the
last such grid of 152 SMs; one direction more takes the general kernel. The
tiles' sums are added in the same order: the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,spread", [(-1.0, 20.0), (1.0, 20.0), (-1.0, 900.0)])
def test_equals_the_general_kernel(cuda, lib, t, spread):
    """spread 900 mm at lambda 1 mm: wide tiles."""
    from pypo_gb300 import engine
    rng = np.random.default_rng(2)
    ns, nt = 2432, 4097
    s7, t7 = np.zeros((7, ns)), np.zeros((7, nt))
    s7[0:2], s7[5], s7[6] = rng.uniform(-spread, spread, (2, ns)), 1.0, 1.0 / ns
    t7[0], t7[1] = rng.uniform(0, 0.2, nt), rng.uniform(-3, 3, nt)
    t7[0, ::7] += np.pi / 2 + 0.3            # beyond the horizon
    cur = rng.standard_normal((12, ns))
    cur[6:] = 0.0
    k = 2 * np.pi
    many = engine.propagate("FF", s7, cur, -1, 0, 0, t7, k, 1.0, t)
    few = engine.propagate("FF", s7, cur, -1, 0, 0, np.ascontiguousarray(t7[:, :-1]), k, 1.0, t)
    np.testing.assert_array_equal(few, many[:, :-1])
