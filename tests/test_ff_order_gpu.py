"""The far field's source order for few sources (po_ff_rank_kernel): against
the radix sort, bit for bit, where the rule passes from one to the other, and
against the FP64 oracle at counts around its CTAs (32 sources) and tiles
(2,048), with coincident sources (equal keys)."""
import numpy as np
import pytest

from tests.common import PHASE_TOL, REL_L2_TOL, errors, rel_l2

pytestmark = pytest.mark.gpu
RANK_MAX = 20000


def _case(ns, nt, seed):
    rng = np.random.default_rng(seed)
    s7 = np.zeros((7, ns))
    s7[0], s7[1] = rng.uniform(-20.0, 20.0, ns), rng.uniform(-15.0, 15.0, ns)
    s7[5], s7[6] = 1.0, 1.0 / ns
    t7 = np.zeros((7, nt))
    t7[0], t7[1] = rng.uniform(0, 0.3, nt), rng.uniform(-3, 3, nt)
    return rng, s7, t7, rng.standard_normal((12, ns))


@pytest.mark.parametrize("m_zero", [True, False])
def test_equals_the_sort(cuda, lib, m_zero):
    """The last source on the curve (the corner of the box where it ends) once
    more, without currents: one source more takes the sort, and fills a place
    of the last tile that a copy of that source pads otherwise."""
    from pypo_gb300 import engine
    rng, s7, t7, cur = _case(RANK_MAX, 70, 5)
    if m_zero:
        cur[6:] = 0.0
    s7[0, 777], s7[1, 777] = 21.0, -16.0
    s7[0, 1234], s7[1, 1234] = -21.0, 16.0
    s7[:2, 4001] = s7[:2, 4000]   # equal keys
    more = np.concatenate([s7, s7[:, 777:778]], axis=1)
    cur_more = np.concatenate([cur, np.zeros((12, 1))], axis=1)
    k = 2 * np.pi
    a = engine.propagate("FF", s7, cur, -1, 0, 0, t7, k)
    b = engine.propagate("FF", more, cur_more, -1, 0, 0, t7, k)
    np.testing.assert_array_equal(a, b)
    cot = rng.standard_normal((12, 70))
    ga = engine.adjoint("FF", s7, cur, -1, 0, 0, t7, k, cot, want=("cur", "ds"))
    gb = engine.adjoint("FF", more, cur_more, -1, 0, 0, t7, k, cot, want=("cur", "ds"))
    for name in ga:
        np.testing.assert_array_equal(ga[name], gb[name][..., :RANK_MAX])


@pytest.mark.parametrize("ns", [1, 2, 31, 32, 33, 257, 2047, 2048, 2049, 4097])
def test_against_oracle(cuda, lib, oracle_mod, ns):
    from pypo_gb300 import engine
    rng, s7, t7, cur = _case(ns, 33, ns)
    s7[:2, ns // 2:] = s7[:2, :ns - ns // 2]   # coincident sources
    k = 2 * np.pi
    got = engine.propagate("FF", s7, cur, -1, 0, 0, t7, k)
    e, p = errors(got, oracle_mod.run("FF", s7, cur, -1, 0, 0, t7, k), "FF")
    assert e <= REL_L2_TOL and p <= PHASE_TOL, (e, p)
    cot = rng.standard_normal((12, 33))
    g = engine.adjoint("FF", s7, cur, -1, 0, 0, t7, k, cot, want=("cur", "ds"))
    w = oracle_mod.adjoint("FF", s7, cur, -1, 0, 0, t7, k, cot)
    for name in g:
        assert rel_l2(g[name], w[name]) <= REL_L2_TOL, name
