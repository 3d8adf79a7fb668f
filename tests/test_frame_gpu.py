"""The frame of the mixed path (po_prep.cu) on both sides of the count where it
comes from two kernels instead of one cluster (60,000 points), around a point a
thread of 152 CTAs (77,824), with either side the more numerous: the frame's
half-extent is the points' box's, exactly, the fields are those of the FP64 sum
at the mixed path's bar, and the list of near-tangent pairs starts empty."""
import numpy as np
import pytest

from tests.common import REL_L2_TOL, rel_l2

pytestmark = pytest.mark.gpu

K = 20.0


def _case(ns, nt, seed):
    rng = np.random.default_rng(seed)
    s7, t7 = np.zeros((7, ns)), np.zeros((7, nt))
    s7[0:2], s7[5], s7[6] = rng.uniform(-1, 1, (2, ns)), 1.0, 1.0 / ns
    t7[0:2], t7[2], t7[5], t7[6] = rng.uniform(-1, 1, (2, nt)), rng.uniform(3, 4, nt), -1.0, 1.0
    # the box's faces at the first and the last point of either side
    s7[0, -1], s7[1, 0], t7[0, -1], t7[1, 0], t7[2, nt // 2] = 1.5, -1.25, -1.75, 1.25, 4.5
    return s7, t7, rng.standard_normal((12, ns))


def _extent(p):
    lo, hi = p.min(axis=1), p.max(axis=1)
    o = 0.5 * (lo + hi)
    return max(np.abs(hi - o).max(), np.abs(lo - o).max()) * (K / (2.0 * np.pi))


@pytest.mark.parametrize("ns,nt", [(59995, 5), (59996, 5), (5, 59996), (30000, 30001), (77819, 5), (77820, 5),
                                   (40, 77785), (200003, 7)])
@pytest.mark.parametrize("mode,m_zero", [("EH", True), ("JM", False), ("scalar", True)])
def test_near_field(cuda, lib, ns, nt, mode, m_zero):
    from pypo_gb300 import engine
    s7, t7, cur = _case(ns, nt, ns + nt)
    if mode == "scalar":
        cur = cur[:2]
    elif m_zero:
        cur[6:] = 0.0
    got = engine.propagate(mode, s7, cur, -1, 0, 0, t7, K)
    assert engine.last_extent() == pytest.approx(_extent(np.concatenate([s7[0:3], t7[0:3]], axis=1)), rel=1e-14)
    some = np.unique(np.concatenate([np.arange(min(nt, 40)), [nt // 2, nt - 1]]))
    want = engine.propagate(mode, s7, cur, -1, 0, 0, np.ascontiguousarray(t7[:, some]), K, precision="fp64")
    assert rel_l2(got[:, some], want) <= REL_L2_TOL
    cot = np.random.default_rng(nt).standard_normal((engine.n_out(mode), nt))
    if ns * nt < 2e6:
        want = engine.adjoint(mode, s7, cur, -1, 0, 0, t7, K, cot, precision="fp64")
        for name, v in engine.adjoint(mode, s7, cur, -1, 0, 0, t7, K, cot).items():
            assert rel_l2(v, want[name]) <= REL_L2_TOL, name


@pytest.mark.parametrize("ns", [60000, 60001, 77824, 77825])
def test_far_field(cuda, lib, ns):
    from pypo_gb300 import engine
    s7, t7, cur = _case(ns, 9, ns)
    cur[6:] = 0.0
    t7[0], t7[1], t7[2:] = np.linspace(0.0, 0.3, 9), np.linspace(-3.0, 3.0, 9), 0.0
    got = engine.propagate("FF", s7, cur, -1, 0, 0, t7, K)
    assert engine.last_extent() == pytest.approx(np.abs(s7[0:3]).max() * (K / (2.0 * np.pi)), rel=1e-14)
    assert rel_l2(got, engine.propagate("FF", s7, cur, -1, 0, 0, t7, K, precision="fp64")) <= REL_L2_TOL
    cot = np.random.default_rng(1).standard_normal((12, 9))
    want = engine.adjoint("FF", s7, cur, -1, 0, 0, t7, K, cot, precision="fp64")
    for name, v in engine.adjoint("FF", s7, cur, -1, 0, 0, t7, K, cot).items():
        assert rel_l2(v, want[name]) <= REL_L2_TOL, name


@pytest.mark.parametrize("ns", [59996, 60001])
def test_missing_points_are_left_out_and_the_pair_list_is_cleared(cuda, lib, ns):
    """A NaN coordinate does not move the box; targets in the sources' plane
    put every pair into the list, the same number in each call."""
    from pypo_gb300 import engine
    s7, t7, cur = _case(ns, 5, 3)
    t7[2] = 0.0
    for _ in range(2):
        engine.propagate("EH", s7, cur, -1, 0, 0, t7, K)
        assert engine.last_band_pairs() == 5 * ns
    s7[0, 17] = np.nan
    engine.propagate("EH", s7, cur, -1, 0, 0, t7, K)
    keep = np.delete(s7, 17, axis=1)
    assert engine.last_extent() == pytest.approx(_extent(np.concatenate([keep[0:3], t7[0:3]], axis=1)), rel=1e-14)
