"""The plain FP64 kernels (po_fp64.cu) against the FP64 oracle where their
blocks, chunks and transposes can go wrong: point counts around the thread
block (128), the shared-memory tile (64) and the chunk and flush width (16),
with and without magnetic currents, both time directions, and every subset of
the gradients. The tolerance is the repository's for FP64 (the same formulas
in another order: 1e-10)."""
import numpy as np
import pytest

from tests.common import FP64_TOL, rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (15, 129), (16, 16), (17, 127), (63, 65), (64, 128), (129, 257), (700, 33), (5, 1300)]


def _case(ns, nt, mode, m_zero, seed):
    """A shallow cup of sources facing targets 3 mm above, lambda 0.2 mm (kR ~ 100 rad)."""
    rng = np.random.default_rng(seed)
    s7 = np.zeros((7, ns))
    s7[0:2] = rng.uniform(-1, 1, (2, ns))
    s7[2] = 0.1 * (s7[0] ** 2 + s7[1] ** 2)
    n = np.stack([-0.2 * s7[0], -0.2 * s7[1], np.ones(ns)])
    s7[3:6] = n / np.linalg.norm(n, axis=0)
    s7[6] = rng.uniform(0.5, 1.5, ns) / ns
    t7 = np.zeros((7, nt))
    if mode == "FF":
        t7[0], t7[1] = rng.uniform(0, 0.3, nt), rng.uniform(-3, 3, nt)
    else:
        t7[0:2] = rng.uniform(-1, 1, (2, nt))
        t7[2] = 3.0 + rng.uniform(-0.3, 0.3, nt)
        t7[5] = -1.0
    t7[6] = 1.0
    cur = rng.standard_normal((2 if mode == "scalar" else 12, ns))
    if m_zero and mode != "scalar":
        cur[6:] = 0.0
    return rng, s7, t7, cur, 2 * np.pi / 0.2


@pytest.mark.parametrize("ns,nt", SIZES)
@pytest.mark.parametrize("mode,m_zero,t", [("EH", True, -1.0), ("JMEH", False, 1.0), ("FF", True, 1.0),
                                           ("FF", False, -1.0), ("scalar", True, -1.0)])
def test_fp64_forward_and_adjoint_against_oracle(cuda, lib, oracle_mod, ns, nt, mode, m_zero, t):
    import torch
    from pypo_gb300 import engine
    rng, s7, t7, cur, k = _case(ns, nt, mode, m_zero, 100 * ns + nt)
    ref = oracle_mod.run(mode, s7, cur, -1, 0, 0, t7, k, 1.0, t)
    dev = [torch.tensor(v, device=cuda) for v in (s7, cur, t7)]
    out = engine.propagate_dev(mode, dev[0], dev[1], -1, 0, 0, dev[2], k, 1.0, t, "fp64", m_zero=m_zero)
    assert rel_l2(out.cpu().numpy(), ref) <= FP64_TOL
    cot = rng.standard_normal(ref.shape)
    want = oracle_mod.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, 1.0, t)
    got = engine.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, 1.0, t, "fp64")
    for name, v in got.items():
        assert rel_l2(v, want[name]) <= FP64_TOL, name
    # a subset of the gradients runs another instantiation: the same values
    for subset in (("cur",), ("ds",)) + (() if mode == "FF" else (("dt",), ("cur", "dt"))):
        part = engine.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, 1.0, t, "fp64", want=subset)
        for name in subset:
            assert rel_l2(part[name], want[name]) <= FP64_TOL, (subset, name)


def test_fp64_long_phases_against_oracle(cuda, lib, oracle_mod):
    """kR ~ 2e6 rad: the quarter-turn reduction with 2/pi in two parts. One
    rounding of R or k R is 2e6 2^-53 ~ 2e-10 rad there, so the bar is 1e-9."""
    from pypo_gb300 import engine
    rng, s7, t7, cur, _ = _case(70, 40, "EH", False, 9)
    k = 2 * np.pi / 1e-5
    ref = oracle_mod.run("EH", s7, cur, -1, 0, 0, t7, k)
    got = engine.propagate("EH", s7, cur, -1, 0, 0, t7, k, precision="fp64")
    assert rel_l2(got, ref) <= 1e-9
