"""The FP64 path's illumination decision (po_fp64.cu) where it passes from the
exponents to the comparisons and to the reference's own rounding: n . d from
0 to 1e-9 R on either side, forward and adjoint, near and far field, against
the oracle, whose decision is the reference's."""
import numpy as np
import pytest

from tests.common import rel_l2

pytestmark = pytest.mark.gpu
STEPS = np.array([0.0, 1e-17, 3e-16, 1e-13, 4e-13, 9e-13, 1e-12, 1.1e-12, 1.8e-12, 2e-12, 3.7e-12, 8e-12, 1e-9])


@pytest.mark.parametrize("mode", ["EH", "FF"])
@pytest.mark.parametrize("scale", [1.0, 0.75, 1.9, 1000.0])
def test_decision_against_oracle(cuda, lib, oracle_mod, mode, scale):
    from pypo_gb300 import engine
    h = np.concatenate([STEPS, -STEPS])
    s7 = np.zeros((7, 3))
    s7[0] = [0.0, 0.3 * scale, -0.2 * scale]
    s7[5], s7[6] = 1.0, 0.25
    t7 = np.zeros((7, h.size))
    if mode == "FF":
        t7[0] = np.pi / 2 - h          # n . r = sin(h)
        t7[1] = np.linspace(-1.0, 1.0, h.size)
    else:
        t7[0], t7[2] = 5.0 * scale, 5.0 * scale * h
        t7[5], t7[6] = -1.0, 1.0
    rng = np.random.default_rng(1)
    cur = rng.standard_normal((12, 3))
    k = 2 * np.pi
    want = oracle_mod.run(mode, s7, cur, -1, 0, 0, t7, k)
    got = engine.propagate(mode, s7, cur, -1, 0, 0, t7, k, precision="fp64")
    for j in range(h.size):   # each target by itself: a wrong decision is of order 1
        assert rel_l2(got[:, j], want[:, j]) <= 1e-9, (h[j], j)
    cot = rng.standard_normal((12, h.size))
    w = oracle_mod.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot)
    g = engine.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, precision="fp64",
                       want=("cur", "ds") if mode == "FF" else ("cur", "ds", "dt"))
    for name in g:
        assert rel_l2(g[name], w[name]) <= 1e-9, name
