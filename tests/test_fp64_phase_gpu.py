"""Phases of any size in the plain FP64 sums (sincos64, po_fp64.cu): its
reduction with 2/pi in two parts ends at 2^51 rad, past which the general
sincos() takes over. The pairs' distances (or r . s) are whole numbers, so
that k R is one rounding on both sides, and the outputs are a few roundings of
each other: 1e-12 against numpy's sin and cos, and the repository's 1e-10
against the oracle for the vector modes and the gradients."""
import numpy as np
import pytest

from tests.common import FP64_TOL, rel_l2

pytestmark = pytest.mark.gpu

#: around 2^51 = 2.25e15 rad, far past it, and an ordinary one
WAVENUMBERS = [6.0, 1e12, 2.0**51 / 9, 2.0**51, 2.0**51 * 1.5707963267948966, 1e17, 3e22]
#: distances 1, 3, 5, 7, 9 from the origin
POINTS = np.array([[0, 0, 1], [1, 2, 2], [0, 3, 4], [2, 3, 6], [4, 4, 7]], float).T


def _one_source():
    s7 = np.zeros((7, 1))
    s7[5], s7[6] = 1.0, 1.0
    t7 = np.zeros((7, POINTS.shape[1]))
    t7[0:3], t7[5], t7[6] = POINTS, -1.0, 1.0
    return s7, t7


@pytest.mark.parametrize("k", WAVENUMBERS)
@pytest.mark.parametrize("t", [-1.0, 1.0])
def test_scalar_against_numpy(cuda, lib, k, t):
    from pypo_gb300 import engine
    s7, t7 = _one_source()
    got = engine.propagate("scalar", s7, np.array([[1.0], [0.5]]), -1, 0, 0, t7, k, 1.0, t, precision="fp64")
    R = np.sqrt((POINTS**2).sum(0))
    want = -k * k / (4.0 * float(np.float32(3.14159265359))) * (1.0 + 0.5j) * (np.cos(k * R) - 1j * t * np.sin(k * R)) / R
    assert np.abs(got[0] + 1j * got[1] - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("k", WAVENUMBERS)
@pytest.mark.parametrize("mode", ["EH", "FF", "scalar"])
def test_modes_and_gradients_against_oracle(cuda, lib, oracle_mod, mode, k):
    from pypo_gb300 import engine
    rng = np.random.default_rng(5)
    s7, t7 = _one_source()
    if mode == "FF":   # along the axis: r . s = 2
        s7[2], t7[0:2] = 2.0, 0.0
    cur = rng.standard_normal((2 if mode == "scalar" else 12, 1))
    ref = oracle_mod.run(mode, s7, cur, -1, 0, 0, t7, k, 1.0, -1.0)
    assert rel_l2(engine.propagate(mode, s7, cur, -1, 0, 0, t7, k, precision="fp64"), ref) <= FP64_TOL
    cot = rng.standard_normal(ref.shape)
    want = oracle_mod.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, 1.0, -1.0)
    for name, v in engine.adjoint(mode, s7, cur, -1, 0, 0, t7, k, cot, precision="fp64").items():
        assert rel_l2(v, want[name]) <= FP64_TOL, name
