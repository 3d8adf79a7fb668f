"""The mixed near-field and scalar adjoint where a block has threads without a
source (a count that is no multiple of 128): they add nothing to grad_dt,
wherever the targets are. Sources on a plane at z = 0 and targets at z = 2000
wavelengths, both centred: a target on the axis is exactly 1000 wavelengths
from the frame's origin. Against the plain FP64 adjoint at the mixed path's bar."""
import numpy as np
import pytest

from tests.common import REL_L2_TOL, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,m_zero", [("EH", True), ("JM", False), ("scalar", True)])
@pytest.mark.parametrize("z", [2000.0, -2000.0, 300.0])
def test_target_on_the_axis(cuda, lib, mode, m_zero, z):
    from pypo_gb300 import engine
    rng = np.random.default_rng(4)
    ax = np.linspace(-20.0, 20.0, 11)
    x, y = (v.ravel() for v in np.meshgrid(ax, ax, indexing="ij"))
    s7, t7 = np.zeros((7, 121)), np.zeros((7, 121))
    s7[0], s7[1], s7[5], s7[6] = x, y, np.sign(z), 16.0
    t7[0], t7[1], t7[2], t7[5], t7[6] = x, y, z, -np.sign(z), 16.0
    cur = rng.standard_normal((2 if mode == "scalar" else 12, 121))
    if m_zero and mode != "scalar":
        cur[6:] = 0.0
    k = 2.0 * np.pi
    cot = rng.standard_normal((engine.n_out(mode), 121))
    want = engine.adjoint(mode, s7, cur, 0, 11, 11, t7, k, cot, precision="fp64")
    for subset in (("cur", "ds", "dt"), ("dt",), ("ds", "dt"), ("cur", "dt")):
        got = engine.adjoint(mode, s7, cur, 0, 11, 11, t7, k, cot, want=subset)
        for name in subset:
            assert np.isfinite(got[name]).all(), (subset, name)
            assert rel_l2(got[name], want[name]) <= REL_L2_TOL, (subset, name)
