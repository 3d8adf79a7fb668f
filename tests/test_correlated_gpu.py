"""The correlated error's integer cosines (po_grid_dev.cu) against the oracle's
FP64 sums, at the counts where stages and shares can go wrong (256 modes a
stage, 32 points a CTA, the modes in 8 shares), near and far from the origin,
and at phases beyond the integers' range (2^28 turns), which take cos(). The
tolerance is the FP64 sums' own: three roundings of the argument, one of the
cosine and one of the addition per mode."""
import numpy as np
import pytest

from oracle import grids as OG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 1000])
@pytest.mark.parametrize("n_modes", [1, 33, 255, 257, 700])
@pytest.mark.parametrize("span,corr_len", [(0.0, 30.0), (1e-3, 30.0), (300.0, 30.0), (1e6, 5.0), (1e3, 1e-7)])
def test_against_oracle(cuda, lib, n, n_modes, span, corr_len):
    import torch
    from pypo_gb300 import engine
    rng = np.random.default_rng(n + n_modes)
    g7 = np.zeros((7, n))
    g7[0:2] = rng.uniform(-span, span, (2, n))
    g7[5] = 1.0
    want = OG.correlated_error(g7[0], g7[1], 0.05, corr_len, seed=3, n_modes=n_modes)
    got = engine.correlated_error_dev(torch.tensor(g7, device=cuda), 0.05, corr_len, seed=3,
                                      n_modes=n_modes).cpu().numpy()
    theta = 6.0 * (np.abs(g7[0]) + np.abs(g7[1])) / corr_len + np.pi   # |k| < 6 / corr_len
    eps = 2.0 ** -53
    tol = 0.05 * np.sqrt(2.0 / n_modes) * n_modes * (3.0 * theta + 1.0 + n_modes) * 2 * eps
    assert np.all(np.abs(got - want) <= tol), float(np.max(np.abs(got - want) / tol))
