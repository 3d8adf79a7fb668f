"""The Gaussian fit on regions around and past one pass of the overlap sums'
grid (po_fitgauss_dev.cu: 1,216 units of 32 points, 38,912 points), where a
block takes a second unit and the rows of unit sums are full. The pattern is
wider on the side of the region's later points, so that sums without them have
another optimum: at 601 points a side its misfit is 2.6e-3 higher, at 701
7.6e-3. Both simplexes stop at 1e-4."""
import numpy as np
import pytest
from scipy.optimize import fmin

from oracle import fitgauss as OF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,points", [(497, 38816), (498, 38932), (601, 56777), (701, 77396)])
def test_misfit_of_a_large_region(cuda, lib, n, points):
    import torch
    from pypo_gb300 import fitgauss as FG
    ax = np.linspace(-0.5, 0.5, n)
    x, y = np.meshgrid(ax, ax, indexing="ij")
    w = np.where(x > 0.01, 0.15, 0.12)
    amp = np.exp(-((x - 0.01) ** 2 / (2 * w**2) + (y + 0.02) ** 2 / (2 * 0.156**2)))
    pat, sel = OF.fit_region(amp, x, y, -11.0, 0)
    assert sel.sum() == points
    start = OF.start_point(amp, x, y, -11.0, 0)
    best = fmin(lambda p: OF.misfit(p, x, y, pat, sel, 0), start, disp=False)
    g7 = torch.zeros((7, n * n), dtype=torch.float64)
    g7[0], g7[1] = torch.from_numpy(x.ravel()), torch.from_numpy(y.ravel())
    popt, p0 = FG.fit_gauss_abs_dev(g7.cuda(), n, n, torch.from_numpy(amp.ravel()).cuda(), None, -11.0, "LIN", None,
                                    full_output=True)
    np.testing.assert_allclose(p0, start, rtol=1e-9, atol=1e-9)
    assert OF.misfit(popt, x, y, pat, sel, 0) <= OF.misfit(best, x, y, pat, sel, 0) + 2e-4


def test_a_beam_wider_than_the_grid_is_an_error(cuda, lib):
    """The reference's window indexes past the grid there (IndexError)."""
    import torch
    from pypo_gb300 import fitgauss as FG
    from pypo_gb300._lib import POError
    n = 401
    ax = np.linspace(-0.5, 0.5, n)
    x, y = np.meshgrid(ax, ax, indexing="ij")
    amp = np.exp(-((x - 0.01) ** 2 / (2 * 0.3**2) + (y + 0.02) ** 2 / (2 * 0.39**2)))
    with pytest.raises(IndexError):
        OF.fit_region(amp, x, y, -11.0, 0)
    g7 = torch.zeros((7, n * n), dtype=torch.float64)
    g7[0], g7[1] = torch.from_numpy(x.ravel()), torch.from_numpy(y.ravel())
    with pytest.raises(POError, match="past the grid"):
        FG.fit_gauss_abs_dev(g7.cuda(), n, n, torch.from_numpy(amp.ravel()).cuda(), None, -11.0, "LIN", None)
