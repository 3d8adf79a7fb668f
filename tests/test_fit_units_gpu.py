"""The Gaussian fit's compaction and overlap sums (po_fitgauss_dev.cu) where
their splits can go wrong: regions around a warp's 32 points, a block's share
and eight units, on ragged grids. The misfit the device reaches is compared
with numpy's at the same parameters, and a fit of an exact Gaussian has to
return its own shape. LIN; sums in another order than numpy's, so the misfits
agree to 1e-12 and the shape within the simplex's xatol of 1e-4."""
import numpy as np
import pytest

from oracle import fitgauss as OF

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore::RuntimeWarning")]


@pytest.mark.parametrize("n,width", [(13, 0.12), (31, 0.05), (61, 0.02), (61, 0.2), (129, 0.1), (300, 0.02), (401, 0.3)])
def test_fit_of_an_exact_gaussian(cuda, lib, n, width):
    import torch
    from pypo_gb300 import fitgauss as FG
    from pypo_gb300._lib import POError
    ax = np.linspace(-0.5, 0.5, n)
    x, y = (v.ravel() for v in np.meshgrid(ax, ax, indexing="ij"))
    amp = np.exp(-((x - 0.01) ** 2 / (2 * width**2) + (y + 0.02) ** 2 / (2 * (1.3 * width) ** 2)))
    g7 = torch.zeros((7, n * n), dtype=torch.float64)
    g7[0], g7[1] = torch.from_numpy(x), torch.from_numpy(y)
    fit = lambda: FG.fit_gauss_abs_dev(g7.cuda(), n, n, torch.from_numpy(amp).cuda(), None, -11.0, "LIN", None)
    try:
        start = OF.start_point(amp.reshape(n, n), x.reshape(n, n), y.reshape(n, n), -11.0, 0)
    except IndexError:   # a beam wider than the grid: the reference's window leaves it, an error on both sides
        with pytest.raises(POError, match="past the grid"):
            fit()
        return
    popt = fit()
    pat, sel = OF.fit_region(amp.reshape(n, n), x.reshape(n, n), y.reshape(n, n), -11.0, 0)
    if not np.all(np.isfinite(start)):   # a region on one line of points: singular moments, no start point
        assert not np.all(np.isfinite(popt))
        return
    args = (x.reshape(n, n), y.reshape(n, n), pat, sel, 0)
    assert OF.misfit(popt, *args) <= OF.misfit(start, *args) + 1e-12
    # sorted: the fit may swap the axes with a quarter turn of theta
    if sel.sum() > 40:
        np.testing.assert_allclose(sorted(np.abs(popt[:2])), sorted((width, 1.3 * width)), atol=2e-3)
        np.testing.assert_allclose(popt[2:4], (0.01, -0.02), atol=2e-3)


def test_fits_on_two_threads_do_not_share_results(cuda, lib):
    """Fits running at the same time on threads and streams of their own give
    the values of the same fits one after the other."""
    import threading
    import torch
    from pypo_gb300 import fitgauss as FG
    n = 101
    ax = np.linspace(-0.5, 0.5, n)
    x, y = (v.ravel() for v in np.meshgrid(ax, ax, indexing="ij"))
    g7 = torch.zeros((7, n * n), dtype=torch.float64)
    g7[0], g7[1] = torch.from_numpy(x), torch.from_numpy(y)
    g7 = g7.cuda()
    amps = [torch.from_numpy(np.exp(-(x**2 + (1.0 + 0.1 * k) * y**2) / (2 * 0.1**2))).cuda() for k in range(4)]
    one = [FG.fit_gauss_abs_dev(g7, n, n, a, None, -11.0, "LIN", None) for a in amps]
    got = [None] * len(amps)

    def work(k):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for _ in range(3):
                got[k] = FG.fit_gauss_abs_dev(g7, n, n, amps[k], None, -11.0, "LIN", None)

    torch.cuda.synchronize()
    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(amps))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, b in zip(one, got):
        np.testing.assert_array_equal(a, b)
