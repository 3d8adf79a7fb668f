"""The device's normal deviates (po_grid_dev.cu) against the oracle's mt19937
and polar method, at the counts where the split into words, counting and
writing can go wrong: one block of words or a few, the CTAs' 256 attempts, and
more blocks than are kept at a time (a second round from the stored state)."""
import numpy as np
import pytest

from oracle import grids as OG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(2, 2), (2, 61), (11, 11), (3, 41), (20, 10), (41, 5), (23, 17), (1000, 520)])
@pytest.mark.parametrize("seed", [0, 4294967295])
def test_against_oracle(cuda, lib, size, seed):
    from pypo_gb300 import engine
    d = OG.plane(list(size), gmode=0, lims_a=[-1.0, 1.0], rms=0.7, rms_seed=seed)
    got = engine.generate_grid_dev(d, device=cuda).cpu().numpy()
    want = OG.generate(dict(d, rms=0.0))[2] + OG.normal_deviates(seed, size[0] * size[1], 0.7)
    np.testing.assert_allclose(got[2], want, rtol=0, atol=1e-14)   # a plane's normal is +z
