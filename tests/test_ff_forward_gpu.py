"""The far-field forward without magnetic currents (po_ff0_kernel) against the
FP64 oracle at the counts where its lanes and tiles can go wrong: directions
around a CTA's 256 and an idle second lane, sources around a tile (128) and an
odd one, both time directions, narrow and wide tiles, and sources that face
away from part of the directions. The bar is the mixed path's. With the
magnetic currents present but zero, the kernel with M gives the same field."""
import numpy as np
import pytest

from tests.common import PHASE_TOL, REL_L2_TOL, errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nt", [(1, 1), (2, 127), (127, 128), (128, 129), (129, 255), (257, 256), (1500, 257),
                                   (40, 700)])
@pytest.mark.parametrize("t,spread,behind", [(-1.0, 1.0, False), (1.0, 1.0, True), (-1.0, 300.0, True)])
def test_against_oracle(cuda, lib, oracle_mod, ns, nt, t, spread, behind):
    import torch
    from pypo_gb300 import engine
    rng = np.random.default_rng(10 * ns + nt)
    s7 = np.zeros((7, ns))
    s7[0:2] = rng.uniform(-spread, spread, (2, ns))
    s7[2] = 0.1 * (s7[0] ** 2 + s7[1] ** 2) / spread
    n = np.stack([-0.4 * s7[0] / spread, -0.4 * s7[1] / spread, np.ones(ns)])
    s7[3:6] = n / np.linalg.norm(n, axis=0)
    s7[6] = 1.0 / ns
    t7 = np.zeros((7, nt))
    t7[0], t7[1] = rng.uniform(0, 0.1, nt), rng.uniform(-3, 3, nt)
    if behind:
        t7[0, ::5] += np.pi / 2 + 0.3
    cur = rng.standard_normal((12, ns))
    cur[6:] = 0.0
    k = 2 * np.pi
    ref = oracle_mod.run("FF", s7, cur, -1, 0, 0, t7, k, 1.0, t)
    dev = [torch.tensor(v, device=cuda) for v in (s7, cur, t7)]
    run = lambda m_zero: engine.propagate_dev("FF", dev[0], dev[1], -1, 0, 0, dev[2], k, 1.0, t,
                                              m_zero=m_zero).cpu().numpy()
    got = run(True)
    e, p = errors(got, ref, "FF")
    assert e <= REL_L2_TOL and p <= PHASE_TOL, (e, p)
    np.testing.assert_allclose(run(False), got, rtol=0, atol=1e-13 * np.abs(ref).max())
