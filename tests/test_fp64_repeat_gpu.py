"""The plain FP64 adjoint gives the same bits each time, grad_dt too, and its
target sums, kept per block of sources and added in order, are right where
they are taken in rounds (more than 1 GiB of them)."""
import numpy as np
import pytest

from tests.common import FP64_TOL

pytestmark = pytest.mark.gpu


def _case(ns, nt, rows, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rand = lambda *shape: torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda")
    s7, t7 = torch.zeros((7, ns), dtype=torch.float64, device="cuda"), torch.zeros((7, nt), dtype=torch.float64, device="cuda")
    s7[0:2], s7[5], s7[6] = 2.0 * rand(2, ns) - 1.0, 1.0, 1.0 / ns
    t7[0:2], t7[2], t7[5] = 2.0 * rand(2, nt) - 1.0, 3.0 + rand(nt), -1.0
    return s7, t7, rand(rows, ns) - 0.5, rand(rows, nt) - 0.5


@pytest.mark.parametrize("mode,rows", [("EH", 12), ("scalar", 2)])
@pytest.mark.parametrize("ns,nt", [(5003, 1501), (20000, 33), (129, 4001)])
def test_same_bits_each_time(cuda, lib, mode, rows, ns, nt):
    import torch
    from pypo_gb300 import engine
    s7, t7, cur, cot = _case(ns, nt, rows, ns)
    runs = []
    for _ in range(4):
        out = (torch.empty_like(cur), torch.empty(ns, dtype=torch.float64, device=cuda),
               torch.empty(nt, dtype=torch.float64, device=cuda))
        engine.adjoint_dev(mode, s7, cur, -1, 0, 0, t7, 30.0, cot, precision="fp64", grad_cur=out[0], grad_ds=out[1],
                           grad_dt=out[2])
        runs.append(out)
    torch.cuda.synchronize()
    for out in runs[1:]:
        for a, b in zip(out, runs[0]):
            assert torch.equal(a, b)


def test_target_sums_in_rounds(cuda, lib):
    """1,101 blocks of sources and 122,000 targets: 1,100 rows of target sums
    fit, one block is left for a second round. The sum over the sources is the
    sum over two parts of them, each of one round."""
    import torch
    from pypo_gb300 import engine
    ns, nt, cut = 1100 * 128 + 1, 122000, 70000
    s7, t7, cur, cot = _case(ns, nt, 2, 1)
    sums = []
    for a, b in ((0, ns), (0, cut), (cut, ns)):
        gt = torch.empty(nt, dtype=torch.float64, device=cuda)
        engine.adjoint_dev("scalar", s7[:, a:b].contiguous(), cur[:, a:b].contiguous(), -1, 0, 0, t7, 30.0, cot,
                           precision="fp64", grad_dt=gt)
        sums.append(gt)
    err = torch.linalg.norm(sums[0] - sums[1] - sums[2]) / torch.linalg.norm(sums[0])
    assert err.item() <= FP64_TOL
