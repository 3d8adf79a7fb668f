"""More targets than 1 GiB of partial sums holds for one source chunk (11.18
million with 12 accumulators): one chunk of all the sources, as for any count."""
import numpy as np
import pytest

from tests.common import REL_L2_TOL, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,precision", [("EH", "mixed"), ("FF", "mixed"), ("EH", "fp64")])
def test_one_chunk_of_sources(cuda, lib, mode, precision):
    import torch
    from pypo_gb300 import engine
    ns, nt = 40, 11_200_001
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    rand = lambda *shape: 2.0 * torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda") - 1.0
    s7 = torch.zeros((7, ns), dtype=torch.float64, device=cuda)
    s7[0:2], s7[5], s7[6] = rand(2, ns), 1.0, 1.0
    cur = rand(12, ns)
    t7 = torch.zeros((7, nt), dtype=torch.float64, device=cuda)
    t7[0:2] = rand(2, nt)
    if mode == "FF":
        t7[0] = 0.3 * t7[0].abs()
    else:
        t7[2], t7[5] = 3.0, -1.0
    out = engine.propagate_dev(mode, s7, cur, -1, 0, 0, t7, 20.0, precision=precision)
    at = torch.cat([torch.arange(300), torch.arange(nt // 2, nt // 2 + 300), torch.arange(nt - 300, nt)]).cuda()
    want = engine.propagate_dev(mode, s7, cur, -1, 0, 0, t7[:, at].contiguous(), 20.0, precision="fp64")
    assert rel_l2(out[:, at].cpu().numpy(), want.cpu().numpy()) <= REL_L2_TOL
