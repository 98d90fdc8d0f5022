"""The load matrix of the stateless solver: rows read 16 bytes at a time, or single words where the matrix or the number of experts does not
allow it; one domain and two, more rows than a round of loads, this rank's row first and last. Against the CPU oracle: bit-exact."""

import numpy as np
import pytest
import torch

import cases as Cs
import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("N,nvl,M,R", [(2, 2, 2, 1), (64, 64, 4, 2), (72, 72, 7, 2), (16, 16, 1, 1), (8, 8, 33, 2), (72, 36, 4, 2), (6, 3, 3, 1)])
def test_loads(native_lib, cuda_device, N, nvl, M, R, off):
    rng = np.random.default_rng(N * M + off)
    lpr = (rng.random((N, N * M)) ** 6 * 4000).astype(np.int32)
    case = Cs.SolveCase("loads", lpr, M, R, nvl, ranks=(0, N - 1))
    flat = torch.zeros(lpr.size + off, dtype=torch.int32, device=cuda_device)
    flat[off:] = torch.from_numpy(lpr).to(cuda_device).view(-1)
    for rank in case.ranks:
        out = G.cuda_solve(case, rank, flat[off:])
        assert np.array_equal(out["global_loads"].cpu().numpy(), lpr.sum(0))
        plan = O.solve_placement(lpr, M, R, nvl, rank, G.oracle_params(case))
        for f in G.PLAN_FIELDS:
            assert np.array_equal(out[f].cpu().numpy(), getattr(plan, f)), (rank, f)
