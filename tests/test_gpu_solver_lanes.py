"""The placement solver where a warp fills its lists of ranks and adds loads up in one, two and three rounds (2 to 72 ranks), with many
masters per rank, many equal loads, quotients beyond 2^20, several floors; and the plan's histogram at widths that do not
divide its threads. Against the CPU oracle, whole numbers: bit-exact."""

import numpy as np
import pytest
import torch

import cases as Cs
import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,R", [(2, 200, 3), (12, 40, 4), (31, 5, 2), (32, 8, 4), (33, 4, 1), (64, 8, 8), (65, 3, 2), (72, 7, 7)])
@pytest.mark.parametrize("kind", ["ties", "zipf", "huge"])
def test_solver_lane_edges(native_lib, cuda_device, N, M, R, kind):
    rng = np.random.default_rng(N * 1000 + M)
    L = N * M
    for i in range(4):
        if kind == "ties":
            loads = rng.integers(0, 3, size=(N, L)) * 16
            loads[:, rng.integers(0, L, size=3)] += 64 * int(rng.integers(1, 30))
        else:
            w = np.arange(1, L + 1) ** -float(rng.uniform(0.8, 2.0))
            loads = rng.multinomial(20000, w[rng.permutation(L)] / w.sum(), size=N)
            if kind == "huge":
                loads = loads * (25000000 // (20000 * N))  # the whole group's tokens stay within 31 bits
        case = Cs.SolveCase(f"{kind}{i}", loads.astype(np.int32), M, R, N, min_tokens=[1, 16, 1024, 1][i], allow_zero=i % 2 == 1,
                            locality=i != 2, eps=[0.01, 0.0, 0.2, 0.01][i], ranks=(0, N - 1))
        for rank in case.ranks:
            out = G.cuda_solve(case, rank)
            plan = O.solve_placement(case.loads_per_rank, M, R, N, rank, G.oracle_params(case))
            for f in G.PLAN_FIELDS:
                assert np.array_equal(out[f].cpu().numpy(), getattr(plan, f)), (kind, i, rank, f)


@pytest.mark.parametrize("T,L", [(1, 96), (2100, 96), (70000, 48), (333, 4096), (100, 4112), (257, 72)])
def test_histogram_map_widths(native_lib, cuda_device, T, L):
    rmap = np.random.default_rng(L).random((T, L)) < 0.4
    got = G.cuda_histogram(torch.from_numpy(rmap).to(cuda_device), L, "map")
    assert np.array_equal(got.cpu().numpy(), rmap.sum(0))
