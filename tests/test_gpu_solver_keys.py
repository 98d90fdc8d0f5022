"""The placement solver where the keys of its ranks change: one, two and three of them a lane, and the largest load of a rank on both sides
of 2^24, from which on a key is the amount alone. Against the CPU oracle, whole numbers: bit-exact."""

import numpy as np
import pytest

import cases as Cs
import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("largest", [(1 << 24) - 1, 1 << 24, (1 << 24) + 1])
@pytest.mark.parametrize("N,M,R", [(2, 2, 1), (32, 3, 2), (33, 3, 1), (64, 2, 3), (65, 4, 2), (72, 7, 1)])
def test_largest_load(native_lib, cuda_device, N, M, R, largest):
    rng = np.random.default_rng(N + largest % 7)
    total = rng.integers(0, 20000, size=N * M)
    total[M:2 * M] = 5000  # equal masters, equal ranks
    total[:M] = largest // (M + 1)
    total[0] += largest - total[:M].sum()
    split = np.stack([total // N + (np.arange(N * M) % N == r) * (total % N) for r in range(N)]).astype(np.int32)
    assert split.sum(0)[:M].sum() == largest
    for i, kw in enumerate((dict(eps=0.01), dict(eps=0.0, min_tokens=1, allow_zero=True))):
        case = Cs.SolveCase(f"{largest} {i}", split, M, R, N, ranks=(0, N - 1), **kw)
        for rank in case.ranks:
            out = G.cuda_solve(case, rank)
            assert out["status"].tolist() == [0, 0]
            plan = O.solve_placement(case.loads_per_rank, M, R, N, rank, G.oracle_params(case))
            for f in G.PLAN_FIELDS:
                assert np.array_equal(out[f].cpu().numpy(), getattr(plan, f)), (i, rank, f)
