"""The placement solver where its lists of ranks can go wrong: thresholds on both sides of 2^24, from which on a rank's key takes 64
bits; ranks that come back with equal slack; one redundant slot, so that nobody comes back; more experts with replicas than warps;
floors that fail. Against the CPU oracle, whole numbers: bit-exact."""

import numpy as np
import pytest
import torch

import cases as Cs
import gpu_util as G
from oracle import uep_oracle as O
from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu


def _check(loads, M, R, what, **kw):
    N = loads.shape[0]
    case = Cs.SolveCase(what, np.ascontiguousarray(loads, dtype=np.int32), M, R, N, ranks=(0, N - 1), **kw)
    for rank in case.ranks:
        out = G.cuda_solve(case, rank)
        assert out["status"].tolist() == [0, 0]
        plan = O.solve_placement(case.loads_per_rank, M, R, N, rank, G.oracle_params(case))
        for f in G.PLAN_FIELDS:
            assert np.array_equal(out[f].cpu().numpy(), getattr(plan, f)), (what, rank, f)


# Mean load of a rank. (The oracle adds slack up in 32 bits: ranks^2 times the mean stays below 2^31.)
@pytest.mark.parametrize("mean", [(1 << 24) - 40000, (1 << 24) - 1, 1 << 24, (1 << 24) + 3, 3 << 23])
@pytest.mark.parametrize("N,M,R", [(2, 3, 1), (4, 2, 2), (8, 5, 3)])
def test_keys_on_both_sides_of_32_bits(native_lib, cuda_device, mean, N, M, R):
    rng = np.random.default_rng(mean % 1000003 + N)
    for eps in (0.0, 0.01):
        w = rng.dirichlet(np.full(N * M, 0.3))
        total = np.floor(w * mean * N).astype(np.int64)
        total[0] += mean * N - total.sum()
        split = np.stack([total // N + (np.arange(N * M) % N == r) for r in range(N)])
        split[0] += total - split.sum(0)
        _check(np.maximum(split, 0), M, R, f"mean {mean}", eps=eps, min_tokens=1 if eps else 1024)


@pytest.mark.parametrize("N,M,R", [(8, 4, 2), (16, 2, 1), (33, 3, 2), (72, 4, 4)])
@pytest.mark.parametrize("min_tokens,bt", [(1, 1.0), (64, 1.0), (4096, 1.0), (256, 1.3)])
def test_equal_slack_and_floors(native_lib, cuda_device, N, M, R, min_tokens, bt):
    rng = np.random.default_rng(N + min_tokens)
    for i in range(3):
        loads = np.zeros((N, N * M), np.int64)
        hot = rng.choice(N, size=max(1, N // 3), replace=False)
        for r in hot:  # sources of several exports each, everyone else equal
            loads[:, r * M:r * M + M] = rng.integers(1, 5, size=M) * 64
        loads[:, rng.choice(N) * M] += 16 * i
        _check(loads, M, R, f"equal {i}", min_tokens=min_tokens, balance_threshold=bt, allow_zero=i == 1)


def _draw(i):
    rng = np.random.default_rng(i)
    nvl = int(rng.choice([2, 3, 4, 8, 16, 31, 48, 72]))
    N = 2 * nvl if nvl <= 8 and i % 3 == 0 else nvl
    M, R = int(rng.integers(1, min(7, 512 // nvl) + 1)), int(rng.integers(1, min(4, 512 // nvl) + 1))
    total = int(rng.integers(50, 30000))
    if i % 2:
        w = rng.permutation(np.arange(1, N * M + 1) ** -float(rng.uniform(0.5, 2.5)))
    else:  # some ranks hold nearly everything in even masters: more exports than slots, or (four slots) exports below the dynamic floor
        w = np.where(np.repeat(rng.random(N) < rng.uniform(0.3, 0.8), M), rng.uniform(0.5, 1.0, N * M), 0.01)
        R = 1 if i % 4 else min(4, 512 // nvl)
    loads = rng.multinomial(total, w / w.sum(), size=N).astype(np.int32)
    return Cs.SolveCase(f"sweep {i}", loads, M, R, nvl, balance_threshold=[1.0, 1.0, 1.02, 1.5][i % 4], min_tokens=[-3, 0, 1, 16, 200, 1024][i // 2 % 6],
                        allow_zero=i % 5 == 0, locality=i % 3 != 0, eps=[0.0, 0.01, 0.1][i % 3], ranks=(i % N,))


def test_every_way_through_the_search(native_lib, cuda_device):
    ways, rounds = set(), set()
    for i in range(300):
        case = _draw(i)
        rank = case.ranks[0]
        plan = O.solve_placement(case.loads_per_rank, case.M, case.R, case.nvl, rank, G.oracle_params(case))
        out = G.cuda_solve(case, rank)
        for f in G.PLAN_FIELDS:
            assert np.array_equal(out[f].cpu().numpy(), getattr(plan, f)), (i, f)
        assert out["status"].tolist() == [0, 0]
        ways |= {int(x) & 15 for x in plan.path}
        rounds |= {int(x) >> 12 & 255 for x in plan.path}
    assert ways == {1, 2, 3} and max(rounds) >= 5  # the builds side by side, the capacity threshold, the probes and how many rounds of them


# inputs for either kernel of the plan: 256 threads, and 512 with a rehearsal
@pytest.mark.parametrize("scale", [1, 60])
@pytest.mark.parametrize("M,R,legal", [(2, 1, {3}), (5, 1, {3}), (6, 4, {1, 2, 3})])
def test_probes_of_hosted_plans(native_lib, cuda_device, scale, M, R, legal):
    N = 8
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=False, sim=True))
    ways = set()
    for seed in range(6):
        rng = np.random.default_rng(seed)
        w = np.where(np.repeat(rng.permutation(N) < 4 + seed % 3, M), rng.uniform(0.5, 1.0, N * M), 0.01)
        loads = (rng.multinomial(12000, w / w.sum(), size=N) * scale).astype(np.int32)
        ids = [torch.from_numpy(rng.permutation(np.repeat(np.arange(N * M, dtype=np.int32), row))[:, None].copy()).to(cuda_device) for row in loads]
        group.update_placement(0, ids)
        torch.cuda.synchronize()
        group.check_status()
        for r in range(N):
            plan = O.solve_placement(loads, M, R, N, r)
            ways |= {int(x) & 15 for x in plan.path}
            got = group.plan(r, 0)
            for f in G.PLAN_FIELDS:
                assert np.array_equal(got[f].cpu().numpy().reshape(-1), getattr(plan, f).reshape(-1)), (seed, r, f)
    assert ways <= legal and ways & {2, 3}
    group.destroy()


def test_wide_keys_of_hosted_plans(native_lib, cuda_device):
    N, M, R = 2, 3, 2
    loads = np.array([[9000001, 5000000, 4000000, 100, 0, 7], [9000001, 6000000, 2000000, 90, 3, 0]], np.int32)  # thresholds above 2^24
    assert loads.sum() // N > 1 << 24
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=False, sim=True))
    experts = torch.arange(N * M, dtype=torch.int32, device=cuda_device)
    ids = [torch.repeat_interleave(experts, torch.from_numpy(row).to(cuda_device))[:, None].contiguous() for row in loads]
    group.update_placement(0, ids)
    torch.cuda.synchronize()
    group.check_status()
    for r in range(N):
        plan = O.solve_placement(loads, M, R, N, r)
        assert plan.lcnts.max() == 2
        got = group.plan(r, 0)
        for f in G.PLAN_FIELDS:
            assert np.array_equal(got[f].cpu().numpy().reshape(-1), getattr(plan, f).reshape(-1)), (r, f)
    group.destroy()
