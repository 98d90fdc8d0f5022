"""Sparse reroute and dispatch positions at the edges of their work split (one entry per thread of one CTA, full clusters,
one cluster against several, the count-table form and its wide tiles), in place and not, against the CPU oracle.
Whole numbers: bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu


def _plan(N, M, R, nvl, seed):
    rng = np.random.default_rng(seed)
    L = N * M
    w = np.arange(1, L + 1, dtype=np.float64) ** -1.3
    p = w[rng.permutation(L)] / w.sum()
    lpr = np.stack([rng.multinomial(40000, p) for _ in range(N)]).astype(np.int32)
    return O.solve_placement(lpr, M, R, nvl, 1 % N, O.SolverParams(min_tokens_per_replica=1)), p


@pytest.mark.parametrize("n", [1, 31, 512, 513, 4096, 4097, 16384, 16385, 32769, 65537, 262144, 262145, 300007, 1048577])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_sparse_reroute_split_edges(native_lib, cuda_device, n, dtype):
    plan, p = _plan(8, 9, 3, 8, 5)  # 72 experts: not a power of two
    rng = np.random.default_rng(n)
    ids = rng.choice(len(p), size=(n, 1), p=p).astype(dtype)
    if n > 40:
        ids[n // 2], ids[n - 1] = -1, len(p)  # outside [0, L): kept, and no ordinal taken
    exp = O.sparse_reroute(ids, plan, True)
    pd = G.plan_to_device(plan, cuda_device)
    dev = torch.from_numpy(ids).to(cuda_device)
    got = G.cuda_sparse_reroute(dev, pd["l2p"], pd["lcnts"], pd["rank_quota_prefix"])
    assert np.array_equal(got.cpu().numpy(), exp)
    G.cuda_sparse_reroute(dev, pd["l2p"], pd["lcnts"], pd["rank_quota_prefix"], inplace=True)
    assert np.array_equal(dev.cpu().numpy(), exp)
    if n > 1:  # a base address that is not 16-byte aligned
        odd = torch.from_numpy(ids).to(cuda_device)[1:]
        got = G.cuda_sparse_reroute(odd, pd["l2p"], pd["lcnts"], pd["rank_quota_prefix"])
        assert np.array_equal(got.cpu().numpy(), O.sparse_reroute(ids[1:], plan, True))


def test_sparse_reroute_many_experts(native_lib, cuda_device):
    """1720 experts: the plan rows are not staged in shared memory."""
    plan, p = _plan(40, 43, 2, 8, 6)
    ids = np.random.default_rng(1).choice(len(p), size=(9000, 4), p=p).astype(np.int32)
    pd = G.plan_to_device(plan, cuda_device)
    got = G.cuda_sparse_reroute(torch.from_numpy(ids).to(cuda_device), pd["l2p"], pd["lcnts"], pd["rank_quota_prefix"])
    assert np.array_equal(got.cpu().numpy(), O.sparse_reroute(ids, plan, True))


def test_interleave_of_large_products(native_lib, cuda_device):
    """ordinal * stride beyond 32 bits, and totals of 2, 3 and powers of two (the reciprocal's rounding)."""
    plan, _ = _plan(8, 1, 2, 8, 7)
    for total in (2, 3, 4, 1 << 16, 150001, 1 << 20):
        plan.lcnts[:] = 2
        plan.l2p[:, 1] = (plan.l2p[:, 0] + 3) % 24
        plan.rank_quota_prefix[:, 0] = total // 3
        plan.rank_quota_prefix[:, 1] = total
        ids = np.random.default_rng(total).choice(2, size=(250000, 1)).astype(np.int32)
        pd = G.plan_to_device(plan, cuda_device)
        got = G.cuda_sparse_reroute(torch.from_numpy(ids).to(cuda_device), pd["l2p"], pd["lcnts"], pd["rank_quota_prefix"])
        assert np.array_equal(got.cpu().numpy(), O.sparse_reroute(ids, plan, True)), total


@pytest.mark.parametrize("n,P", [(512, 31), (513, 32), (16385, 80), (65537, 160), (262145, 80), (40000, 4500), (4097, 7255), (2048, 256), (2049, 255), (4096, 1023),
                                 (8193, 1024)])
@pytest.mark.parametrize("in_place", [False, True])
def test_dispatch_positions_split_edges(native_lib, cuda_device, n, P, in_place):
    rng = np.random.default_rng(n)
    phys = np.minimum(rng.zipf(1.3, size=n) - 1, P + 3).astype(np.int32)  # hot experts first, some keys outside [0, P)
    phys[n // 3] = -7
    exp_pos, exp_off = O.dispatch_positions(phys, P)
    pos, off = G.cuda_dispatch_positions(torch.from_numpy(phys).to(cuda_device), P, in_place)
    assert np.array_equal(pos.cpu().numpy(), exp_pos)
    assert np.array_equal(off.cpu().numpy(), exp_off)
