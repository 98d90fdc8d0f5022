"""Dense reroute forward with tables that send several experts of one instance to one physical column, of which a tile of 64 tokens routes
to one at most: the others' empty columns leave it alone. Against the CPU oracle; copies, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu

TILE = 64


@pytest.mark.parametrize("L", [24, 300, 700])
@pytest.mark.parametrize("several", [False, True])
def test_one_column_of_two_experts(native_lib, cuda_device, L, several):
    rng = np.random.default_rng(L)
    T, half, D = 5 * TILE + 17, L // 2, 3
    P = half + 2
    l2p = np.full((L, D), -1, np.int32)
    l2p[:, 0] = np.arange(L) % half  # experts e and e + half
    counts = np.ones(L, np.int32)
    prefix = np.zeros((L, D), np.int32)
    if several:  # expert 0 has an instance in that column and two that are its own
        counts[0] = 3
        l2p[0, 1:] = half, half + 1
        prefix[0] = 10, 25, 60
    z = np.zeros((L, D), np.int32)
    plan = O.Plan(np.zeros(P, np.int32), l2p, counts, z, z, prefix)
    rmap = rng.random((T, L)) < 0.3
    for t0 in range(0, T, TILE):  # a tile routes to one expert of each pair, now the lower, now the upper one
        lower = rng.random(half) < 0.5
        rmap[t0:t0 + TILE, :half] &= lower
        rmap[t0:t0 + TILE, half:2 * half] &= ~lower
    probs = rng.random((T, L), dtype=np.float32)
    want_probs, want_map = O.dense_reroute_forward(rmap, probs, plan, P, True, quota=True)
    pd = G.plan_to_device(plan, cuda_device)
    for _ in range(3):
        got_probs, got_map = G.cuda_dense_reroute(torch.from_numpy(rmap).to(cuda_device), torch.from_numpy(probs).to(cuda_device), pd["l2p"], pd["lcnts"],
                                                  pd["rank_quota_prefix"], P, True, True)
        assert np.array_equal(got_map.cpu().numpy(), want_map)
        assert np.array_equal(got_probs.cpu().numpy().view(np.uint32), want_probs.view(np.uint32))
