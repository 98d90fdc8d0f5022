"""Dense reroute forward of inputs so long that a CTA counts four tiles: ends of the input inside the first, second and last of the four,
widths that add packed words and widths that do not, ranks hosted together of which some end long before others. Against the CPU
oracle; copies, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_dense_tiles import _random_plan
from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,L,P", [(256 * 230, 128, 160), (256 * 230 + 5, 16, 48), (256 * 231 + 70, 96, 130), (256 * 230 + 200, 37, 50), (256 * 229 + 255, 64, 81)])
def test_counts_of_four_tiles(native_lib, cuda_device, T, L, P):
    rng = np.random.default_rng(T)
    plan = _random_plan(L, P, 8, 8, rng)
    rmap = rng.random((T, L), dtype=np.float32) < np.linspace(0.01, 0.2, L, dtype=np.float32)
    rmap[:, 0] = True
    probs = rng.random((T, L), dtype=np.float32)
    want_probs, want_map = O.dense_reroute_forward(rmap, probs, plan, P, True, quota=True)
    pd = G.plan_to_device(plan, cuda_device)
    got_probs, got_map = G.cuda_dense_reroute(torch.from_numpy(rmap).to(cuda_device), torch.from_numpy(probs).to(cuda_device), pd["l2p"], pd["lcnts"],
                                              pd["rank_quota_prefix"], P, True, True)
    assert np.array_equal(got_map.cpu().numpy(), want_map)
    assert np.array_equal(got_probs.cpu().numpy().view(np.uint32), want_probs.view(np.uint32))


# 95 tiles a rank at most: more CTAs of one tile than the device holds
@pytest.mark.parametrize("M", [8, 12, 16])
@pytest.mark.parametrize("longest", [0, 7])
def test_hosted_ranks_of_different_lengths(native_lib, cuda_device, M, longest):
    N, R, L = 8, 2, 8 * M
    lengths = [64 * 3 + 5, 1, 64, 64 * 4, 64 * 4 + 1, 64 * 90 + 63, 0, 64 * 6]
    lengths[longest] = 64 * 94 + 9
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=True, sim=True))
    rng = np.random.default_rng(M)
    popular = rng.random(L) ** 3
    for _ in range(2):
        maps = [rng.random((t, L)) < popular for t in lengths]
        probs = [rng.random(m.shape, dtype=np.float32) for m in maps]
        d_maps, d_probs = ([torch.from_numpy(x).to(cuda_device) for x in xs] for xs in (maps, probs))
        group.update_placement(0, d_maps)
        got_probs, got_maps = group.reroute_dense(0, d_maps, d_probs)
        torch.cuda.synchronize()
        group.check_status()
        loads = np.stack([m.sum(0) for m in maps]).astype(np.int32)
        for r in range(N):
            plan = O.solve_placement(loads, M, R, N, r)
            if len(maps[r]):
                want_probs, want_map = O.dense_reroute_forward(maps[r], probs[r], plan, group.P, True, quota=True)
                assert np.array_equal(got_maps[r].cpu().numpy(), want_map), r
                assert np.array_equal(got_probs[r].cpu().numpy().view(np.uint32), want_probs.view(np.uint32)), r
            else:
                assert got_maps[r].numel() == 0
    group.destroy()
