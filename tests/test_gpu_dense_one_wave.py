"""Dense reroute forward at the numbers of tiles between which a CTA of the scatter kernel has 128 threads (four and eight tiles an SM, seven
for several ranks of more than 128 experts, never for one rank from 256 on). Against the CPU oracle; copies, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_dense_tiles import _random_plan
from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_per_sm,extra", [(4, 0), (4, 1), (8, 0), (8, 1), (5, -17)])
@pytest.mark.parametrize("L,P,D", [(16, 48, 8), (130, 147, 4), (255, 270, 4), (256, 270, 4), (300, 330, 10)])
def test_around_the_lines(native_lib, cuda_device, tiles_per_sm, extra, L, P, D):
    T = 64 * tiles_per_sm * torch.cuda.get_device_properties(cuda_device).multi_processor_count + extra
    rng = np.random.default_rng(T + L)
    plan = _random_plan(L, P, D, D, rng)
    rmap = rng.random((T, L), dtype=np.float32) < np.linspace(0.005, 0.1, L, dtype=np.float32)
    rmap[:, 0] = True
    probs = rng.random((T, L), dtype=np.float32)
    want_probs, want_map = O.dense_reroute_forward(rmap, probs, plan, P, True, quota=True)
    pd = G.plan_to_device(plan, cuda_device)
    got_probs, got_map = G.cuda_dense_reroute(torch.from_numpy(rmap).to(cuda_device), torch.from_numpy(probs).to(cuda_device), pd["l2p"], pd["lcnts"],
                                              pd["rank_quota_prefix"], P, True, True)
    assert np.array_equal(got_map.cpu().numpy(), want_map)
    assert np.array_equal(got_probs.cpu().numpy().view(np.uint32), want_probs.view(np.uint32))


@pytest.mark.parametrize("M", [64, 65])
@pytest.mark.parametrize("tiles_per_sm,extra", [(4, 0), (4, 1), (7, 0), (7, 1), (8, 0), (8, 1)])
def test_two_ranks_around_the_lines(native_lib, cuda_device, M, tiles_per_sm, extra):
    N, R, L = 2, 3, 2 * M
    T = 32 * tiles_per_sm * torch.cuda.get_device_properties(cuda_device).multi_processor_count + extra
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=True, sim=True))
    gen = torch.Generator(device=cuda_device).manual_seed(T + L)
    popular = torch.rand(L, generator=gen, device=cuda_device) ** 4 * 0.2
    maps = [torch.rand((T, L), generator=gen, device=cuda_device) < popular for _ in range(N)]
    probs = [torch.rand((T, L), generator=gen, device=cuda_device) for _ in range(N)]
    group.update_placement(0, maps)
    got_probs, got_maps = group.reroute_dense(0, maps, probs)
    torch.cuda.synchronize()
    group.check_status()
    for r in range(N):
        loads = np.stack([m.sum(0).cpu().numpy() for m in maps]).astype(np.int32)
        plan = O.solve_placement(loads, M, R, N, r)
        want_probs, want_map = O.dense_reroute_forward(maps[r].cpu().numpy(), probs[r].cpu().numpy(), plan, N * (M + R), True, quota=True)
        assert np.array_equal(got_maps[r].cpu().numpy(), want_map), r
        assert np.array_equal(got_probs[r].cpu().numpy().view(np.uint32), want_probs.view(np.uint32)), r
    group.destroy()
