"""Dense reroute forward at the numbers of tiles between which a CTA of the scatter kernel has 128 threads (four and eight tiles an SM), and
with more experts than that. Against the CPU oracle; copies, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_dense_tiles import _random_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_per_sm,extra", [(4, 0), (4, 1), (8, 0), (8, 1), (5, -17)])
@pytest.mark.parametrize("L,P,D", [(16, 48, 8), (130, 147, 4), (300, 330, 10)])
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
