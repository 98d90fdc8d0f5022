"""Dense reroute forward of inputs so long that a CTA counts four tiles: ends of the input inside the first, second and last of the four,
widths that add packed words and widths that do not. Against the CPU oracle; copies, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_dense_tiles import _random_plan

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
