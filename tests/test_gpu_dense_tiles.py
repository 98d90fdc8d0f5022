"""Dense reroute, forward and backward, at the edges of its tiles: row counts around a tile and a segment, widths that
allow one, two and four columns per store, unaligned maps, experts with more instances than the staged rows hold, outputs
wider than one column chunk, the paths that add up earlier tiles. Against the CPU oracle; copies, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu


def _random_plan(L, P, D, max_copies, rng):
    """Any replica counts, distinct physical slots, increasing prefixes (some of them equal)."""
    counts = np.minimum(rng.integers(1, max_copies + 1, size=L), D)
    counts[rng.random(L) < 0.6] = 1
    while counts.sum() > P:
        counts[np.argmax(counts)] -= 1
    slots = rng.permutation(P)[:counts.sum()]
    l2p = np.full((L, D), -1, np.int32)
    prefix = np.zeros((L, D), np.int32)
    at = 0
    for e, c in enumerate(counts):
        l2p[e, :c] = slots[at:at + c]
        prefix[e, :c] = np.cumsum(rng.integers(0, 40, size=c))
        at += c
    z = np.zeros((L, D), np.int32)
    return O.Plan(np.zeros(P, np.int32), l2p, counts.astype(np.int32), z, z, prefix)


SHAPES = [  # T, L, P, D, most instances, rows of the buffer in front of the map
    (1, 8, 12, 4, 3, 0), (7, 64, 66, 2, 2, 0), (64, 64, 80, 8, 8, 0), (65, 128, 160, 8, 8, 0), (1030, 128, 161, 8, 5, 0),
    (130, 96, 98, 3, 3, 0), (4200, 96, 130, 8, 8, 0), (513, 37, 50, 6, 6, 0), (200, 30, 64, 16, 12, 0), (33, 66, 101, 70, 40, 1),
    (9000, 16, 48, 8, 8, 0), (70, 1340, 9001, 8, 8, 0), (70, 1340, 8200, 8, 8, 0), (129, 36, 60, 8, 8, 1), (2100, 256, 320, 8, 8, 0),
]


@pytest.mark.parametrize("T,L,P,D,copies,front", SHAPES)
@pytest.mark.parametrize("quota,interleave", [(True, True), (True, False), (False, False)])
def test_dense_tile_edges(native_lib, cuda_device, T, L, P, D, copies, front, quota, interleave):
    rng = np.random.default_rng(T * 7 + L)
    plan = _random_plan(L, P, D, copies, rng)
    rmap = rng.random((T + front, L)) < np.linspace(0.02, 0.3, L)
    rmap[:, 0] = True  # an expert in every row
    probs = rng.random((T + front, L)).astype(np.float32)
    d_map, d_probs = torch.from_numpy(rmap).to(cuda_device)[front:], torch.from_numpy(probs).to(cuda_device)[front:]
    rmap, probs = rmap[front:], probs[front:]
    exp_probs, exp_map = O.dense_reroute_forward(rmap, probs, plan, P, interleave, quota=quota)
    pd = G.plan_to_device(plan, cuda_device)
    got_probs, got_map = G.cuda_dense_reroute(d_map, d_probs, pd["l2p"], pd["lcnts"], pd["rank_quota_prefix"], P, interleave, quota)
    assert np.array_equal(got_map.cpu().numpy(), exp_map)
    assert np.array_equal(got_probs.cpu().numpy().view(np.uint32), exp_probs.view(np.uint32))

    grad = rng.normal(size=(T, P)).astype(np.float32)
    exp_map[rng.random(T) < 0.1] = False  # cells that no instance took: zero gradient
    exp = O.dense_reroute_backward(grad, rmap, exp_map, plan)
    if quota and interleave and T * L < 1 << 22:  # the tile kernel starts at that many cells: the same rows again and again
        n = -(-(1 << 22) // (T * L))
        rep = lambda t: torch.cat([t] * n)
        got = G.cuda_dense_reroute_backward(rep(torch.from_numpy(grad).to(cuda_device)), rep(d_map),
                                            rep(torch.from_numpy(exp_map).to(cuda_device)), pd["l2p"], pd["lcnts"])
        assert np.array_equal(got.cpu().numpy().reshape(n, T, L).view(np.uint32), np.broadcast_to(exp.view(np.uint32), (n, T, L)))
    got = G.cuda_dense_reroute_backward(torch.from_numpy(grad).to(cuda_device), d_map, torch.from_numpy(exp_map).to(cuda_device),
                                        pd["l2p"], pd["lcnts"])
    assert np.array_equal(got.cpu().numpy().view(np.uint32), exp.view(np.uint32))
