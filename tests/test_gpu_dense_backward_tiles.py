"""Dense reroute backward in tiles: heights of 64, 32, 16 and 8 rows with a ragged last one, experts with more instances than
the staged rows hold, cells that no instance or several instances took, widths that no vector divides. A copy of one
gradient each, so bit-exact."""

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,L,P,D,copies", [
    (8193, 128, 160, 8, 8), (20001, 128, 161, 8, 3), (8251, 256, 322, 8, 8), (40003, 256, 320, 8, 8), (2077, 512, 800, 16, 14),
    (10951, 96, 131, 3, 3), (15437, 68, 69, 4, 2), (2100, 500, 4099, 8, 8),
])
def test_backward_tiles(native_lib, cuda_device, T, L, P, D, copies):
    rng = np.random.default_rng(T)
    counts = np.minimum(rng.integers(1, copies + 1, size=L), D)
    counts[rng.random(L) < 0.5] = 1
    while counts.sum() > P:
        counts[np.argmax(counts)] -= 1
    slots, at = rng.permutation(P), 0
    l2p = np.full((L, D), -1, np.int32)
    for e, c in enumerate(counts):
        l2p[e, :c] = slots[at:at + c]
        at += c
    z = np.zeros((L, D), np.int32)
    plan = O.Plan(np.zeros(P, np.int32), l2p, counts.astype(np.int32), z, z, z)
    rmap = rng.random((T, L), dtype=np.float32) < 0.06
    rmap[T // 2] = True  # a full row, more than a warp's round of cells
    rmap[:, 0] = True
    took = rng.random((T, P), dtype=np.float32) < 0.4  # none, one or several instances of a cell
    grad = rng.normal(size=(T, P)).astype(np.float32)
    exp = O.dense_reroute_backward(grad, rmap, took, plan)
    dev = lambda x: torch.from_numpy(x).to(cuda_device)
    got = G.cuda_dense_reroute_backward(dev(grad), dev(rmap), dev(took), dev(l2p), dev(plan.lcnts))
    assert np.array_equal(got.cpu().numpy().view(np.uint32), exp.view(np.uint32))
