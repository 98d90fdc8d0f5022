"""Reroute of eight hosted ranks in one launch with uneven token counts (none, one, a tile and one entry more, thousands), whose
grid is the longest rank's: ids of both widths, in place and not, with and without a weight_sync beside it, against the CPU
oracle. Whole numbers and copies: bit-exact."""

import numpy as np
import pytest
import torch

from oracle import uep_oracle as O
from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu
N, K, R = 8, 8, 2

TOKENS = {  # entries of the longest rank: one cluster's, a tile more, the walk alone, behind the repeated counting
    "one cluster": [0, 1, 300, 2048, 33, 700, 257, 1500],
    "tiles": [0, 1, 300, 2049, 33, 700, 2048, 1500],
    "long": [8193, 0, 5, 1, 4097, 64, 8192, 2100],
    "longest": [32800, 1, 7, 0, 513, 4096, 2, 16],
}


def _case(tokens, L, seed, device):
    rng = np.random.default_rng(seed)
    pop = -1.3 * np.log(rng.permutation(L) + 1.0)
    ids = [np.argsort(-(pop + rng.gumbel(size=(t, L))), axis=1)[:, :K].astype(np.int32).reshape(t, K) for t in tokens]
    lpr = np.stack([np.bincount(x.reshape(-1), minlength=L) for x in ids]).astype(np.int32)
    return ids, [O.solve_placement(lpr, L // N, R, N, r) for r in range(N)], [torch.from_numpy(x).to(device) for x in ids]


@pytest.mark.parametrize("tokens", TOKENS)
@pytest.mark.parametrize("L,beside", [(64, False), (64, True), (256, True), (72, False)])
def test_hosted_reroute_of_uneven_ranks(native_lib, cuda_device, tokens, L, beside):
    ids, plans, dev = _case(TOKENS[tokens], L, L, cuda_device)
    group = sim.SimGroup(sim.make_config(N, L // N, R, 1, fc1_numel=64, fc2_numel=64, is_train=True, sim=True))
    group.update_placement(0, dev)
    tables = [group.pointer_tables([[torch.zeros(64, dtype=torch.bfloat16, device=cuda_device)] * (L // N)] * N) for _ in range(2)]
    want = [O.sparse_reroute(x, p, True) if len(x) else x for x, p in zip(ids, plans)]
    for dtype in (torch.int32, torch.int64):
        for in_place in (False, True):
            done = group.weight_sync(0, *tables, async_finish=True) if beside else None
            src = [x.to(dtype, copy=True) for x in dev]
            got = group.reroute_sparse(0, src, src if in_place else None)
            if done is not None:
                group.wait_event(done)
            for g, w in zip(got, want):
                assert g.dtype == dtype and np.array_equal(g.cpu().numpy(), w)
            group.update_placement(0, dev)
    if tokens != "longest":
        maps = [torch.zeros((len(x), L), dtype=torch.bool, device=cuda_device).scatter_(1, x.long(), True) for x in dev]
        probs = [torch.rand(m.shape, device=cuda_device) * m for m in maps]
        out_probs, out_maps = group.reroute_dense(0, maps, probs)
        grads = [torch.randn(p.shape, device=cuda_device) for p in out_probs]
        back = group.reroute_dense_backward(0, grads, maps, out_maps)
        for m, p, plan, op, om, g, b in zip(maps, probs, plans, out_probs, out_maps, grads, back):
            if len(m) == 0:
                continue
            exp_probs, exp_map = O.dense_reroute_forward(m.cpu().numpy(), p.cpu().numpy(), plan, group.P, True)
            assert np.array_equal(om.cpu().numpy(), exp_map) and np.array_equal(op.cpu().numpy().view(np.uint32), exp_probs.view(np.uint32))
            exp = O.dense_reroute_backward(g.cpu().numpy(), m.cpu().numpy(), exp_map, plan)
            assert np.array_equal(b.cpu().numpy().view(np.uint32), exp.view(np.uint32))
    group.check_status()
