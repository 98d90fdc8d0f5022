"""Which side clears a consumed replica gradient: the CTA that pulled it, where the replica lies on a rank of the same launch,
else its owner. Both leave the same bits."""

import pytest
import torch

from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu

RANKS, MASTERS, REDUNDANT = 4, 4, 3


# a tile is 4096 elements: one element short of it, one vector more, several rounds of a CTA's rings, and a size that is
# no multiple of four (plain loads)
@pytest.mark.parametrize("fc1,fc2,ctas", [(4, 4092, 2), (4100, 8192, 2), (40 * 4096, 37 * 4096 + 4, 2), (4101, 6, 2), (12288, 4096, 42)])
@pytest.mark.parametrize("owners", [False, True])
def test_reduce_clears_what_it_consumed(native_lib, cuda_device, fc1, fc2, ctas, owners):
    group = sim.SimGroup(sim.make_config(RANKS, MASTERS, REDUNDANT, 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=16,
                                         is_train=True, sim=True, grad_reduce_num_sms=ctas))
    gen = torch.Generator(device=cuda_device).manual_seed(fc1 + fc2)
    L = RANKS * MASTERS
    keys = -1.5 * torch.log(torch.arange(L, device=cuda_device) + 1.0)
    ids = []
    for _ in range(RANKS):
        u = torch.rand((512, L), generator=gen, device=cuda_device).clamp(1e-30, 1 - 1e-7)
        ids.append(torch.topk(keys - torch.log(-torch.log(u)), 4, dim=1).indices.int())
    group.update_placement(0, ids)
    plan = {k: v.cpu() for k, v in group.plan(0, 0).items()}
    assert int((plan["lcnts"] - 1).sum()) > 2  # some master has several replicas or several have one

    grads = [[[torch.randn(n, generator=gen, device=cuda_device) for _ in range(MASTERS)] for _ in range(RANKS)] for n in (fc1, fc2)]
    tables = [group.pointer_tables(g) for g in grads]
    replicas = [group.buffer(r, capi.BUF_REPLICA_GRAD) for r in range(RANKS)]
    if owners:
        capi.check(group.lib.uep_debug_withhold_rank(group.handle, RANKS))  # no such rank: nobody is withheld
    for _ in range(2):  # the second call continues the epochs and the barriers of a new launch
        for t in replicas:
            t.normal_(0.0, 1.0, generator=gen)
        want_replicas = [t.clone() for t in replicas]
        want = [[[t.clone() for t in row] for row in g] for g in grads]
        for l in range(L):
            for j in range(1, int(plan["lcnts"][l])):
                rank, slot = divmod(int(plan["l2p"][l, j]), MASTERS + REDUNDANT)
                row = want_replicas[rank][slot - MASTERS]
                want[0][l // MASTERS][l % MASTERS] += row[:fc1]
                want[1][l // MASTERS][l % MASTERS] += row[fc1:]
                row.zero_()
        group.wait_event(group.grad_reduce(0, *tables, async_finish=True))
        torch.cuda.synchronize()
        group.check_status()
        for got, exp in zip(replicas, want_replicas):
            assert torch.equal(got, exp)
        for g, w in zip(grads, want):
            for got_row, exp_row in zip(g, w):
                for got, exp in zip(got_row, exp_row):
                    assert torch.equal(got, exp)
    group.destroy()
