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


def _group(ranks, masters, redundant, fc1, fc2, tokens, fill_slots=False, **kw):
    """A group with a skewed plan in which every rank has hot masters, or with a plan that uses every slot; replica gradients to
    reduce, and what the reduce must leave."""
    group = sim.SimGroup(sim.make_config(ranks, masters, redundant, 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=16,
                                         is_train=True, sim=True, grad_reduce_num_sms=4, **kw))
    dev, L = group.device, ranks * masters
    gen = torch.Generator(device=dev).manual_seed(L)
    keys = (-1.5 * torch.log(torch.arange(L, device=dev) + 1.0)).view(masters, ranks).t().reshape(-1)
    ids = []
    for _ in range(ranks):
        u = torch.rand((tokens, L), generator=gen, device=dev).clamp(1e-30, 1 - 1e-7)
        ids.append(torch.topk(keys - torch.log(-torch.log(u)), 4, dim=1).indices.int())
    group.update_placement(0, ids)
    if fill_slots:  # every master has one replica, on another rank: written over the solved plan
        for me in range(ranks):
            p = group.plan(me, 0)
            for r in range(ranks):
                for s in range(redundant):
                    l, phys = (r + 1 + s % (ranks - 1)) % ranks * masters + s, r * (masters + redundant) + masters + s
                    p["lcnts"][l], p["l2p"][l, 1], p["p2l"][phys] = 2, phys, l
    plan = {k: v.cpu() for k, v in group.plan(0, 0).items()}
    slots = [(l, *divmod(int(plan["l2p"][l, j]), masters + redundant)) for l in range(L) for j in range(1, int(plan["lcnts"][l]))]
    grads = [[[torch.randn(n, generator=gen, device=dev) for _ in range(masters)] for _ in range(ranks)] for n in (fc1, fc2)]
    replicas = [group.buffer(r, capi.BUF_REPLICA_GRAD) for r in range(ranks)]

    def fill():
        for t in replicas:
            t.normal_(0.0, 1.0, generator=gen)
        want_replicas = [t.clone() for t in replicas]
        want = [[[t.clone() for t in row] for row in g] for g in grads]
        for l, rank, slot in slots:
            row = want_replicas[rank][slot - masters]
            want[0][l // masters][l % masters] += row[:fc1]
            want[1][l // masters][l % masters] += row[fc1:]
        return want_replicas, want

    def reduce():
        group.grad_reduce(0, *[group.pointer_tables(g) for g in grads])
        torch.cuda.synchronize()

    def check(want_replicas, want, kept=()):
        for l, rank, slot in slots:
            if l // masters not in kept:
                want_replicas[rank][slot - masters].zero_()
        for got, exp in zip(replicas, want_replicas):
            assert torch.equal(got, exp)
        for g, w in zip(grads, want):
            for got_row, exp_row in zip(g, w):
                for got, exp in zip(got_row, exp_row):
                    assert torch.equal(got, exp)

    return group, slots, fill, reduce, check


# bulk stores and, with sizes that are no multiple of four, plain ones; a tile is 4096 elements, a release a 16th of the tiles
@pytest.mark.parametrize("fc1,fc2", [(40 * 4096, 37 * 4096 + 4), (21 * 4096 + 1, 18 * 4096 + 2)])
def test_a_rank_that_reports_nothing_holds_back_its_own_slots_only(native_lib, cuda_device, fc1, fc2):
    group, slots, fill, reduce, check = _group(RANKS, MASTERS, REDUNDANT, fc1, fc2, 512, wait_timeout_ms=150)
    owners = sorted({l // MASTERS for l, _, _ in slots})
    assert len(owners) > 1
    victim = owners[0]
    want = fill()
    capi.check(group.lib.uep_debug_withhold_rank(group.handle, victim))
    reduce()
    assert group.status(0)[0] == 2  # a wait for a progress word ran out
    check(*want, kept=(victim,))
    capi.check(group.lib.uep_debug_withhold_rank(group.handle, -1))
    capi.check(group.lib.uep_clear_status(group.handle))
    for owners_clear in (False, True):  # and the calls behind it are whole again
        if owners_clear:
            capi.check(group.lib.uep_debug_withhold_rank(group.handle, RANKS))
        want = fill()
        reduce()
        group.check_status()
        check(*want)
    group.destroy()


def test_more_slots_than_a_warp_has_lanes(native_lib, cuda_device):
    group, slots, fill, reduce, check = _group(8, 8, 8, 9 * 4096, 8 * 4096 + 8, 64, fill_slots=True)
    assert len(slots) == 64
    capi.check(group.lib.uep_debug_withhold_rank(group.handle, 8))
    for _ in range(2):
        want = fill()
        reduce()
        group.check_status()
        check(*want)
    group.destroy()
