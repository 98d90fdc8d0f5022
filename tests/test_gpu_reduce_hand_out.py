"""The reduce of a group hosted whole hands its items to the CTAs as they ask for them where experts are long: the same bits, every replica
cleared, and counters that the next launch finds as this one did."""

import pytest
import torch

from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu

RANKS, MASTERS, REDUNDANT, TILE = 4, 4, 3, 4096
SLOTS = MASTERS + REDUNDANT


def _write_plan(group, masters_of):
    """masters_of[rank]: the masters (of other ranks) that its redundant slots hold, in turn."""
    where = {}
    for rank, row in enumerate(masters_of):
        for s, l in enumerate(row):
            where.setdefault(l, []).append((rank, s))
    for me in range(RANKS):
        p = group.plan(me, 0)
        p["lcnts"].fill_(1)
        p["l2p"][:, 1:] = -1
        p["p2l"].view(RANKS, SLOTS)[:, MASTERS:] = -1
        for l, at in where.items():
            p["lcnts"][l] = 1 + len(at)
            for j, (rank, s) in enumerate(at):
                phys = rank * SLOTS + MASTERS + s
                p["l2p"][l, 1 + j], p["p2l"][phys] = phys, l
    return where


EACH = [[(r + 1 + s) % RANKS * MASTERS + s for s in range(REDUNDANT)] for r in range(RANKS)]  # twelve masters, a replica each
ELEVEN = [row[:2] if r == 2 else row for r, row in enumerate(EACH)]
HOT = [[4, 8], [0, 1, 12], [0, 1], [0, 4]]  # five masters: three replicas, two and one
FOUR = [[4], [0, 8], [0, 12], [0, 4]]


# 2048 tiles an expert and 64 items a CTA are the lines. A tile below the first; on it, and below and above the second in the kernel that
# could (four masters and five on 144 CTAs); runs of two and of many items; sizes with a remainder in either matrix; an odd number of items.
@pytest.mark.parametrize("masters_of,fc1,fc2,ctas", [
    (EACH, 1300 * TILE - 4, 747 * TILE, 36), (FOUR, 1300 * TILE - 4, 748 * TILE, 36), (HOT, 1300 * TILE - 4, 748 * TILE, 36),
    (ELEVEN, 2047 * TILE + 4, 4, 36), (ELEVEN, 8, 2048 * TILE + 12, 8), (EACH, 1500 * TILE, 601 * TILE - 4, 2), (HOT, 1100 * TILE + 2, 1000 * TILE, 36),
    # six sevenths of 148 SMs are the third line
    (EACH, 1300 * TILE - 4, 748 * TILE, 30), (EACH, 1300 * TILE - 4, 748 * TILE, 32), (ELEVEN, 8, 2048 * TILE + 12, 32)])
def test_items_handed_out(native_lib, cuda_device, masters_of, fc1, fc2, ctas):
    group = sim.SimGroup(sim.make_config(RANKS, MASTERS, REDUNDANT, 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=16,
                                         is_train=True, sim=True, grad_reduce_num_sms=ctas))
    gen = torch.Generator(device=cuda_device).manual_seed(fc1 + fc2)
    where = _write_plan(group, masters_of)
    grads = [[[torch.randn(n, generator=gen, device=cuda_device) for _ in range(MASTERS)] for _ in range(RANKS)] for n in (fc1, fc2)]
    tables = [group.pointer_tables(g) for g in grads]
    replicas = [group.buffer(r, capi.BUF_REPLICA_GRAD) for r in range(RANKS)]
    for _ in range(3):
        for t in replicas:
            t.normal_(0.0, 1.0, generator=gen)
        want = [[[t.clone() for t in row] for row in g] for g in grads]
        want_replicas = [t.clone() for t in replicas]
        for l, at in where.items():
            for rank, s in at:  # in the order of the instances, as 32-bit sums
                row = want_replicas[rank][s]
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


@pytest.mark.parametrize("ctas", [2, 36])
def test_items_without_a_replica(native_lib, cuda_device, ctas):
    """A plan with an entry that names no slot: reported, its master left as it is, the others reduced."""
    fc1, fc2 = 1400 * TILE, 700 * TILE
    group = sim.SimGroup(sim.make_config(RANKS, MASTERS, REDUNDANT, 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=16,
                                         is_train=True, sim=True, grad_reduce_num_sms=ctas))
    where = _write_plan(group, EACH)
    bad = EACH[1][1]
    for me in range(RANKS):
        group.plan(me, 0)["l2p"][bad, 1] = -1
    grads = [[[torch.ones(n, device=cuda_device) for _ in range(MASTERS)] for _ in range(RANKS)] for n in (fc1, fc2)]
    replicas = [group.buffer(r, capi.BUF_REPLICA_GRAD) for r in range(RANKS)]
    for t in replicas:
        t.fill_(2.0)
    group.grad_reduce(0, *[group.pointer_tables(g) for g in grads])
    torch.cuda.synchronize()
    assert group.status(0)[0] != 0 or any(group.status(r)[0] != 0 for r in range(RANKS))
    for l in range(RANKS * MASTERS):
        want = 3.0 if l in where and l != bad else 1.0
        for g in grads:
            assert torch.equal(g[l // MASTERS][l % MASTERS], torch.full_like(g[l // MASTERS][l % MASTERS], want))
    for l, at in where.items():
        for rank, s in at:
            assert torch.equal(replicas[rank][s], torch.full_like(replicas[rank][s], 2.0 if l == bad else 0.0))
    group.destroy()


def test_runs_of_many_items(native_lib, cuda_device):
    """More items than the CTAs can keep runs of two: four masters of 37 000 tiles, a replica each, on 128 CTAs. Twice."""
    fc1, fc2 = 36998 * TILE + 16, 2 * TILE
    group = sim.SimGroup(sim.make_config(RANKS, 1, 1, 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=1, is_train=True, sim=True,
                                         grad_reduce_num_sms=32))
    for me in range(RANKS):
        p = group.plan(me, 0)
        p["lcnts"].fill_(2)
        for l in range(RANKS):
            phys = (l + 1) % RANKS * 2 + 1
            p["l2p"][l, 1], p["p2l"][phys] = phys, l
    gen = torch.Generator(device=cuda_device).manual_seed(5)
    grads = [[[torch.randn(n, generator=gen, device=cuda_device)] for _ in range(RANKS)] for n in (fc1, fc2)]
    tables = [group.pointer_tables(g) for g in grads]
    replicas = [group.buffer(r, capi.BUF_REPLICA_GRAD) for r in range(RANKS)]
    for _ in range(2):
        for t in replicas:
            t.normal_(0.0, 1.0, generator=gen)
        want = [[grads[0][r][0] + replicas[(r + 1) % RANKS][0][:fc1], grads[1][r][0] + replicas[(r + 1) % RANKS][0][fc1:]] for r in range(RANKS)]
        group.grad_reduce(0, *tables)
        torch.cuda.synchronize()
        group.check_status()
        for r in range(RANKS):
            assert torch.equal(grads[0][r][0], want[r][0]) and torch.equal(grads[1][r][0], want[r][1]), r
            assert not replicas[r].any()
    group.destroy()
