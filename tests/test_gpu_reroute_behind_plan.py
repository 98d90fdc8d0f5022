"""The reroute may count its tokens while the plan in front of it in the stream is still being made. It must use that plan all the
same, and the ids as the stream leaves them: eager, behind a kernel or another stream's event in between, and replayed as a graph."""

import pytest
import torch

import gpu_util as G
from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu

RANKS, L, K = 8, 64, 8


def _draw(tokens, dtype, seed, device):
    gen = torch.Generator(device=device).manual_seed(seed)
    out = []
    for r in range(RANKS):
        order = torch.randperm(L, generator=gen, device=device) if r == 0 else order
        keys = -1.4 * torch.log(order.float() + 1.0)
        u = torch.rand((max(tokens - 3 * r, 1), L), generator=gen, device=device).clamp(1e-30, 1 - 1e-7)
        out.append(torch.topk(keys - torch.log(-torch.log(u)), K, dim=1).indices.to(dtype))
    return out


def _expect(group, ids):
    torch.cuda.synchronize()
    group.check_status()
    plans = [group.plan(r, 0) for r in range(RANKS)]
    return [G.cuda_sparse_reroute(x, p["l2p"].contiguous(), p["lcnts"].contiguous(), p["rank_quota_prefix"].contiguous())
            for x, p in zip(ids, plans)]


# one launch over clusters, a count kernel in front, and the walk
@pytest.mark.parametrize("tokens", [1, 33, 600, 4099, 9000])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_sparse(native_lib, cuda_device, tokens, dtype):
    group = sim.SimGroup(sim.make_config(RANKS, L // RANKS, 2, 1, is_train=False, sim=True))
    ids = _draw(tokens, dtype, 0, cuda_device)
    other = torch.cuda.Stream()
    for seed in range(1, 9):
        fresh = _draw(tokens, dtype, seed, cuda_device)
        last = _draw(tokens, dtype, seed + 100, cuda_device)
        torch.cuda.synchronize()
        for dst, src in zip(ids, fresh):
            dst.copy_(src)
        group.update_placement(0, ids)
        got = group.reroute_sparse(0, ids)
        for a, b in zip(got, _expect(group, fresh)):
            assert torch.equal(a, b), seed
        group.update_placement(0, ids)  # the ids change between the plan and the reroute, in the stream itself
        for dst, src in zip(ids, last):
            dst.copy_(src)
        got = group.reroute_sparse(0, ids)
        for a, b in zip(got, _expect(group, last)):
            assert torch.equal(a, b), seed
        with torch.cuda.stream(other):  # ... and in another one that it waits for
            torch.cuda._sleep(200_000)
            for dst, src in zip(ids, fresh):
                dst.copy_(src)
        group.update_placement(0, last)
        torch.cuda.current_stream().wait_stream(other)
        got = group.reroute_sparse(0, ids)
        for a, b in zip(got, _expect(group, fresh)):
            assert torch.equal(a, b), seed
        group.update_placement(0, ids)  # in place
        want = [x.clone() for x in fresh]
        group.reroute_sparse(0, ids, ids)
        for a, b in zip(ids, _expect(group, want)):
            assert torch.equal(a, b), seed
    group.destroy()


@pytest.mark.parametrize("tokens", [1, 65, 3000])
def test_dense(native_lib, cuda_device, tokens):
    group = sim.SimGroup(sim.make_config(RANKS, L // RANKS, 2, 1, is_train=True, sim=True))
    for seed in range(6):
        maps = [torch.zeros((x.shape[0], L), dtype=torch.bool, device=cuda_device).scatter_(1, x, True)
                for x in _draw(tokens, torch.int64, seed, cuda_device)]
        probs = [torch.rand(m.shape, device=cuda_device) * m for m in maps]
        group.update_placement(0, maps)
        got_probs, got_maps = group.reroute_dense(0, maps, probs)
        torch.cuda.synchronize()
        group.check_status()
        for r in range(RANKS):
            p = group.plan(r, 0)
            want_probs, want_map = G.cuda_dense_reroute(maps[r], probs[r], p["l2p"].contiguous(), p["lcnts"].contiguous(),
                                                        p["rank_quota_prefix"].contiguous(), group.P)
            assert torch.equal(got_probs[r], want_probs) and torch.equal(got_maps[r], want_map), (seed, r)
    group.destroy()


@pytest.mark.parametrize("tokens", [33, 4099])
def test_replayed(native_lib, cuda_device, tokens):
    group = sim.SimGroup(sim.make_config(RANKS, L // RANKS, 2, 1, is_train=False, sim=True))
    ids = _draw(tokens, torch.int32, 0, cuda_device)
    out = [torch.empty_like(x) for x in ids]

    def step():
        group.update_placement(0, ids)
        group.reroute_sparse(0, ids, out)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()  # sizes the scratch
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for seed in range(1, 6):
        for dst, src in zip(ids, _draw(tokens, torch.int32, seed, cuda_device)):
            dst.copy_(src)
        graph.replay()
        graph.replay()
        for a, b in zip(out, _expect(group, ids)):
            assert torch.equal(a, b), seed
    group.destroy()


def test_gather_behind_positions(native_lib, cuda_device):
    gen = torch.Generator(device=cuda_device).manual_seed(3)
    for n in (1, 31, 4096, 70001):
        rows = torch.randn((n, 72), generator=gen, device=cuda_device)
        phys = torch.randint(0, 80, (n,), generator=gen, device=cuda_device, dtype=torch.int32)
        pos, _ = G.cuda_dispatch_positions(phys, 80)
        out, status = G.cuda_gather_rows(rows, pos)
        torch.cuda.synchronize()
        assert not status.any()
        assert torch.equal(out, rows[pos.long()])
