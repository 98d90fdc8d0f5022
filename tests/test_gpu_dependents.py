"""Plans, solves, positions and backwards are dependent launches: behind a kernel that starts its dependents early and writes their input
later, they use what it has written. The plan hands its rows over inside a cluster: groups of one to eight ranks, widths whose rows
are not whole vectors, one CTA a rank and many, one rank without tokens. Against the CPU oracle, bit-exact."""

import ctypes as C

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_reroute_behind_plan import late_write  # noqa: F401  (fixture)
from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu

FIELDS = ("p2l", "l2p", "lcnts", "quota", "quota_prefix", "rank_quota_prefix")


def _group_input(kind, N, L, T, seed):
    """(one flat array, each rank's slice and shape, loads): ids with values outside [0, L), or a map; the last rank has no tokens."""
    rng = np.random.default_rng(seed)
    parts = []
    for r in range(N):
        t = 0 if N > 2 and r == N - 1 else T - r
        if kind == "map":
            parts.append(rng.random((t, L)) < rng.random(L) ** 3)
        else:
            parts.append(np.minimum(rng.geometric(0.2, size=(t, 4)) - 2, L).astype(kind))
    loads = np.stack([p.sum(0) if kind == "map" else np.bincount(p[(p >= 0) & (p < L)].reshape(-1), minlength=L) for p in parts])
    return np.concatenate([p.reshape(-1) for p in parts]), [p.shape for p in parts], loads.astype(np.int32)


@pytest.mark.parametrize("N,M,R", [(1, 5, 1), (2, 3, 1), (3, 5, 2), (5, 2, 1), (7, 4, 2), (8, 1, 1), (8, 16, 4), (8, 64, 2)])
@pytest.mark.parametrize("kind,T", [("int32", 9), ("int64", 3001), ("map", 40), ("map", 2600)])
def test_plan_behind_an_early_kernel(native_lib, cuda_device, late_write, N, M, R, kind, T):
    L = N * M
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=True, sim=True))
    for seed in range(3):
        data, shapes, _ = _group_input(kind, N, L, T, seed)
        late, _, loads = _group_input(kind, N, L, T, seed + 10)
        flat, source = torch.from_numpy(data).to(cuda_device), torch.from_numpy(late).to(cuda_device)
        views, at = [], 0
        for shape in shapes:
            views.append(flat[at:at + shape[0] * shape[1]].view(shape))
            at += shape[0] * shape[1]
        group.update_placement(0, views)  # of what is overwritten
        late_write(flat.view(torch.uint8), source.view(torch.uint8), seed % 2 == 1)
        group.update_placement(0, views)
        torch.cuda.synchronize()
        group.check_status()
        for r in range(N):
            want, got = O.solve_placement(loads, M, R, N, r), group.plan(r, 0)
            for f in FIELDS:
                assert np.array_equal(got[f].cpu().numpy().reshape(-1), getattr(want, f).reshape(-1)), (seed, r, f)
    group.destroy()


@pytest.mark.parametrize("N,M,R", [(8, 4, 2), (40, 3, 1)])
def test_solve_behind_an_early_kernel(native_lib, cuda_device, late_write, N, M, R):
    L, P = N * M, N * (M + R)
    rng = np.random.default_rng(N)
    lib, params = capi.lib(), capi.SolverParams.defaults()
    shapes = dict(p2l=P, l2p=L * N, lcnts=L, quota=L * N, quota_prefix=L * N, rank_quota_prefix=L * N)
    out = {k: torch.empty(n, dtype=torch.int32, device=cuda_device) for k, n in shapes.items()}
    total, status = torch.empty(L, dtype=torch.int32, device=cuda_device), torch.zeros(2, dtype=torch.int32, device=cuda_device)
    for seed in range(4):
        old, new = ((rng.random((N, L)) ** 6 * 3000).astype(np.int32) for _ in range(2))
        loads, source = torch.from_numpy(old).to(cuda_device), torch.from_numpy(new).to(cuda_device)
        torch.cuda.synchronize()
        late_write(loads, source, seed % 2 == 1)
        capi.check(lib.uep_solve_placement(loads.data_ptr(), total.data_ptr(), *(out[k].data_ptr() for k in FIELDS), N, N, M, R, N, C.byref(params), 0,
                                           status.data_ptr(), G.stream_ptr()))
        torch.cuda.synchronize()
        want = O.solve_placement(new, M, R, N, 0)
        assert not status.any() and np.array_equal(total.cpu().numpy(), new.sum(0))
        for f in FIELDS:
            assert np.array_equal(out[f].cpu().numpy().reshape(-1), getattr(want, f).reshape(-1)), (seed, f)


# one launch and two (n > 2^18)
@pytest.mark.parametrize("n", [100, 70000, 262145])
def test_positions_behind_an_early_kernel(native_lib, cuda_device, late_write, n):
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    draw = lambda: torch.randint(0, 80, (n,), generator=gen, device=cuda_device, dtype=torch.int32)
    for dependent in (False, True, True):
        phys, late = draw(), draw()
        want = torch.empty_like(phys)
        want[torch.argsort(late, stable=True)] = torch.arange(n, dtype=torch.int32, device=cuda_device)
        torch.cuda.synchronize()
        late_write(phys, late, dependent)
        pos, _ = G.cuda_dispatch_positions(phys, 80)
        torch.cuda.synchronize()
        assert torch.equal(pos, want)


# cell by cell, and tiles
@pytest.mark.parametrize("tokens", [30, 1500])
def test_backward_of_several_ranks_behind_an_early_kernel(native_lib, cuda_device, late_write, tokens):
    N, M, R = 8, 16, 2
    L, P = N * M, N * (M + R)
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=True, sim=True))
    gen = torch.Generator(device=cuda_device).manual_seed(tokens)
    maps = [torch.rand((tokens, L), generator=gen, device=cuda_device) < 0.05 for _ in range(N)]
    probs = [torch.rand((tokens, L), generator=gen, device=cuda_device) for _ in range(N)]
    group.update_placement(0, maps)
    _, expanded = group.reroute_dense(0, maps, probs)
    for dependent in (False, True, True):
        late = torch.randn((N, tokens, P), generator=gen, device=cuda_device)
        grads = torch.randn((N, tokens, P), generator=gen, device=cuda_device)
        torch.cuda.synchronize()
        late_write(grads, late, dependent)
        got = group.reroute_dense_backward(0, list(grads), maps, expanded)
        torch.cuda.synchronize()
        for r in range(N):
            p = group.plan(r, 0)
            want = G.cuda_dense_reroute_backward(late[r], maps[r], expanded[r], p["l2p"].contiguous(), p["lcnts"].contiguous())
            assert torch.equal(got[r], want), r
    group.destroy()
