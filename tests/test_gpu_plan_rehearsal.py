"""Plans of hosted groups whose inputs are large: 256 or 512 threads that count, bytes of the bool map summed in a warp before they are
counted, and a second crew of threads in the owners' CTAs that rehearses the solver on a problem of its own beside them. The widths of the map
decide how the lanes share the sums; the smallest group is smaller than the rehearsal's. Loads and plan against the CPU oracle,
bit-exact, twice in a row."""

import ctypes as C

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu

# ranks, masters, slots, tokens. 512 threads count from 22 KB of input for each CTA that a rank has (two ranks have 32 each, eight 15):
# 45056 and 45057 are on either side of that line. The last ones' rows are no whole vectors, and are counted byte by byte.
SHAPES = [(8, 16, 4, 1100), (2, 1, 1, 300000), (2, 8, 1, 40000), (3, 32, 2, 9000), (5, 5, 2, 25000), (7, 16, 0, 5000), (8, 4, 2, 12000), (8, 64, 8, 1500),
          (2, 1, 1, 400000), (2, 8, 1, 50000), (8, 16, 4, 9000), (2, 8, 1, 45056), (2, 8, 1, 45057),
          (6, 20, 2, 4000), (3, 40, 2, 5561), (7, 10, 2, 1000), (8, 15, 2, 8192), (5, 1, 1, 70000), (2, 255, 1, 3000)]


@pytest.mark.parametrize("N,M,R,T", SHAPES)
def test_large_maps(native_lib, cuda_device, N, M, R, T):
    L = N * M
    group = sim.SimGroup(sim.make_config(N, M, R, 1, fc1_numel=64, fc2_numel=64, is_train=True, sim=True))
    for seed in (1, 2):
        gen = torch.Generator(device=cuda_device).manual_seed(seed)
        popular = torch.rand(L, generator=gen, device=cuda_device) ** 4
        maps = [torch.rand((T - 17 * r, L), generator=gen, device=cuda_device) < popular for r in range(N)]
        maps[0][:, 0] = True  # a byte of every row: the largest sums
        group.update_placement(0, maps)
        torch.cuda.synchronize()
        loads = np.stack([m.sum(0).cpu().numpy() for m in maps]).astype(np.int32)
        for r in range(N):
            want = O.solve_placement(loads, M, R, N, r)
            got = group.plan(r, 0)
            for f in ("p2l", "l2p", "lcnts", "quota", "quota_prefix", "rank_quota_prefix"):
                assert np.array_equal(got[f].cpu().numpy().reshape(-1), getattr(want, f).reshape(-1)), (seed, r, f)
    group.check_status()
    group.destroy()


def test_who_rehearses(native_lib, cuda_device):
    """A group that is hosted whole and has something to solve by quotas; not one rank among ranks on other devices."""
    def form(N, R, hosted, legacy=0):
        cfg = sim.make_config(N, 4, R, 1, is_train=True, sim=hosted)
        cfg.legacy_placement = legacy
        handle = C.c_void_p()
        capi.check(capi.lib().uep_manager_create(C.byref(cfg), C.byref(handle)))
        got = capi.lib().uep_debug_plan_form(handle)
        capi.check(capi.lib().uep_manager_destroy(handle))
        return got

    assert [form(2, 1, True), form(8, 2, True), form(8, 0, True), form(1, 2, True), form(8, 2, True, legacy=1)] == [3, 3, 1, 1, 1]
    assert [form(2, 1, False), form(8, 2, False), form(1, 2, False)] == [0, 0, 1]


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("N,M,R,T,K", [(2, 3, 1, 50, 2), (3, 5, 2, 4000, 4), (8, 16, 4, 8192, 8), (8, 64, 8, 33, 8), (8, 2, 1, 9000, 4)])
def test_rehearsal_of_what_is_out_of_line(native_lib, cuda_device, kind, N, M, R, T, K):
    """A rehearsal that comes to the probes or to wide keys, whose code takes the shared memory of the plan beside it, leaves that alone."""
    L = N * M
    group = sim.SimGroup(sim.make_config(N, M, R, 1, is_train=True, sim=True))
    capi.check(group.lib.uep_debug_hard_rehearsal(group.handle, kind))
    for seed in range(4):
        rng = np.random.default_rng(seed)
        ids = [np.minimum(rng.geometric(0.15, size=(T, K)) - 1, L - 1).astype(np.int32) for _ in range(N)]
        group.update_placement(0, [torch.from_numpy(x).to(cuda_device) for x in ids])
        torch.cuda.synchronize()
        group.check_status()
        loads = np.stack([np.bincount(x.reshape(-1), minlength=L) for x in ids]).astype(np.int32)
        for r in range(N):
            want, got = O.solve_placement(loads, M, R, N, r), group.plan(r, 0)
            for f in ("p2l", "l2p", "lcnts", "quota", "quota_prefix", "rank_quota_prefix"):
                assert np.array_equal(got[f].cpu().numpy().reshape(-1), getattr(want, f).reshape(-1)), (seed, r, f)
    group.destroy()


# around eight rounds of a CTA's threads and the last one's rest, one column to more than threads, rows that begin anywhere in memory
@pytest.mark.parametrize("T,L", [(1, 1), (255, 1), (2049, 1), (3, 5), (700, 7), (4099, 24), (1000, 100), (33, 257), (9, 5001), (300, 64)])
@pytest.mark.parametrize("offset", [0, 1, 7])
def test_counts_byte_by_byte(native_lib, cuda_device, T, L, offset):
    gen = torch.Generator(device=cuda_device).manual_seed(T * L + offset)
    flat = torch.rand(T * L + offset, generator=gen, device=cuda_device) < 0.3
    flat.view(torch.uint8)[::3] *= 255  # any byte but zero counts once
    rmap = flat[offset:].view(T, L)
    want = (rmap.view(torch.uint8) != 0).sum(0, dtype=torch.int32)
    if L % 16 == 0 and offset == 0:
        pytest.skip("whole vectors")
    assert torch.equal(G.cuda_histogram(rmap, L, "map"), want)
