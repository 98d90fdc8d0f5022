"""How the ranks of a plan hand each other their load rows: inside a cluster, as a group that is hosted whole does, and in words through
memory, as ranks of several devices do (which the hook that withholds a rank asks for, also with a rank that does not exist). To a good
end against the CPU oracle, bit-exact, in turn on one group; and with one rank's row missing, which the others name."""

import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from oracle import uep_oracle as O
from test_gpu_dependents import FIELDS, _group_input
from test_gpu_reroute_behind_plan import late_write  # noqa: F401  (fixture)
from test_gpu_sync_repeats import _ids
from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu

IN_CLUSTER = 1
TIMEOUT_GATHER = 1


def _through_memory(group, on):
    capi.check(group.lib.uep_debug_withhold_rank(group.handle, group.N if on else -1))
    assert bool(group.lib.uep_debug_plan_form(group.handle) & IN_CLUSTER) == (not on)


def _inputs(kind, N, L, T, seed, device):
    flat, shapes, loads = _group_input(kind, N, L, T, seed)
    views, at = [], 0
    for shape in shapes:
        views.append(torch.from_numpy(flat[at:at + shape[0] * shape[1]].reshape(shape)).to(device))
        at += shape[0] * shape[1]
    return views, loads


def _assert_plan(group, layer, want, r):
    got = group.plan(r, layer)
    for f in FIELDS:
        assert np.array_equal(got[f].cpu().numpy().reshape(-1), getattr(want, f).reshape(-1)), (r, f)


@pytest.mark.parametrize("N,M,R", [(1, 5, 1), (2, 3, 1), (3, 5, 2), (7, 4, 2), (8, 1, 1), (8, 16, 4), (8, 64, 2)])
@pytest.mark.parametrize("kind,T", [("int32", 9), ("map", 2600)])
@pytest.mark.parametrize("legacy", [0, 1])
def test_both_forms_in_turn(native_lib, cuda_device, N, M, R, kind, T, legacy):
    L = N * M
    cfg = sim.make_config(N, M, R, 1, is_train=True, sim=True)
    cfg.legacy_placement = legacy
    group = sim.SimGroup(cfg)
    for seed, words in enumerate((True, False, True, True, False, False, True)):
        _through_memory(group, words)
        views, loads = _inputs(kind, N, L, T, seed, cuda_device)
        group.update_placement(0, views)
        torch.cuda.synchronize()
        group.check_status()
        for r in range(N):
            got = group.buffer(r, capi.BUF_LOADS_PER_RANK).cpu().numpy().reshape(N, L)
            assert np.array_equal(got, loads), (seed, r)
            _assert_plan(group, 0, O.legacy_solve_placement(loads.sum(0), N, M, R, N, 1.0) if legacy else O.solve_placement(loads, M, R, N, r), r)
    group.destroy()


@pytest.mark.parametrize("N,M,R,victim", [(2, 3, 1, 1), (3, 5, 2, 0), (8, 16, 4, 5), (8, 1, 1, 7), (8, 8, 0, 2)])
@pytest.mark.parametrize("words", [False, True])
@pytest.mark.parametrize("kind,T", [("int32", 9), ("map", 2600)])
def test_missing_row_is_named(native_lib, cuda_device, N, M, R, victim, words, kind, T):
    L = N * M
    group = sim.SimGroup(sim.make_config(N, M, R, 2, is_train=True, sim=True, wait_timeout_ms=100))
    hook = group.lib.uep_debug_withhold_rank if words else group.lib.uep_debug_withhold_row
    views, loads = _inputs(kind, N, L, T, 1, cuda_device)
    init = O.init_master_placement(N, M, R)
    for layer in range(2):
        capi.check(hook(group.handle, victim))
        assert bool(group.lib.uep_debug_plan_form(group.handle) & IN_CLUSTER) == (not words)
        group.update_placement(layer, views)
        torch.cuda.synchronize()
        for r in range(N):
            if r == victim and not words:  # it has everybody's row
                assert group.status(r) == (0, 0)
                _assert_plan(group, layer, O.solve_placement(loads, M, R, N, r), r)
            else:
                assert group.status(r) == (TIMEOUT_GATHER, victim), r
                assert np.array_equal(group.plan(r, layer)["lcnts"].cpu().numpy(), init.lcnts)  # as it was
        with pytest.raises(capi.UepError):
            group.check_status()
        capi.check(hook(group.handle, -1))
        capi.check(group.lib.uep_clear_status(group.handle))
        for _ in range(2):
            group.update_placement(layer, views)
            torch.cuda.synchronize()
            group.check_status()
            for r in range(N):
                _assert_plan(group, layer, O.solve_placement(loads, M, R, N, r), r)
    group.destroy()


@pytest.mark.parametrize("N,M,R", [(2, 3, 1), (8, 8, 2)])
@pytest.mark.parametrize("offset", [0, 4])
def test_weights_behind_tickets_and_flags(native_lib, cuda_device, N, M, R, offset):
    """weight_sync with the completion flags that ranks of several devices raise, in turn with the form that needs none. Bytes exact."""
    L, Lp, sizes = N * M, M + R, (16 * 4099, 16 * 513)
    gen = torch.Generator(device=cuda_device).manual_seed(N)
    group = sim.SimGroup(sim.make_config(N, M, R, 1, fc1_numel=sizes[0], fc2_numel=sizes[1], weight_elem_bytes=1, is_train=False, sim=True))
    pool = torch.randint(0, 256, (2, L, max(sizes) + 16), dtype=torch.uint8, device=cuda_device, generator=gen)
    shards = [[[pool[i, r * M + m, offset:offset + n] for m in range(M)] for r in range(N)] for i, n in enumerate(sizes)]
    tables = [group.pointer_tables(s) for s in shards]
    seen = 0
    for kind, words in (("many", True), ("one hot", False), ("even", True), ("one hot", True), ("many", False), ("many", True)):
        _through_memory(group, words)
        replicas = [group.buffer(r, capi.BUF_REPLICA_WEIGHT) for r in range(N)]
        for t in replicas:
            t.zero_()
        group.update_placement(0, _ids(kind, N, L, gen, cuda_device))
        group.weight_sync(0, *tables)
        torch.cuda.synchronize()
        group.check_status()
        p2l = group.plan(0, 0)["p2l"].cpu().view(N, Lp)[:, M:]
        for r in range(N):
            for s in range(R):
                e = int(p2l[r, s])
                want = torch.cat([shards[i][e // M][e % M] for i in range(2)]) if e >= 0 else torch.zeros(sum(sizes), dtype=torch.uint8, device=cuda_device)
                seen += int(e >= 0)
                assert torch.equal(replicas[r][s], want), (kind, r, s)
    assert seen > 0
    group.destroy()


@pytest.mark.parametrize("N,M,R", [(2, 3, 1), (8, 16, 4)])
@pytest.mark.parametrize("kind,T", [("int64", 9), ("map", 2600)])
def test_legacy_plan_behind_an_early_kernel(native_lib, cuda_device, late_write, N, M, R, kind, T):  # noqa: F811
    """Counts-only plans through the cluster, behind a kernel that starts its dependents early and writes the input later."""
    cfg = sim.make_config(N, M, R, 1, is_train=True, sim=True)
    cfg.legacy_placement = 1
    group = sim.SimGroup(cfg)
    for seed in range(3):
        data, shapes, _ = _group_input(kind, N, N * M, T, seed)
        late, _, loads = _group_input(kind, N, N * M, T, seed + 10)
        flat, source = torch.from_numpy(data).to(cuda_device), torch.from_numpy(late).to(cuda_device)
        views, at = [], 0
        for shape in shapes:
            views.append(flat[at:at + shape[0] * shape[1]].view(shape))
            at += shape[0] * shape[1]
        late_write(flat.view(torch.uint8), source.view(torch.uint8), seed % 2 == 1)
        group.update_placement(0, views)
        torch.cuda.synchronize()
        group.check_status()
        for r in range(N):
            _assert_plan(group, 0, O.legacy_solve_placement(loads.sum(0), N, M, R, N, 1.0), r)
    group.destroy()


def test_without_dependent_launches(native_lib, cuda_device):
    """UEP_DISABLE_PDL=1, which a process reads once: both exchanges, plan and reroute, solves and positions as ordinary launches."""
    here = os.path.dirname(os.path.abspath(__file__))
    chosen = ["test_gpu_plan_exchange.py::test_both_forms_in_turn", "test_gpu_reroute_behind_plan.py::test_sparse",
              "test_gpu_reroute_behind_plan.py::test_dense", "test_gpu_dependents.py::test_solve_behind_an_early_kernel",
              "test_gpu_dependents.py::test_positions_behind_an_early_kernel"]
    run = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider", *(os.path.join(here, c) for c in chosen)],
                         env=dict(os.environ, UEP_DISABLE_PDL="1"), capture_output=True, text=True, timeout=600)
    assert run.returncode == 0 and " passed" in run.stdout and "failed" not in run.stdout, run.stdout[-3000:] + run.stderr[-1000:]
