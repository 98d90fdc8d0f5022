"""Manager.reroute as autograd sees it, on a group of one rank: the gradients that reach the node, and the forms of
differentiation that it refuses; and a plan from ids that are not contiguous."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD
import torch.distributed as dist

from ultra_ep_b200 import EventHandle, Manager
from ultra_ep_b200.native import load

pytestmark = pytest.mark.gpu
T, L, R = 70, 16, 2


@pytest.fixture
def manager(native_lib, cuda_device):
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    mgr = Manager(dist.group.WORLD, 1, L, R, 2 * 64, 64, is_train=True)
    weights = [[torch.zeros(n, dtype=torch.bfloat16, device=cuda_device) for _ in range(L)] for n in (128, 64)]
    grads = [[torch.zeros(n, device=cuda_device) for _ in range(L)] for n in (128, 64)]
    mgr.construct_local_master_ptr_pool(1, *weights, *grads)
    mgr.keep = (weights, grads)
    return mgr


@pytest.fixture
def inputs(manager, cuda_device):
    gen = torch.Generator(device=cuda_device).manual_seed(4)
    rmap = torch.rand((T, L), generator=gen, device=cuda_device) < 0.3
    probs = torch.rand((T, L), generator=gen, device=cuda_device) * rmap
    layer = manager.allocate_microbatch_slot(1)
    manager.update_placement(layer, rmap)
    return layer, probs.requires_grad_(True), rmap


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_plan_from_ids_that_are_not_contiguous(manager, cuda_device, dtype):
    """The plan reads a copy of them on the communication stream; memory that is asked for meanwhile must not be that copy."""
    gen = torch.Generator(device=cuda_device).manual_seed(9)
    ids = torch.randint(0, L, (6, 700), generator=gen, device=cuda_device, dtype=dtype).t()
    want = torch.bincount(ids.reshape(-1), minlength=L).int()
    layer = manager.allocate_microbatch_slot(1)
    manager.update_placement_sparse(layer, ids)
    torch.cuda.synchronize()
    with torch.cuda.stream(manager.get_comm_stream()):
        torch.cuda._sleep(40_000_000)  # the plan waits for work in front of it
    manager.update_placement_sparse(layer, ids)
    others = [torch.zeros((700, 6), device=cuda_device, dtype=dtype) for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(manager.runtime.get_global_logical_expert_loads_tensor(), want)
    assert all(not x.any() for x in others)


def test_forward_mode_is_refused(manager, inputs):
    layer, probs, rmap = inputs
    with fwAD.dual_level():
        dual = fwAD.make_dual(probs, torch.ones_like(probs))
        with pytest.raises(NotImplementedError):
            manager.reroute(layer, dual, rmap)


def test_functional_transforms_are_refused(manager, inputs):
    layer, probs, rmap = inputs
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda p: manager.reroute(layer, p, rmap)[0].sum())(probs)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda p: manager.reroute(layer, p, rmap)[0])(torch.stack([probs, probs]))


def test_gradients_that_reach_the_node(manager, inputs, cuda_device):
    """Contiguous, expanded (stride 0), through a slice, twice through one graph, and none at all."""
    layer, probs, rmap = inputs
    out, emap = manager.reroute(layer, probs, rmap)
    assert torch.equal(out, manager.reroute(layer, probs.detach(), rmap)[0]) and not emap.requires_grad
    upstream = torch.randn(out.shape, device=cuda_device)
    p2l = manager.physical_to_logical_map[layer].long()
    want = torch.zeros((T, L), device=cuda_device).index_add_(1, p2l[p2l >= 0], torch.where(emap, upstream, 0.0)[:, p2l >= 0])
    (first,) = torch.autograd.grad(out, probs, upstream, retain_graph=True)
    (second,) = torch.autograd.grad(out, probs, upstream.t().contiguous().t(), retain_graph=True)
    assert torch.equal(first, want) and torch.equal(second, want)
    (ones,) = torch.autograd.grad(out.sum(), probs, retain_graph=True)
    assert torch.equal(ones, rmap.float())
    (part,) = torch.autograd.grad(out[:, :3].sum(), probs)
    assert torch.equal(part[:, 3:], torch.zeros_like(part[:, 3:])) and torch.equal(part[:, :3], rmap[:, :3].float())
    with torch.no_grad():
        assert not manager.reroute(layer, probs, rmap)[0].requires_grad
    other = torch.zeros(3, device=cuda_device, requires_grad=True)
    unused, _ = manager.reroute(layer, probs, rmap)
    assert torch.autograd.grad(other.sum() + 0 * emap.float().sum(), [probs], allow_unused=True) == (None,)
    del unused


def test_one_rank_orders_behind_a_previous_event(manager, inputs, cuda_device):
    """Nothing is launched for a group of one rank, and the order it promises still holds."""
    layer, _, _ = inputs
    side = torch.cuda.Stream()
    mark = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    torch.cuda.synchronize()
    for call in (manager.weight_sync, manager.grad_reduce):
        for asynchronous in (True, False):
            mark.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                torch.cuda._sleep(20_000_000)
                mark += 1
                before = EventHandle(load().EventHandle())
            done = call(layer, previous_event=before, async_finish=asynchronous)
            if asynchronous:
                done.current_stream_wait()
            seen = mark.clone()
            torch.cuda.synchronize()
            assert seen.item() == 1
