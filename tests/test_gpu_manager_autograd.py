"""Manager.reroute as autograd sees it, on a group of one rank: the gradients that reach the node, and the forms of
differentiation that it refuses."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD
import torch.distributed as dist

from ultra_ep_b200 import Manager

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


def test_forward_mode_is_refused(manager, inputs):
    layer, probs, rmap = inputs
    with fwAD.dual_level():
        dual = fwAD.make_dual(probs, torch.ones_like(probs))
        with pytest.raises(NotImplementedError):
            manager.reroute(layer, dual, rmap)
