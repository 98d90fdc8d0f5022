"""Sparse reroute of eight hosted ranks beside a weight_sync that is not long: up to 32768 entries of the longest rank go in one cluster of
eight entries a thread. At both ends of that and one token beyond, with ranks that have none, one and most of it, ids of both
widths, in place and not. Whole numbers against the CPU oracle."""

import numpy as np
import pytest
import torch

from oracle import uep_oracle as O
from test_gpu_hosted_reroute import _case
from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu
N, R = 8, 2


@pytest.mark.parametrize("longest", [2049, 3333, 4095, 4096, 4097])
@pytest.mark.parametrize("L", [64, 200])
def test_beside_a_weight_sync(native_lib, cuda_device, longest, L):
    ids, plans, dev = _case([longest, 1, 0, 2048, 513, longest - 1, 64, 2050], L, longest, cuda_device)
    group = sim.SimGroup(sim.make_config(N, L // N, R, 1, fc1_numel=4096, fc2_numel=2048, is_train=True, sim=True))
    tables = [group.pointer_tables([[torch.zeros(n, dtype=torch.bfloat16, device=cuda_device)] * (L // N)] * N) for n in (4096, 2048)]
    want = [O.sparse_reroute(x, p, True) if len(x) else x for x, p in zip(ids, plans)]
    for dtype in (torch.int32, torch.int64):
        for in_place in (False, True):
            group.update_placement(0, dev)
            done = group.weight_sync(0, *tables, async_finish=True)
            src = [x.to(dtype, copy=True) for x in dev]
            got = group.reroute_sparse(0, src, src if in_place else None)
            group.wait_event(done)
            for g, w in zip(got, want):
                assert g.dtype == dtype and np.array_equal(g.cpu().numpy(), w)
    group.check_status()
    group.destroy()
