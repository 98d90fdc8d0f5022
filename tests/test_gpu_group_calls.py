"""The calls of a group hosted on one device as Python sees them: what they accept in the place of a list, and that other
Python threads run while one of them waits for the device."""

import threading
import time

import pytest
import torch

from ultra_ep_b200 import sim

pytestmark = pytest.mark.gpu
L = 16


@pytest.fixture
def group(native_lib, cuda_device):
    return sim.SimGroup(sim.make_config(2, L // 2, 2, 1, is_train=True, sim=True))


def _ids(tokens, device, seed=1):
    gen = torch.Generator(device=device).manual_seed(seed)
    return [torch.rand((t, L), generator=gen, device=device).topk(4, dim=1).indices.int() for t in tokens]


def test_other_threads_run_while_a_call_waits(group, cuda_device):
    small, large = _ids([8, 8], cuda_device), _ids([60000, 60000], cuda_device)
    group.update_placement(0, small)
    group.reroute_sparse(0, small)
    out = [torch.empty_like(x) for x in large]
    torch.cuda.synchronize()
    beats, stop = [], threading.Event()

    def beat():
        while not stop.is_set():
            beats.append(time.perf_counter())
            time.sleep(0.002)

    thread = threading.Thread(target=beat)
    thread.start()
    try:
        torch.cuda._sleep(700_000_000)  # about a third of a second of device work in front
        begin = time.perf_counter()
        group.reroute_sparse(0, large, out)  # its scratch buffer grows, which waits for the device
        end = time.perf_counter()
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert end - begin > 0.1, "the call did not wait: this test shows nothing"
    inside = [b for b in beats if begin < b < end]
    assert len(inside) > 0.1 * (end - begin) / 0.002
