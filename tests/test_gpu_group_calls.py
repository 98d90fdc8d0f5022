"""The calls of a group hosted on one device as Python sees them: what they accept in the place of a list, and that other
Python threads run while one of them waits for the device."""

import ctypes as C
import threading
import time

import pytest
import torch

from ultra_ep_b200 import capi, sim

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


def test_any_iterable_of_tensors_is_taken(group, cuda_device):
    tokens = [33, 70]
    ids = _ids(tokens, cuda_device)
    maps = [torch.zeros((t, L), dtype=torch.bool, device=cuda_device).scatter_(1, x.long(), True) for t, x in zip(tokens, ids)]
    probs = [torch.rand(m.shape, device=cuda_device) * m for m in maps]
    group.update_placement(0, maps)
    exp_probs, exp_maps = group.reroute_dense(0, maps, probs)
    exp_grads = group.reroute_dense_backward(0, exp_probs, maps, exp_maps)
    exp_ids = group.reroute_sparse(0, ids)
    as_dict = lambda ts: dict(enumerate(ts)).values()  # noqa: E731
    host = lambda ts: [t.cpu().pin_memory() for t in ts]  # noqa: E731
    spare = [torch.zeros((4, L), dtype=torch.bool, device=cuda_device)] * 9
    for got_probs, got_maps in (group.reroute_dense(0, tuple(maps), (p for p in probs)), group.reroute_dense(0, as_dict(maps), probs),
                                group.reroute_dense(0, maps + spare, probs + [s.float() for s in spare]),
                                group.reroute_dense(0, host(maps), host(probs))):
        assert all(torch.equal(a, b) for a, b in zip(got_probs, exp_probs)) and all(torch.equal(a, b) for a, b in zip(got_maps, exp_maps))
        assert got_probs[0].is_cuda and got_maps[0].is_cuda
    grads = group.reroute_dense_backward(0, as_dict(exp_probs), (m for m in maps), tuple(exp_maps))
    assert all(torch.equal(a, b) for a, b in zip(grads, exp_grads))
    assert all(torch.equal(a, b) for a, b in zip(group.reroute_sparse(0, tuple(ids), tuple(torch.empty_like(x) for x in ids)), exp_ids))
    same = torch.stack([ids[0], ids[0]])
    assert torch.equal(group.reroute_sparse(0, same)[0], exp_ids[0])
    with pytest.raises(TypeError):
        group.reroute_sparse(0, [ids[0], 3])
    for call in (lambda: group.reroute_sparse(0, ids[:1]), lambda: group.update_placement(0, ids[:1]), lambda: group.reroute_dense(0, maps, probs[:1])):
        with pytest.raises(ValueError):
            call()


def test_events_are_waited_for_by_address_too(group, cuda_device):
    group.update_placement(0, _ids([8, 8], cuda_device))
    tables = group.pointer_tables([[torch.zeros(1, device=cuda_device)] * (L // 2)] * 2)
    group.wait_event(group.weight_sync(0, tables, tables, async_finish=True))
    group.wait_event(group.weight_sync(0, iter(tables), tables, async_finish=True).value)
    with pytest.raises(RuntimeError):
        group.wait_event(None)


@pytest.mark.parametrize("managers", [0, 1])
def test_events_in_flight_and_used_again(native_lib, cuda_device, managers):
    """More events than the library keeps, given back while another stream still waits for their record, and recorded anew."""
    held = [sim.SimGroup(sim.make_config(2, 2, 0, 1, is_train=False, sim=True)) for _ in range(managers)]
    first, second, other = (torch.cuda.Stream() for _ in range(3))
    n = 40
    marks, copies = torch.zeros(n, dtype=torch.int64, device=cuda_device), torch.zeros(n, dtype=torch.int64, device=cuda_device)
    torch.cuda.synchronize()
    for _ in range(2):
        marks.zero_()
        torch.cuda.synchronize()
        events = []
        for i in range(n):
            with torch.cuda.stream(first):
                torch.cuda._sleep(200_000)
                marks[i] = i + 1
            events.append(C.c_void_p())
            capi.check(native_lib.uep_event_record(first.cuda_stream, C.byref(events[i])))
        for i, ev in enumerate(events):
            capi.check(native_lib.uep_event_stream_wait(ev, second.cuda_stream))
            native_lib.uep_event_destroy(ev)
            again = C.c_void_p()
            capi.check(native_lib.uep_event_record(other.cuda_stream, C.byref(again)))
            capi.check(native_lib.uep_event_synchronize(again))
            native_lib.uep_event_destroy(again)
            with torch.cuda.stream(second):
                copies[i] = marks[i]
        torch.cuda.synchronize()
        assert copies.tolist() == list(range(1, n + 1))
    for g in held:
        g.destroy()
