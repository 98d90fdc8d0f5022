"""The reroute may be on its SMs while the plan in front of it in the stream is still being made. It must use that plan all the
same, and the ids or maps as the stream leaves them: eager, behind a kernel or another stream's event in between, and replayed as
a graph. A kernel in between may itself start its dependents early. One rank's kernels, forward and backward, one behind the other and
behind such a kernel."""

import ctypes as C

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_dense_tiles import _random_plan
from ultra_ep_b200 import capi, sim

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


# Lets its dependents start at once, waits for what it depends on itself, and writes its bytes 30 us later (at most 2^16 looks at
# the clock).
LATE_WRITER = r"""
extern "C" __global__ void late_writer(unsigned char* dst, const unsigned char* src, long long bytes) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    unsigned long long begin, now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(begin));
    for (int i = 0; i < 65536; ++i) {
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
        if (now - begin > 30000) break;
    }
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < bytes; i += (long long)gridDim.x * blockDim.x) dst[i] = src[i];
}
"""


@pytest.fixture(scope="module")
def late_write():
    """late_write(dst, src, dependent): on the current stream, as an ordinary launch or as a programmatic dependent one."""
    from cuda.bindings import driver, nvrtc

    def ok(result):
        assert int(result[0]) == 0, result[0]
        return result[1] if len(result) == 2 else result[1:]

    torch.cuda.synchronize()  # the context is there
    program = ok(nvrtc.nvrtcCreateProgram(LATE_WRITER.encode(), b"late_writer.cu", 0, [], []))
    ok(nvrtc.nvrtcCompileProgram(program, 1, [b"--gpu-architecture=sm_100a"]))
    image = b" " * ok(nvrtc.nvrtcGetCUBINSize(program))
    ok(nvrtc.nvrtcGetCUBIN(program, image))
    module = ok(driver.cuModuleLoadData(image))
    kernel = ok(driver.cuModuleGetFunction(module, b"late_writer"))

    def launch(dst, src, dependent):
        assert dst.is_contiguous() and src.is_contiguous() and dst.nbytes == src.nbytes
        config = driver.CUlaunchConfig()
        config.gridDimX, config.gridDimY, config.gridDimZ = 16, 1, 1
        config.blockDimX, config.blockDimY, config.blockDimZ = 256, 1, 1
        config.hStream = driver.CUstream(torch.cuda.current_stream().cuda_stream)
        attribute = driver.CUlaunchAttribute()
        attribute.id = driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_PROGRAMMATIC_STREAM_SERIALIZATION
        attribute.value.programmaticStreamSerializationAllowed = 1
        config.attrs, config.numAttrs = ([attribute], 1) if dependent else ([], 0)
        values = (dst.data_ptr(), src.data_ptr(), dst.nbytes)
        ok(driver.cuLaunchKernelEx(config, kernel, (values, (C.c_void_p, C.c_void_p, C.c_longlong)), 0))

    yield launch
    torch.cuda.synchronize()
    ok(driver.cuModuleUnload(module))


def _flat(parts):
    """One buffer behind all ranks' tensors (one of them empty), and the ranks' views of it."""
    flat = torch.cat([x.reshape(-1) for x in parts])
    views, at = [], 0
    for x in parts:
        views.append(flat[at:at + x.numel()].view(x.shape))
        at += x.numel()
    return flat, views


def _ranks_draw(ranks, tokens, dtype, seed, device):
    parts = _draw(tokens, dtype, seed, device)[:ranks]
    if ranks > 3:
        parts[3] = parts[3][:0].contiguous()  # a rank without tokens
    return parts


# eight ranks: one launch, a count kernel in front, the walk; one rank: the same without the walk
@pytest.mark.parametrize("ranks,tokens", [(RANKS, 33), (RANKS, 4099), (RANKS, 9000), (1, 33), (1, 4099), (1, 40000)])
@pytest.mark.parametrize("dependent", [False, True])
def test_sparse_behind_an_early_kernel(native_lib, cuda_device, late_write, ranks, tokens, dependent):
    group = sim.SimGroup(sim.make_config(ranks, L // ranks, 2, 1, is_train=False, sim=True))
    for seed in range(4):
        flat, ids = _flat(_ranks_draw(ranks, tokens, torch.int32, seed, cuda_device))
        late_flat, late = _flat(_ranks_draw(ranks, tokens, torch.int32, seed + 50, cuda_device))
        group.update_placement(0, ids)
        late_write(flat, late_flat, dependent)
        got = group.reroute_sparse(0, ids)
        for r, (a, b) in enumerate(zip(got, _expect_of(group, late))):
            assert torch.equal(a, b), (seed, r)
        torch.cuda.synchronize()
        late_write(flat, late_flat.flip(0).contiguous(), dependent)  # the kept plan again
        got = group.reroute_sparse(0, ids)
        for r, (a, b) in enumerate(zip(got, _expect_of(group, [x.clone() for x in ids]))):
            assert torch.equal(a, b), (seed, r)
    group.destroy()


@pytest.mark.parametrize("ranks,tokens", [(RANKS, 65), (RANKS, 3000), (1, 65), (1, 9000)])
@pytest.mark.parametrize("between", ["late", "late dependent", "copy", "event", "nothing"])
def test_dense_maps_change_behind_the_plan(native_lib, cuda_device, late_write, ranks, tokens, between):
    group = sim.SimGroup(sim.make_config(ranks, L // ranks, 2, 1, is_train=True, sim=True))
    other = torch.cuda.Stream()
    to_map = lambda x: torch.zeros((x.shape[0], L), dtype=torch.bool, device=cuda_device).scatter_(1, x, True)
    for seed in range(4):
        flat, maps = _flat([to_map(x) for x in _ranks_draw(ranks, tokens, torch.int64, seed, cuda_device)])
        late_flat, late = _flat([to_map(x) for x in _ranks_draw(ranks, tokens, torch.int64, seed + 50, cuda_device)])
        probs = [torch.rand(m.shape, device=cuda_device) for m in maps]
        torch.cuda.synchronize()
        group.update_placement(0, maps)
        if between.startswith("late"):
            late_write(flat, late_flat, between.endswith("dependent"))
        elif between == "copy":
            flat.copy_(late_flat)
        elif between == "event":
            with torch.cuda.stream(other):
                other.wait_stream(torch.cuda.current_stream())
                torch.cuda._sleep(200_000)
                flat.copy_(late_flat)
            torch.cuda.current_stream().wait_stream(other)
        got_probs, got_maps = group.reroute_dense(0, maps, probs)
        want = maps if between == "nothing" else late
        _check_dense(group, want, probs, got_probs, got_maps, seed)
    group.destroy()


def test_dense_replayed(native_lib, cuda_device):
    group = sim.SimGroup(sim.make_config(RANKS, L // RANKS, 2, 1, is_train=True, sim=True))
    to_map = lambda x: torch.zeros((x.shape[0], L), dtype=torch.bool, device=cuda_device).scatter_(1, x, True)
    draw = lambda seed: _flat([to_map(x) for x in _ranks_draw(RANKS, 700, torch.int64, seed, cuda_device)])
    flat, maps = draw(0)
    next_flat = flat.clone()
    probs = [torch.rand(m.shape, device=cuda_device) for m in maps]

    def step():
        group.update_placement(0, maps)
        flat.copy_(next_flat)
        return group.reroute_dense(0, maps, probs)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()  # sizes the scratch
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got_probs, got_maps = step()
    for seed in range(1, 5):
        next_flat.copy_(draw(seed)[0])
        graph.replay()
        graph.replay()
        _check_dense(group, maps, probs, got_probs, got_maps, seed)
    group.destroy()


def _expect_of(group, ids):
    torch.cuda.synchronize()
    group.check_status()
    out = []
    for r, x in enumerate(ids):
        p = group.plan(r, 0)
        out.append(G.cuda_sparse_reroute(x, p["l2p"].contiguous(), p["lcnts"].contiguous(), p["rank_quota_prefix"].contiguous())
                   if x.numel() else x)
    return out


def _check_dense(group, maps, probs, got_probs, got_maps, what):
    torch.cuda.synchronize()
    group.check_status()
    for r, m in enumerate(maps):
        if m.numel() == 0:
            assert got_probs[r].numel() == 0 and got_maps[r].numel() == 0
            continue
        p = group.plan(r, 0)
        want_probs, want_map = G.cuda_dense_reroute(m, probs[r], p["l2p"].contiguous(), p["lcnts"].contiguous(),
                                                    p["rank_quota_prefix"].contiguous(), group.P)
        assert torch.equal(got_probs[r], want_probs) and torch.equal(got_maps[r], want_map), (what, r)


# in one launch, in two (n > 2^18), and in place
@pytest.mark.parametrize("n", [4096, 262145, 300001])
@pytest.mark.parametrize("in_place", [False, True])
def test_gather_behind_positions_of_many(native_lib, cuda_device, n, in_place):
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    rows = torch.randn((n, 8), generator=gen, device=cuda_device)
    phys = torch.randint(-1, 80, (n,), generator=gen, device=cuda_device, dtype=torch.int32)
    want = torch.empty_like(phys)
    keys = torch.where(phys < 0, 80, phys)
    want[torch.argsort(keys, stable=True)] = torch.arange(n, dtype=torch.int32, device=cuda_device)
    lib = capi.lib()
    pos = phys if in_place else torch.empty_like(phys)
    scratch = torch.empty(lib.uep_dispatch_scratch_elems(n, 80), dtype=torch.int32, device=cuda_device)
    out = torch.empty_like(rows)
    status = torch.zeros(2, dtype=torch.int32, device=cuda_device)
    torch.cuda.synchronize()
    capi.check(lib.uep_dispatch_positions(phys.data_ptr(), n, 80, pos.data_ptr(), None, scratch.data_ptr(), G.stream_ptr()))
    capi.check(lib.uep_gather_rows(rows.data_ptr(), pos.data_ptr(), out.data_ptr(), n, n, 32, status.data_ptr(), G.stream_ptr()))
    torch.cuda.synchronize()
    assert not status.any()
    assert torch.equal(pos, want) and torch.equal(out, rows[want.long()])


# One rank of eight, 1.2 million cells: the tiles of the backward, and a count kernel in front of both forwards. Each step's inputs are
# written by the kernel in front of its first reroute, in the memory of the step before, and one scratch serves all of them.
@pytest.mark.parametrize("dependent", [False, True])
@pytest.mark.parametrize("backward_first", [False, True])
def test_one_rank_back_to_back(native_lib, cuda_device, late_write, dependent, backward_first):
    ranks, masters, slots, tokens, steps = 8, 16, 4, 9600, 5
    experts, physical = ranks * masters, ranks * (masters + slots)
    rng = np.random.default_rng(7)
    popular = np.arange(1, experts + 1) ** -1.2
    plan = _random_plan(experts, physical, ranks, 5, rng)
    assert (plan.lcnts > 1).sum() > 10
    draws, wanted = [], []
    for step in range(steps):
        keys = np.log(popular)[rng.permutation(experts)] + rng.gumbel(size=(tokens, experts))
        ids = np.argsort(-keys, axis=1)[:, :K].astype(np.int32)
        rmap = np.zeros((tokens, experts), bool)
        np.put_along_axis(rmap, ids, True, 1)
        probs = rng.random((tokens, experts), dtype=np.float32)
        grad = rng.normal(size=(tokens, physical)).astype(np.float32)
        out_probs, out_map = O.dense_reroute_forward(rmap, probs, plan, physical)
        expanded = out_map & (rng.random((tokens, 1)) < 0.9)  # the backward's: not what the forward of this step writes
        draws.append([grad, probs, ids, rmap, expanded])
        wanted.append((O.sparse_reroute(ids, plan), out_probs, out_map, O.dense_reroute_backward(grad, rmap, expanded, plan)))
    sources = [torch.cat([torch.from_numpy(np.ascontiguousarray(x)).view(torch.uint8).reshape(-1) for x in d]).to(cuda_device) for d in draws]
    flat = torch.zeros_like(sources[0])
    views, at = [], 0
    for x in draws[0]:
        part = flat[at:at + x.nbytes]
        views.append(part.view({"f": torch.float32, "i": torch.int32, "b": torch.bool}[x.dtype.kind]).view(x.shape))
        at += x.nbytes
    grad, probs, ids, rmap, expanded = views
    p = G.plan_to_device(plan, cuda_device)
    lib, D = capi.lib(), plan.l2p.shape[1]
    scratch = torch.empty(max(lib.uep_reroute_scratch_elems(tokens, 0, experts), lib.uep_reroute_scratch_elems(tokens, K, experts)),
                          dtype=torch.int32, device=cuda_device)
    outs = [(torch.empty((tokens, K), dtype=torch.int32, device=cuda_device), torch.empty((tokens, physical), device=cuda_device),
             torch.empty((tokens, physical), dtype=torch.bool, device=cuda_device), torch.empty((tokens, experts), device=cuda_device))
            for _ in range(steps)]
    l2p, counts, prefix = p["l2p"].data_ptr(), p["lcnts"].data_ptr(), p["rank_quota_prefix"].data_ptr()

    def backward(out):
        capi.check(lib.uep_dense_reroute_backward(grad.data_ptr(), rmap.data_ptr(), expanded.data_ptr(), l2p, counts, out[3].data_ptr(), tokens,
                                                  experts, physical, D, G.stream_ptr()))

    torch.cuda.synchronize()
    for source, out in zip(sources, outs):
        late_write(flat, source, dependent)
        if backward_first:
            backward(out)
        capi.check(lib.uep_sparse_reroute_i32(ids.data_ptr(), out[0].data_ptr(), tokens, K, experts, l2p, counts, prefix, D, 1, scratch.data_ptr(),
                                              G.stream_ptr()))
        capi.check(lib.uep_dense_reroute_forward(rmap.data_ptr(), probs.data_ptr(), l2p, counts, prefix, out[2].data_ptr(), out[1].data_ptr(),
                                                 scratch.data_ptr(), tokens, experts, physical, D, 1, 1, G.stream_ptr()))
        if not backward_first:
            backward(out)
    torch.cuda.synchronize()
    for step, (out, want) in enumerate(zip(outs, wanted)):
        for a, b in zip(out, want):
            assert np.array_equal(a.cpu().numpy().view(np.uint8), np.ascontiguousarray(b).view(np.uint8)), step
