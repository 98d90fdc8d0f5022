"""Every output ends where it ends: the entry points write into buffers that lie between guards, and read inputs that lie between
values which would show in a result. The guards are wider than a tile, so an access beyond the end stays inside the
allocation; rows, entries and widths are the ones that leave a last tile partly empty."""

import ctypes as C

import numpy as np
import pytest
import torch

import gpu_util as G
from oracle import uep_oracle as O
from test_gpu_dense_tiles import _random_plan
from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu
GUARD = 1 << 20  # bytes on either side: 64 rows of 1340 floats are 335 KiB


class Guarded:
    """Tensors on the device between guards of one byte value."""

    def __init__(self, device, fill=0x5A):
        self.device, self.fill, self.made = device, fill, []

    def _place(self, nbytes):
        raw = torch.full((GUARD + nbytes + GUARD,), self.fill, dtype=torch.uint8, device=self.device)
        self.made.append((raw, nbytes))
        return raw[GUARD:GUARD + nbytes]

    def empty(self, shape, dtype):
        return self._place(int(np.prod(shape)) * torch.empty((), dtype=dtype).element_size()).view(dtype).view(shape)

    def like(self, x):
        t = torch.from_numpy(np.ascontiguousarray(x)) if isinstance(x, np.ndarray) else x
        out = self.empty(t.shape, t.dtype)
        out.copy_(t)
        return out

    def untouched(self):
        return all(bool((raw[:GUARD] == self.fill).all()) and bool((raw[GUARD + n:] == self.fill).all()) for raw, n in self.made)


BACKWARD = [  # T, L, P, D: either side of 2^20 cells (2^22 up to 64 experts), tiles of 64, 32, 16 and 8 rows, a last tile of any height
    (1, 8, 12, 4), (1030, 128, 161, 8), (513, 37, 50, 6), (32769, 128, 192, 8), (32771, 128, 160, 8), (32790, 128, 160, 8), (32799, 128, 160, 8),
    (65601, 64, 128, 8), (65599, 64, 80, 8), (16385, 256, 320, 8), (16391, 256, 320, 8), (43700, 96, 98, 3), (3131, 1340, 1400, 8), (116600, 36, 60, 8),
    (8195, 512, 544, 8), (8130, 516, 540, 8),
    (8191, 128, 160, 8), (8193, 128, 161, 8), (8251, 256, 322, 8), (2077, 512, 800, 16), (2100, 500, 4099, 8), (20001, 128, 160, 8), (10951, 96, 131, 3),
]


@pytest.mark.parametrize("T,L,P,D", BACKWARD)
def test_dense_backward_ends_at_its_last_row(native_lib, cuda_device, T, L, P, D):
    rng = np.random.default_rng(T + L)
    plan = _random_plan(L, P, D, D, rng)
    gen = torch.Generator(device=cuda_device).manual_seed(T)
    rmap = torch.rand((T, L), generator=gen, device=cuda_device) < 0.06
    grad = torch.randn((T, P), generator=gen, device=cuda_device)
    first = torch.from_numpy(plan.l2p[:, 0]).to(cuda_device).long()  # every routed cell at its expert's first instance
    emap = torch.zeros((T, P), dtype=torch.bool, device=cuda_device)
    emap[:, first] = rmap
    marked, guard = Guarded(cuda_device, fill=1), Guarded(cuda_device)  # beyond the maps' ends every cell is marked
    d_map, d_emap, d_grad, out = marked.like(rmap), marked.like(emap), marked.like(grad), guard.empty((T, L), torch.float32)
    pd = G.plan_to_device(plan, cuda_device)
    capi.check(native_lib.uep_dense_reroute_backward(d_grad.data_ptr(), d_map.data_ptr(), d_emap.data_ptr(), pd["l2p"].data_ptr(),
                                                     pd["lcnts"].data_ptr(), out.data_ptr(), T, L, P, D, G.stream_ptr()))
    assert torch.equal(out, torch.where(rmap, grad[:, first], 0.0))
    assert guard.untouched()


@pytest.mark.parametrize("T", [1, 7, 63, 64, 65, 130, 4111])
@pytest.mark.parametrize("L,P,D", [(128, 160, 8), (96, 130, 8), (37, 51, 6), (256, 320, 8), (16, 4100, 8)])
def test_dense_forward_ends_at_its_last_row(native_lib, cuda_device, T, L, P, D):
    rng = np.random.default_rng(T + L)
    plan = _random_plan(L, P, D, D, rng)
    rmap, probs = rng.random((T, L)) < 0.1, rng.random((T, L)).astype(np.float32)
    exp_probs, exp_map = O.dense_reroute_forward(rmap, probs, plan, P, True)
    marked, guard = Guarded(cuda_device, fill=1), Guarded(cuda_device)
    d_map, d_probs = marked.like(rmap), marked.like(probs)
    out_map, out_probs = guard.empty((T, P), torch.uint8), guard.empty((T, P), torch.float32)
    scratch = guard.empty((int(native_lib.uep_reroute_scratch_elems(T, 0, L)),), torch.int32)
    pd = {k: guard.like(v) for k, v in G.plan_to_device(plan, cuda_device).items()}
    capi.check(native_lib.uep_dense_reroute_forward(d_map.data_ptr(), d_probs.data_ptr(), pd["l2p"].data_ptr(), pd["lcnts"].data_ptr(),
                                                    pd["rank_quota_prefix"].data_ptr(), out_map.data_ptr(), out_probs.data_ptr(),
                                                    scratch.data_ptr(), T, L, P, D, 1, 1, G.stream_ptr()))
    assert np.array_equal(out_map.cpu().numpy(), exp_map.astype(np.uint8))
    assert np.array_equal(out_probs.cpu().numpy().view(np.uint32), exp_probs.view(np.uint32))
    assert guard.untouched()


@pytest.mark.parametrize("n", [1, 33, 513, 4099, 16387, 65539, 262149])
@pytest.mark.parametrize("dtype,in_place", [(torch.int32, False), (torch.int64, False), (torch.int32, True), (torch.int64, True)])
def test_sparse_reroute_and_positions_end_at_their_last_entry(native_lib, cuda_device, n, dtype, in_place):
    rng = np.random.default_rng(n)
    L, P, D = 72, 96, 8
    plan = _random_plan(L, P, D, D, rng)
    ids = rng.integers(0, L, size=(n, 1)).astype(np.int64 if dtype == torch.int64 else np.int32)
    exp = O.sparse_reroute(ids, plan, True)
    marked, guard = Guarded(cuda_device, fill=0), Guarded(cuda_device)  # beyond the ids' end: expert 0
    d_ids = (guard if in_place else marked).like(ids)
    out = d_ids if in_place else guard.empty((n, 1), dtype)
    scratch = guard.empty((int(native_lib.uep_reroute_scratch_elems(n, 1, L)),), torch.int32)
    pd = {k: guard.like(v) for k, v in G.plan_to_device(plan, cuda_device).items()}
    fn = native_lib.uep_sparse_reroute_i64 if dtype == torch.int64 else native_lib.uep_sparse_reroute_i32
    capi.check(fn(d_ids.data_ptr(), out.data_ptr(), n, 1, L, pd["l2p"].data_ptr(), pd["lcnts"].data_ptr(), pd["rank_quota_prefix"].data_ptr(),
                  D, 1, scratch.data_ptr(), G.stream_ptr()))
    assert np.array_equal(out.cpu().numpy(), exp)
    assert guard.untouched()
    if dtype == torch.int32 and not in_place:
        exp_pos, exp_off = O.dispatch_positions(exp.reshape(-1), P)
        pos, offsets = guard.empty((n,), torch.int32), guard.empty((P + 1,), torch.int32)
        scratch = guard.empty((int(native_lib.uep_dispatch_scratch_elems(n, P)),), torch.int32)
        capi.check(native_lib.uep_dispatch_positions(out.data_ptr(), n, P, pos.data_ptr(), offsets.data_ptr(), scratch.data_ptr(), G.stream_ptr()))
        assert np.array_equal(pos.cpu().numpy(), exp_pos) and np.array_equal(offsets.cpu().numpy(), exp_off)
        assert guard.untouched()


@pytest.mark.parametrize("n,row_bytes", [(1, 16), (31, 48), (2369, 2064), (9473, 4096), (75775, 16), (700, 16400), (33, 7)])
def test_gather_ends_at_its_last_row(native_lib, cuda_device, n, row_bytes):
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    src = max(1, min(n, 5000))
    guard = Guarded(cuda_device)
    rows = guard.like(torch.randint(0, 256, (src, row_bytes), dtype=torch.uint8, device=cuda_device, generator=gen))
    pos = guard.like(torch.randint(0, src, (n,), dtype=torch.int32, device=cuda_device, generator=gen))
    out = guard.empty((n, row_bytes), torch.uint8)
    status = torch.zeros(2, dtype=torch.int32, device=cuda_device)
    capi.check(native_lib.uep_gather_rows(rows.data_ptr(), pos.data_ptr(), out.data_ptr(), n, src, row_bytes, status.data_ptr(), G.stream_ptr()))
    assert torch.equal(out, rows[pos.long()]) and status.tolist() == [0, 0]
    assert guard.untouched()


@pytest.mark.parametrize("N,M,R", [(8, 9, 3), (64, 4, 2), (72, 7, 4), (5, 3, 1), (1, 6, 2)])
def test_solver_ends_at_its_last_row(native_lib, cuda_device, N, M, R):
    rng = np.random.default_rng(N)
    L, P = N * M, N * (M + R)
    lpr = rng.zipf(1.5, size=(N, L)).clip(0, 5000).astype(np.int32)
    exp = O.solve_placement(lpr, M, R, N, 0, O.SolverParams())
    guard = Guarded(cuda_device)
    loads, total = guard.like(lpr), guard.empty((L,), torch.int32)
    shapes = dict(p2l=(P,), l2p=(L, N), lcnts=(L,), quota=(L, N), quota_prefix=(L, N), rank_quota_prefix=(L, N))
    plan = {k: guard.empty(shapes[k], torch.int32) for k in G.PLAN_FIELDS}
    status = torch.zeros(2, dtype=torch.int32, device=cuda_device)
    prm = capi.SolverParams.defaults()
    capi.check(native_lib.uep_solve_placement(loads.data_ptr(), total.data_ptr(), *(plan[k].data_ptr() for k in G.PLAN_FIELDS), N, N, M, R, N,
                                              C.byref(prm), 0, status.data_ptr(), G.stream_ptr()))
    for k in G.PLAN_FIELDS:
        assert np.array_equal(plan[k].cpu().numpy(), getattr(exp, k)), k
    assert np.array_equal(total.cpu().numpy(), lpr.sum(0)) and status.tolist() == [0, 0]
    assert guard.untouched()


@pytest.mark.parametrize("L,rows", [(128, [6243, 5852, 5463, 5072, 4683, 4292, 3902, 3511]), (64, [9, 0, 1, 65, 63, 128, 7, 300])])
def test_hosted_ranks_end_at_their_last_row(native_lib, cuda_device, L, rows):
    """The dense pair for eight ranks in one launch: the grid is the longest rank's."""
    R = 8
    P = L + 8 * R
    group = sim.SimGroup(sim.make_config(8, L // 8, R, 1, is_train=True, sim=True))
    gen = torch.Generator(device=cuda_device).manual_seed(L)
    marked, guard = Guarded(cuda_device, fill=1), Guarded(cuda_device)
    maps = [marked.like(torch.rand((T, L), generator=gen, device=cuda_device) < 0.06) for T in rows]
    probs = [marked.like(torch.rand((T, L), generator=gen, device=cuda_device)) for T in rows]
    group.update_placement(0, maps)
    to = ([guard.empty((T, P), torch.float32) for T in rows], [guard.empty((T, P), torch.bool) for T in rows])
    group.reroute_dense(0, maps, probs, out=to)
    grads = [marked.like(torch.randn((T, P), generator=gen, device=cuda_device)) for T in rows]
    outs = [guard.empty((T, L), torch.float32) for T in rows]
    ptrs = lambda ts: (C.c_void_p * 8)(*[t.data_ptr() for t in ts])  # noqa: E731
    capi.check(native_lib.uep_reroute_dense_backward(group.handle, 0, ptrs(grads), ptrs(maps), ptrs(to[1]), ptrs(outs), (C.c_int * 8)(*rows), P,
                                                     G.stream_ptr()))
    p2l = group.plan(0, 0)["p2l"].long()
    used = p2l >= 0
    for T, m, p, ep, em, g, o in zip(rows, maps, probs, *to, grads, outs):
        back = torch.zeros((T, L), device=cuda_device).index_add_(1, p2l[used], torch.where(em, g, 0.0)[:, used])
        count = torch.zeros((T, L), device=cuda_device).index_add_(1, p2l[used], em.float()[:, used])
        assert torch.equal(count, m.float()) and not em[:, ~used].any()
        assert torch.equal(ep[:, used], torch.where(em[:, used], p[:, p2l[used]], 0.0)) and not ep[:, ~used].any()
        assert torch.equal(o, back)
    assert guard.untouched()
