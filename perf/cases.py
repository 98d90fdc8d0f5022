"""The work a user of this library has it do, as cases that can be timed and compared.

Two ways lead into the library. `Manager` is what a framework's MoE layer holds, one rank per process; with one GPU
its group has one rank, so its cases show what a call costs on the host and what one rank's kernels cost, not the
exchange. `SimGroup` hosts all ranks of an expert-parallel group on one device and runs the same kernels on real
replication plans, replica slots and reductions. The stateless entry points of the C ABI serve callers that keep
their own plan storage: the solver at group sizes that no single GPU can host, the reroute of one rank of a
group, and the token-gradient gather.

Sizes follow the library's own configurations (`ultra_ep_b200/workloads.py`): 64 to 256 experts, top-8, 4096 to 16384
tokens per rank in training and prefill, a handful to a few hundred in decode, layers of hidden size 2048 to
7168 with bf16 or fp8 experts. Routing is drawn without replacement from a Zipf popularity over a permuted expert
order, as the configurations draw it, on the device and from the seed alone.
"""

import ctypes as C
import math

import torch
import torch.distributed as dist

from ultra_ep_b200 import Manager, capi, sim

DEV = "cuda"


def listed():
    return [
        # Serving, decode: one rank's step through the Manager on int64 top-k ids, in place. A few kernels on a few
        # hundred ids: launches and host work are all there is.
        dict(name="manager_decode", kind="manager_sparse", tokens=64, experts=128, redundant=4, topk=8, zipf=1.3),
        # Training through the Manager: plan from the bool map, weight_sync beside the differentiable dense reroute,
        # its backward and the gradient reduce of one layer and microbatch.
        dict(name="manager_train", kind="manager_dense", tokens=4096, experts=64, redundant=2, topk=8, zipf=1.2),
        # The smallest group step: decode on eight ranks, uneven token counts, no weights to move.
        dict(name="group_decode", kind="forward", ids="int32", tokens=33, ragged=True, experts=64, redundant=2, topk=8,
             zipf=1.2, hidden=0, ffn=0, weights="none", train=False, hot=False),
        # Plan and reroute alone, the 64-expert configuration.
        dict(name="group_plan_reroute", kind="forward", ids="int32", tokens=4096, ragged=False, experts=64, redundant=2,
             topk=8, zipf=1.2, hidden=0, ffn=0, weights="none", train=False, hot=False),
        # Training forward of the 30B-shaped layer: bool maps and probabilities, bf16 experts.
        dict(name="group_forward_dense_bf16", kind="forward", ids="map", tokens=8192, ragged=False, experts=128, redundant=4,
             topk=8, zipf=1.2, hidden=2048, ffn=768, weights="bf16", train=True, hot=False),
        # The benchmark's own step: the 235B-shaped layer with fp8 experts and their scales.
        dict(name="group_forward_fp8", kind="forward", ids="int32", tokens=8192, ragged=False, experts=128, redundant=4,
             topk=8, zipf=1.3, hidden=4096, ffn=1536, weights="fp8", train=False, hot=False),
        # Extreme skew, the largest layer: 256 experts, one expert in every token's top-k, uneven ranks, int64 ids.
        dict(name="group_forward_skewed_fp8", kind="forward", ids="int64", tokens=16384, ragged=True, experts=256,
             redundant=8, topk=8, zipf=1.5, hidden=7168, ffn=2048, weights="fp8", train=False, hot=True),
        # Backward of the 30B-shaped layer: gradients of the expanded probabilities, then the replica Wgrad reduce.
        dict(name="group_backward_bf16", kind="backward", tokens=8192, ragged=False, experts=128, redundant=4, topk=8,
             zipf=1.2, hidden=2048, ffn=768),
        # Backward of the 235B-shaped layer: the largest reduce.
        dict(name="group_backward_fp8", kind="backward", tokens=8192, ragged=False, experts=128, redundant=4, topk=8,
             zipf=1.3, hidden=4096, ffn=1536),
        # Token gradients of one rank back from physical-expert order to (token, k) order.
        dict(name="token_gradients", kind="gather", tokens=8192, topk=8, physical=160, hidden=4096, zipf=1.3),
        # Plan of a 64-rank group from its gathered loads: the solver alone.
        dict(name="solve_64_ranks", kind="solve", ranks=64, masters=4, redundant=2, topk=8, tokens=8192, zipf=1.2),
        # One rank of an eight-rank group on its own GPU: sparse ids, dense map and the dense backward.
        dict(name="one_rank_reroute", kind="reroute", tokens=8191, experts=256, redundant=8, topk=8, zipf=1.5, ranks=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["manager_sparse", "manager_dense", "forward", "forward", "forward", "backward", "backward",
                       "gather", "solve", "reroute"])
    zipf = round(rng.uniform(1.0, 1.6), 2)
    topk = rng.choice([4, 6, 8, 8])
    if kind == "manager_sparse":
        return dict(kind=kind, tokens=_log_int(rng, 1, 2048), experts=rng.choice([64, 96, 128, 256]),
                    redundant=rng.choice([0, 2, 4]), topk=topk, zipf=zipf)
    if kind == "manager_dense":
        return dict(kind=kind, tokens=_log_int(rng, 512, 8192), experts=rng.choice([64, 96, 128, 256]),
                    redundant=rng.choice([2, 4]), topk=topk, zipf=zipf)
    if kind == "forward":
        weights = rng.choice(["none", "bf16", "fp8"])
        ids = rng.choice(["int32", "int64", "map"])
        hidden = 0 if weights == "none" else rng.choice([1024, 2048, 2880, 4096])
        return dict(kind=kind, ids=ids, tokens=_log_int(rng, 8, 8192), ragged=rng.random() < 0.5,
                    experts=rng.choice([64, 128, 256]), redundant=rng.choice([2, 4, 8]), topk=topk, zipf=zipf,
                    hidden=hidden, ffn=0 if weights == "none" else rng.choice([512, 768, 1536]), weights=weights,
                    train=ids == "map", hot=rng.random() < 0.25)
    if kind == "backward":
        return dict(kind=kind, tokens=_log_int(rng, 512, 8192), ragged=rng.random() < 0.5, experts=rng.choice([64, 128]),
                    redundant=rng.choice([2, 4, 8]), topk=topk, zipf=zipf, hidden=rng.choice([1024, 2048, 2880, 4096]),
                    ffn=rng.choice([512, 768, 1536]))
    if kind == "gather":
        return dict(kind=kind, tokens=_log_int(rng, 64, 8192), topk=topk, physical=rng.choice([80, 160, 320]),
                    hidden=rng.choice([1024, 2048, 2880, 4096]), zipf=zipf)
    if kind == "solve":
        ranks = rng.choice([16, 32, 48, 64, 72])
        return dict(kind=kind, ranks=ranks, masters=rng.choice([2, 4, 7]), redundant=rng.choice([1, 2, 4]), topk=topk,
                    tokens=_log_int(rng, 512, 16384), zipf=zipf)
    return dict(kind=kind, tokens=_log_int(rng, 64, 16384), experts=rng.choice([64, 128, 256]),
                redundant=rng.choice([2, 4, 8]), topk=topk, zipf=zipf, ranks=8)


# -- inputs --------------------------------------------------------------------------------
class _Inputs:
    """Seeded values on the device; a case's popularity order comes from the seed too."""

    def __init__(self, seed, experts, zipf):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)
        rank = torch.randperm(experts, generator=self.gen, device=DEV)
        self.logits = -zipf * torch.log(rank.float() + 1.0)
        self.hottest = int(torch.argmin(rank))

    def topk_ids(self, tokens, topk, hot=False):
        """int32 [tokens, topk]: distinct experts per token, drawn without replacement (Gumbel top-k)."""
        u = torch.rand((tokens, self.logits.numel()), generator=self.gen, device=DEV).clamp_(1e-30, 1.0 - 1e-7)
        keys = self.logits - torch.log(-torch.log(u))
        if hot:
            keys[:, self.hottest] = math.inf
        return torch.topk(keys, topk, dim=1).indices.int()

    def normal(self, shape, std, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=self.gen)

    def raw_bytes(self, shape):
        n = math.prod(shape)
        words = torch.empty((n + 7) // 8, dtype=torch.int64, device=DEV)
        return words.random_(generator=self.gen).view(torch.uint8)[:n].view(shape)

    def probs(self, rmap):
        return torch.rand(rmap.shape, generator=self.gen, device=DEV) * rmap


def _to_map(ids, experts):
    m = torch.zeros((ids.shape[0], experts), dtype=torch.bool, device=DEV)
    return m.scatter_(1, ids.long(), True)


def _tokens_per_rank(case, ranks=8):
    """Rank r's token count: the case's own, or (ragged) down to half of it with an odd step, as uneven batches are."""
    t = case["tokens"]
    return [max(1, t - (r * t) // (2 * ranks) - r % 2) for r in range(ranks)] if case["ragged"] else [t] * ranks


def _layer_sizes(case):
    fc1, fc2 = 2 * case["hidden"] * case["ffn"], case["hidden"] * case["ffn"]
    fp8 = case["weights"] == "fp8"
    return fc1, fc2, (1 if fp8 else 2), (fc1 // 128 if fp8 else 0), (fc2 // 128 if fp8 else 0)


# -- what a program keeps --------------------------------------------------------------------
def _owned(tensors, owner):
    """Views of memory that the library owns are valid until their manager is destroyed: each view keeps it."""
    for t in tensors:
        t.owner = owner
    return tensors


_PLAN = ("p2l", "l2p", "lcnts", "quota", "quota_prefix", "rank_quota_prefix")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _one_rank_group():
    """The process group of a one-GPU job."""
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    return dist.group.WORLD


def _manager(case, inputs, train):
    # With one rank no expert has a replica, so the experts' size is of no consequence: small ones.
    masters, fc1, fc2 = case["experts"], 2 * 256 * 96, 256 * 96
    mgr = Manager(_one_rank_group(), 1, masters, case["redundant"], fc1, fc2, is_train=train)
    weights = [[inputs.normal((n,), 0.02, torch.bfloat16) for _ in range(masters)] for n in (fc1, fc2)]
    grads = [[inputs.normal((n,), 1e-4) for _ in range(masters)] for n in (fc1, fc2)] if train else [None, None]
    mgr.construct_local_master_ptr_pool(1, weights[0], weights[1], grads[0], grads[1])
    plan = [mgr.physical_to_logical_map[1], mgr.logical_to_physical_map[1], mgr.logical_replica_counts[1],
            mgr.logical_instance_quota[1], mgr.logical_instance_quota_prefix[1], mgr.rank_quota_prefix[1]]
    return dict(mgr=mgr, keep=(weights, grads), plan=_owned(plan, mgr))


def _group(case, train, fc1=0, fc2=0, elem=2, s1=0, s2=0):
    cfg = sim.make_config(8, case["experts"] // 8, case["redundant"], 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=elem,
                          fc1_scale_numel=s1, fc2_scale_numel=s2, is_train=train, sim=True)
    return sim.SimGroup(cfg)


def _plan_buffers(ranks, masters, redundant):
    L, P = ranks * masters, ranks * (masters + redundant)
    shapes = dict(p2l=(P,), l2p=(L, ranks), lcnts=(L,), quota=(L, ranks), quota_prefix=(L, ranks), rank_quota_prefix=(L, ranks))
    return {k: torch.empty(shapes[k], dtype=torch.int32, device=DEV) for k in _PLAN}


def _solve(lib, loads, total, plan, ranks, masters, redundant, params, my_rank, status):
    capi.check(lib.uep_solve_placement(loads.data_ptr(), total.data_ptr(), *(plan[k].data_ptr() for k in _PLAN), ranks, ranks,
                                       masters, redundant, ranks, C.byref(params), my_rank, status.data_ptr(), _stream()),
               "uep_solve_placement")


def _count(ids, experts):
    return torch.bincount(ids.reshape(-1).long(), minlength=experts).int()


# -- prepare ---------------------------------------------------------------------------------
def _prepare_manager_sparse(case, seed):
    inputs = _Inputs(seed, case["experts"], case["zipf"])
    s = _manager(case, inputs, train=False)
    s["ids"] = inputs.topk_ids(case["tokens"], case["topk"]).long()
    return s


def _prepare_manager_dense(case, seed):
    inputs = _Inputs(seed, case["experts"], case["zipf"])
    s = _manager(case, inputs, train=True)
    s["rmap"] = _to_map(inputs.topk_ids(case["tokens"], case["topk"]), case["experts"])
    s["probs"] = inputs.probs(s["rmap"]).requires_grad_(True)
    s["upstream"] = inputs.normal((case["tokens"], case["experts"] + case["redundant"]), 1e-3)
    return s


def _prepare_forward(case, seed):
    inputs = _Inputs(seed, case["experts"], case["zipf"])
    fc1, fc2, elem, s1, s2 = _layer_sizes(case)
    g = _group(case, case["train"], fc1, fc2, elem, s1, s2)
    masters = case["experts"] // 8
    s = dict(group=g, ids=[inputs.topk_ids(t, case["topk"], case["hot"]) for t in _tokens_per_rank(case)])
    if case["ids"] == "int64":
        s["ids"] = [x.long() for x in s["ids"]]
    if case["ids"] == "map":
        s["maps"] = [_to_map(x, case["experts"]) for x in s.pop("ids")]
        s["probs"] = [inputs.probs(m) for m in s["maps"]]
    else:
        s["phys"] = [torch.empty_like(x) for x in s["ids"]]
    s["out"] = [v for r in range(8) for v in ([g.plan(r, 0)["rank_quota_prefix"]] if r else g.plan(0, 0).values())]
    if case["weights"] != "none":
        s["tables"], s["keep"] = [], []
        for nbytes in (fc1 * elem, fc2 * elem, s1, s2):
            if nbytes == 0:
                s["tables"].append(None)
                continue
            if elem == 2:
                per_rank = [inputs.normal((masters, nbytes // 2), 0.02, torch.bfloat16) for _ in range(8)]
            else:
                per_rank = [inputs.raw_bytes((masters, nbytes)) for _ in range(8)]
            s["keep"].append(per_rank)
            s["tables"].append(g.pointer_tables([list(t) for t in per_rank]))
        s["out"] += [g.buffer(r, capi.BUF_REPLICA_WEIGHT) for r in range(8)]
        if s1:
            s["out"] += [g.buffer(r, capi.BUF_REPLICA_SCALE) for r in range(8)]
    _owned(s["out"], g)
    return s


def _prepare_backward(case, seed):
    inputs = _Inputs(seed, case["experts"], case["zipf"])
    fc1, fc2 = 2 * case["hidden"] * case["ffn"], case["hidden"] * case["ffn"]
    g = _group(case, True, fc1, fc2)
    masters = case["experts"] // 8
    maps = [_to_map(inputs.topk_ids(t, case["topk"]), case["experts"]) for t in _tokens_per_rank(case)]
    g.update_placement(0, maps)  # the forward made the plan and the expanded maps
    _, expanded = g.reroute_dense(0, maps, [inputs.probs(m) for m in maps])
    grads = [[inputs.normal((masters, n), 1e-4) for _ in range(8)] for n in (fc1, fc2)]
    replicas = _owned([g.buffer(r, capi.BUF_REPLICA_GRAD) for r in range(8)], g)
    for t in replicas:
        t.normal_(0.0, 1e-4, generator=inputs.gen)
    return dict(group=g, maps=maps, expanded=expanded, upstream=[inputs.normal(m.shape, 1e-3) for m in expanded],
                grads=grads, tables=[g.pointer_tables([list(t) for t in per_rank]) for per_rank in grads], replicas=replicas)


def _prepare_gather(case, seed):
    inputs = _Inputs(seed, case["physical"], case["zipf"])
    lib = capi.lib()
    n = case["tokens"] * case["topk"]
    rows = inputs.normal((n, case["hidden"]), 1e-3, torch.bfloat16)
    return dict(lib=lib, rows=rows, out=torch.empty_like(rows), phys=inputs.topk_ids(case["tokens"], case["topk"]),
                pos=torch.empty(n, dtype=torch.int32, device=DEV), physical=case["physical"],
                offsets=torch.empty(case["physical"] + 1, dtype=torch.int32, device=DEV),
                scratch=torch.empty(lib.uep_dispatch_scratch_elems(n, case["physical"]), dtype=torch.int32, device=DEV),
                status=torch.zeros(2, dtype=torch.int32, device=DEV))


def _prepare_solve(case, seed):
    L = case["ranks"] * case["masters"]
    inputs = _Inputs(seed, L, case["zipf"])
    loads = torch.stack([_count(inputs.topk_ids(case["tokens"], case["topk"]), L) for _ in range(case["ranks"])])
    return dict(lib=capi.lib(), loads=loads, total=torch.empty(L, dtype=torch.int32, device=DEV),
                plan=_plan_buffers(case["ranks"], case["masters"], case["redundant"]),
                shape=(case["ranks"], case["masters"], case["redundant"]), params=capi.SolverParams.defaults(),
                status=torch.zeros(2, dtype=torch.int32, device=DEV))


def _prepare_reroute(case, seed):
    N, L, R, T, K = case["ranks"], case["experts"], case["redundant"], case["tokens"], case["topk"]
    M, P = L // N, L + N * R
    inputs = _Inputs(seed, L, case["zipf"])
    lib = capi.lib()
    ids = [inputs.topk_ids(T, K) for _ in range(N)]
    plan = _plan_buffers(N, M, R)
    _solve(lib, torch.stack([_count(x, L) for x in ids]), torch.empty(L, dtype=torch.int32, device=DEV), plan, N, M, R,
           capi.SolverParams.defaults(), 0, torch.zeros(2, dtype=torch.int32, device=DEV))
    rmap = _to_map(ids[0], L)
    scratch = max(lib.uep_reroute_scratch_elems(T, 0, L), lib.uep_reroute_scratch_elems(T, K, L))
    return dict(lib=lib, ids=ids[0], phys=torch.empty_like(ids[0]), rmap=rmap, probs=inputs.probs(rmap), plan=plan,
                shape=(T, K, L, P, N), upstream=inputs.normal((T, P), 1e-3),
                expanded_map=torch.empty((T, P), dtype=torch.bool, device=DEV),
                expanded_probs=torch.empty((T, P), dtype=torch.float32, device=DEV),
                grad=torch.empty((T, L), dtype=torch.float32, device=DEV),
                scratch=torch.empty(scratch, dtype=torch.int32, device=DEV))


_PREPARE = dict(manager_sparse=_prepare_manager_sparse, manager_dense=_prepare_manager_dense, forward=_prepare_forward,
                backward=_prepare_backward, gather=_prepare_gather, solve=_prepare_solve, reroute=_prepare_reroute)


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


# -- run -------------------------------------------------------------------------------------
def _run_manager_sparse(s):
    mgr = s["mgr"]
    layer = mgr.allocate_microbatch_slot(1)
    mgr.update_placement_sparse(layer, s["ids"])
    done = mgr.weight_sync(layer, async_finish=True)
    mgr.reroute_sparse(layer, s["ids"])  # in place; one rank's physical slots begin with its masters, so the ids stay
    done.current_stream_wait()
    return [s["ids"], s["plan"]]


def _run_manager_dense(s):
    mgr = s["mgr"]
    layer = mgr.allocate_microbatch_slot(1)
    mgr.update_placement(layer, s["rmap"])
    done = mgr.weight_sync(layer, async_finish=True)
    probs, rmap = mgr.reroute(layer, s["probs"], s["rmap"])
    done.current_stream_wait()
    (grad,) = torch.autograd.grad(probs, s["probs"], s["upstream"])
    reduced = mgr.grad_reduce(layer, async_finish=True)
    reduced.current_stream_wait()
    return [probs, rmap, grad, s["plan"]]


def _run_forward(s):
    g = s["group"]
    g.update_placement(0, s["maps"] if "maps" in s else s["ids"])
    done = g.weight_sync(0, *s["tables"], async_finish=True) if "tables" in s else None
    routed = g.reroute_dense(0, s["maps"], s["probs"]) if "maps" in s else g.reroute_sparse(0, s["ids"], s["phys"])
    if done is not None:
        g.wait_event(done)
    return [routed, s["out"]]


def _run_backward(s):
    g = s["group"]
    probs = g.reroute_dense_backward(0, s["upstream"], s["maps"], s["expanded"])
    done = g.grad_reduce(0, *s["tables"], async_finish=True)
    g.wait_event(done)
    return [probs, s["grads"], s["replicas"]]


def _run_gather(s):
    lib, n = s["lib"], s["pos"].numel()
    capi.check(lib.uep_dispatch_positions(s["phys"].data_ptr(), n, s["physical"], s["pos"].data_ptr(), s["offsets"].data_ptr(),
                                          s["scratch"].data_ptr(), _stream()), "uep_dispatch_positions")
    capi.check(lib.uep_gather_rows(s["rows"].data_ptr(), s["pos"].data_ptr(), s["out"].data_ptr(), n, n,
                                   s["rows"].shape[1] * 2, s["status"].data_ptr(), _stream()), "uep_gather_rows")
    return [s["pos"], s["offsets"], s["out"], s["status"]]


def _run_solve(s):
    _solve(s["lib"], s["loads"], s["total"], s["plan"], *s["shape"], s["params"], 0, s["status"])
    return [s["total"], s["plan"], s["status"]]


def _run_reroute(s):
    lib, p, (T, K, L, P, D) = s["lib"], s["plan"], s["shape"]
    l2p, counts, prefix = p["l2p"].data_ptr(), p["lcnts"].data_ptr(), p["rank_quota_prefix"].data_ptr()
    rmap, expanded = s["rmap"].data_ptr(), s["expanded_map"].data_ptr()
    capi.check(lib.uep_sparse_reroute_i32(s["ids"].data_ptr(), s["phys"].data_ptr(), T, K, L, l2p, counts, prefix, D, 1,
                                          s["scratch"].data_ptr(), _stream()), "uep_sparse_reroute_i32")
    capi.check(lib.uep_dense_reroute_forward(rmap, s["probs"].data_ptr(), l2p, counts, prefix, expanded,
                                             s["expanded_probs"].data_ptr(), s["scratch"].data_ptr(), T, L, P, D, 1, 1,
                                             _stream()), "uep_dense_reroute_forward")
    capi.check(lib.uep_dense_reroute_backward(s["upstream"].data_ptr(), rmap, expanded, l2p, counts, s["grad"].data_ptr(), T, L,
                                              P, D, _stream()), "uep_dense_reroute_backward")
    return [s["phys"], s["expanded_map"], s["expanded_probs"], s["grad"]]


_RUN = dict(manager_sparse=_run_manager_sparse, manager_dense=_run_manager_dense, forward=_run_forward,
            backward=_run_backward, gather=_run_gather, solve=_run_solve, reroute=_run_reroute)


def run(state):
    return _RUN[state["kind"]](state)


# -- work ------------------------------------------------------------------------------------
def _replicas(case):
    """(experts with replicas, replicas) of a typical plan of this case: the one of seed 0's routing."""
    inputs = _Inputs(0, case["experts"], case["zipf"])
    loads = torch.stack([_count(inputs.topk_ids(t, case["topk"], case.get("hot", False)), case["experts"])
                         for t in _tokens_per_rank(case)])
    plan = _plan_buffers(8, case["experts"] // 8, case["redundant"])
    _solve(capi.lib(), loads, torch.empty(case["experts"], dtype=torch.int32, device=DEV), plan, 8, case["experts"] // 8,
           case["redundant"], capi.SolverParams.defaults(), 0, torch.zeros(2, dtype=torch.int32, device=DEV))
    extra = plan["lcnts"] - 1
    return int((extra > 0).sum()), int(extra.sum())


def _dense_bytes(T, K, L, P):
    return T * L + 4 * T * K + 5 * T * P  # map and the routed probabilities read, both expanded outputs written


def work(case):
    kind = case["kind"]
    if kind == "solve":
        N, L, P = case["ranks"], case["ranks"] * case["masters"], case["ranks"] * (case["masters"] + case["redundant"])
        return {"bytes": 4 * (N * L + 2 * L + P + 4 * L * N), "flops": 0}
    T, K = case["tokens"], case["topk"]
    if kind == "gather":
        return {"bytes": T * K * (4 + 4 + 4 * case["hidden"]), "flops": 0}
    L, R = case["experts"], case["redundant"]
    if kind == "manager_sparse":  # ids read and written, and the plan
        return {"bytes": 16 * T * K + 4 * (6 * L + R), "flops": 0}
    if kind == "manager_dense":
        return {"bytes": _dense_bytes(T, K, L, L + R) + 4 * T * K + 4 * T * L, "flops": 0}
    P = L + 8 * R
    if kind == "reroute":
        return {"bytes": 8 * T * K + _dense_bytes(T, K, L, P) + 4 * T * K + 4 * T * L, "flops": 0}
    total = sum(_tokens_per_rank(case))
    if kind == "forward":
        bytes_ = 8 * 4 * (P + L + 4 * L * 8)
        bytes_ += _dense_bytes(total, K, L, P) if case["ids"] == "map" else 2 * total * K * (8 if case["ids"] == "int64" else 4)
        if case["weights"] != "none":
            fc1, fc2, elem, s1, s2 = _layer_sizes(case)
            bytes_ += sum(_replicas(case)) * ((fc1 + fc2) * elem + s1 + s2)  # each such master read once, each replica written
        return {"bytes": bytes_, "flops": 0}
    hot, replicas = _replicas(case)
    numel = 3 * case["hidden"] * case["ffn"]
    # masters with replicas read and written, replicas read and cleared, one addition per replica element
    return {"bytes": 8 * numel * (hot + replicas) + total * (L + 4 * K + 4 * L), "flops": numel * replicas}


def tolerance(case):
    """Plans, ids, copied bytes and probabilities are copies or whole numbers; reduced gradients are summed in a fixed
    order in fp32, so they are the same bits too."""
    return "exact"
