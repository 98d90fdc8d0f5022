"""weight_sync of a group that is hosted whole puts its counters back while its last copies are on their way: launch after launch on one
group, with plans of no replica, of few and of many, shorter and longer than the launch has CTAs, aligned masters and others. Bytes exact."""

import pytest
import torch

from ultra_ep_b200 import capi, sim

pytestmark = pytest.mark.gpu


def _ids(kind, N, L, gen, device):
    if kind == "even":  # every expert alike: nothing to replicate
        return [torch.arange(4 * L, dtype=torch.int32, device=device).remainder(L).view(-1, 4) for _ in range(N)]
    weights = torch.full((L,), 1.0, device=device)
    weights[torch.randint(0, L, (1 if kind == "one hot" else L // 3,), generator=gen, device=device)] = 60.0
    return [torch.multinomial(weights, 4 * 300, replacement=True, generator=gen).int().view(-1, 4) for _ in range(N)]


@pytest.mark.parametrize("N,M,R", [(2, 3, 1), (3, 5, 2), (8, 8, 2), (8, 40, 8)])
@pytest.mark.parametrize("fc1,fc2", [(64, 16), (16 * 4099, 16 * 513), (3 << 20, 1 << 20)])
@pytest.mark.parametrize("offset", [0, 4])
def test_launch_after_launch(native_lib, cuda_device, N, M, R, fc1, fc2, offset):
    if N * M > 100 and fc1 > 1 << 20:
        pytest.skip("memory")
    L, Lp = N * M, M + R
    gen = torch.Generator(device=cuda_device).manual_seed(N + fc1)
    group = sim.SimGroup(sim.make_config(N, M, R, 1, fc1_numel=fc1, fc2_numel=fc2, weight_elem_bytes=1, is_train=False, sim=True))
    pool = torch.randint(0, 256, (2, L, max(fc1, fc2) + 16), dtype=torch.uint8, device=cuda_device, generator=gen)
    shards = [[[pool[i, r * M + m, offset:offset + n] for m in range(M)] for r in range(N)] for i, n in enumerate((fc1, fc2))]
    tables = [group.pointer_tables(s) for s in shards]
    seen = 0
    for kind in ("many", "even", "one hot", "even", "even", "many", "one hot", "many"):
        replicas = [group.buffer(r, capi.BUF_REPLICA_WEIGHT) for r in range(N)]
        for t in replicas:
            t.zero_()
        group.update_placement(0, _ids(kind, N, L, gen, cuda_device))
        group.weight_sync(0, *tables)
        torch.cuda.synchronize()
        group.check_status()
        p2l = group.plan(0, 0)["p2l"].cpu().view(N, Lp)[:, M:]
        assert kind != "even" or (p2l < 0).all()
        for r in range(N):
            for s in range(R):
                e = int(p2l[r, s])
                want = torch.zeros(fc1 + fc2, dtype=torch.uint8, device=cuda_device)
                if e >= 0:
                    want = torch.cat([shards[i][e // M][e % M] for i in range(2)])
                    seen += 1
                assert torch.equal(replicas[r][s], want), (kind, r, s)
    assert seen > 0
    group.destroy()
