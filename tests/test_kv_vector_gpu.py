"""DeviceKVVector on one GPU (fused and NCCL-baseline code paths) against a dictionary model."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("impl", ["fused", "nccl"])
@pytest.mark.parametrize("k", [1, 3, 8])
def test_push_pull_roundtrip(impl, k):
    from parameter_server_b200.parallel.kv_vector import DeviceKVVector
    from parameter_server_b200.parallel.peer import PeerGroup

    rng = np.random.RandomState(k)
    server = np.unique(rng.randint(0, 2**62, size=5000).astype(np.uint64) * 3)
    kv = DeviceKVVector(PeerGroup.single(torch.device("cuda", 0)), k=k, impl=impl)
    mine = kv.merge_keys(torch.from_numpy(server.view(np.int64)).cuda())
    assert np.array_equal(mine.cpu().numpy().view(np.uint64), server)
    kv.set_keys(mine)
    q = np.concatenate([rng.choice(server, 3000, replace=False), np.array([1, 2], dtype=np.uint64)])   # two unknown keys
    owner, slot = kv.resolve(torch.from_numpy(q.view(np.int64)).cuda())
    assert (slot[-2:] == -1).all() and (slot[:-2] >= 0).all() and (owner == 0).all()
    assert np.array_equal(server[slot[:-2].cpu().numpy()], q[:-2])
    v1 = torch.randn(len(q), k, device="cuda")
    kv.push(owner, slot, v1)
    kv.push(owner, slot, v1)                          # pushes accumulate
    out = kv.pull(owner, slot)
    torch.testing.assert_close(out[:-2], 2 * v1[:-2])
    assert (out[-2:] == 0).all()
    assert kv.local_values.abs().sum().item() == pytest.approx((2 * v1[:-2]).abs().sum().item(), rel=1e-4)


@pytest.mark.parametrize("n", [1, 255, 511, 512, 513, 4000])
@pytest.mark.parametrize("shards", [1, 3])
@pytest.mark.parametrize("held", [0, 1, 33, 5000, 60000])
def test_resolve_over_list_orders_and_run_lengths(n, shards, held):
    """Ordered lists (short and long runs of the shard per tile), unordered ones, tiles over several owners (their
    shards side by side on this GPU), empty shards, keys below, between and above those held."""
    import ctypes as C

    from parameter_server_b200.ops import _native as N
    from parameter_server_b200.parallel.kv_vector import KvPeers
    from parameter_server_b200.utils.range import Range

    rng = np.random.RandomState(n + held)
    server = np.unique(rng.randint(0, 2**63, size=held).astype(np.uint64) * 2 + 1)
    seps = Range.all().separators(shards)
    P, keep = KvPeers(), []
    for r in range(shards):
        mine = server[(server >= seps[r]) & (server < np.uint64(seps[r + 1]))]
        keep.append((mine, torch.from_numpy(mine.view(np.int64).copy()).cuda() if len(mine) else torch.zeros(1, dtype=torch.int64, device="cuda")))
        P.keys[r], P.vals[r], P.nkeys[r] = keep[-1][1].data_ptr(), keep[-1][1].data_ptr(), len(mine)
    for i in range(N.MAX_RANKS + 1):
        P.seps.sep[i] = seps[i] if i < len(seps) else N.EMPTY_KEY
    P.seps.world, P.k = shards, 1
    known = rng.choice(server, min(n, len(server)), replace=False) if len(server) else server
    q = np.concatenate([known, rng.randint(0, 2**63, size=n).astype(np.uint64) * 2])[:n]
    q[-1] = 0 if n % 2 else 2**64 - 2
    for query in (np.sort(q), q, np.sort(q)[::-1].copy(), np.repeat(q[:1], n)):
        t = torch.from_numpy(query.view(np.int64).copy()).cuda()
        owner, slot = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        N.check(N.lib().psb_kv_resolve(C.byref(P), N.ptr(t), C.c_size_t(n), N.ptr(owner), N.ptr(slot), N.stream_ptr()), "resolve")
        o = np.searchsorted(np.array(seps[1:-1], dtype=np.uint64), query, side="right")
        want = np.full(n, -1)
        for r in range(shards):
            at = np.searchsorted(keep[r][0], query)
            hit = (o == r) & (at < len(keep[r][0]))
            hit[hit] = keep[r][0][at[hit]] == query[hit]
            want[hit] = at[hit]
        assert np.array_equal(owner.cpu().numpy(), o) and np.array_equal(slot.cpu().numpy(), want)


@pytest.mark.parametrize("n,held", [(151_551, 60_000), (151_552, 400_000), (151_553, 60_000), (303_103, 60_000), (303_104, 1_000_000),
                                    (303_105, 60_000), (2_600_000, 4_000_000)])
@pytest.mark.parametrize("shards", [1, 3])
def test_resolve_with_several_queries_a_thread(n, shards, held):
    """Two and four queries a thread (from 151,552 and 303,104 on), and more tiles than the grid has thread blocks."""
    test_resolve_over_list_orders_and_run_lengths(n, shards, held)
