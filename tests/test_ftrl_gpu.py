"""FTRL fused kernels on one GPU against the fp64 CPU restatement of the reference."""
import numpy as np
import pytest
import torch

from baseline.cpu_ref.ftrl_ref import FTRLRef
from parameter_server_b200.data.synthetic import ctr_minibatch

pytestmark = pytest.mark.gpu


def _engine(impl="fused", rule="count", **kw):
    from parameter_server_b200.models.ftrl import FTRLEngine, FTRLHyper
    from parameter_server_b200.parallel.peer import PeerGroup

    hyper = FTRLHyper(alpha=0.02, beta=1.0, lambda1=0.05, lambda2=0.1, rule=rule)
    args = dict(table_capacity=1 << 16, max_rows=4096, max_nnz=1 << 19, local_capacity=1 << 16)
    args.update(kw)
    return FTRLEngine(PeerGroup.single(torch.device("cuda", 0)), hyper, impl=impl, **args), hyper


def _batches(n, rows=700, log2=13):
    return [ctr_minibatch(rows, seed=100 + i, device="cuda", key_space_log2=log2, bias=-0.5, wstar_frac=0.2,
                          wstar_std=1.0) for i in range(n)]


@pytest.mark.parametrize("impl,rule,counts", [("fused", "count", None), ("fused", "sumsq", None),
                                              ("fused", "sumsq", True), ("nccl", "count", None)])
def test_ftrl_matches_oracle(impl, rule, counts):
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, hy = _engine(impl, rule, track_counts=counts)
    assert eng.track_counts == (rule == "count" or bool(counts))
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, rule)
    for off, keys, y in _batches(6):
        eng.step(DeviceMinibatch(off, keys, y))
        st = eng.read_stats()
        eng.check_status()
        loss = ref.step([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), y.cpu().numpy().astype(np.float64))])
        assert st["rows"] == y.numel()
        assert st["loss_sum"] == pytest.approx(loss, rel=2e-4)
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert len(rk) > 50
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)
    st = eng.read_stats(reset=False)
    assert st["nnz_w"] == ref.nnz
    assert st["norm1"] == pytest.approx(ref.norm1, rel=1e-3)
    assert st["table_entries"] == len(ref.model)
    assert eng.penalty(st) == pytest.approx(ref.objv(), rel=1e-3)


@pytest.mark.parametrize("rule", ["count", "sumsq"])
def test_ftrl_valued_features_and_predict(rule):
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, hy = _engine(rule=rule)
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, rule)
    g = torch.Generator(device="cuda").manual_seed(3)
    for off, keys, y in _batches(4, rows=300, log2=10):
        vals = torch.rand(keys.numel(), generator=g, device="cuda") + 0.5
        eng.step(DeviceMinibatch(off, keys, y, vals))
        ref.step([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), y.cpu().numpy().astype(np.float64),
                   vals.cpu().numpy())])
    off, keys, y = _batches(1, rows=200, log2=10)[0]
    xw = eng.predict(DeviceMinibatch(off, keys, y)).cpu().numpy()
    _, _, _, _, _, rxw = ref.worker_gradient(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64),
                                             y.cpu().numpy().astype(np.float64))
    np.testing.assert_allclose(xw, rxw, rtol=2e-3, atol=2e-4)
    # predict leaves training state untouched: one more step still matches
    eng.step(DeviceMinibatch(off, keys, y))
    ref.step([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), y.cpu().numpy().astype(np.float64))])
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)
    eng.check_status()


@pytest.mark.parametrize("impl", ["fused", "nccl"])
def test_tail_feature_filter_matches_oracle(impl):
    """Keys enter the model only once their count-min estimate exceeds tail_feature_freq."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch, FTRLEngine, FTRLHyper
    from parameter_server_b200.parallel.peer import PeerGroup

    hy = FTRLHyper(alpha=0.02, beta=1.0, lambda1=0.05, lambda2=0.1, tail_feature_freq=3, countmin_n=1 << 15, countmin_k=2)
    eng = FTRLEngine(PeerGroup.single(torch.device("cuda", 0)), hy, impl=impl, table_capacity=1 << 16, max_rows=4096,
                     max_nnz=1 << 19, local_capacity=1 << 16)
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, tail_freq=3, countmin_n=hy.countmin_n, countmin_k=2)
    seen = set()
    for off, keys, y in _batches(4, rows=300, log2=14):
        eng.step(DeviceMinibatch(off, keys, y))
        eng.check_status()
        hk = keys.cpu().numpy().view(np.uint64)
        seen.update(hk.tolist())
        ref.step([(off.cpu().numpy(), hk, y.cpu().numpy().astype(np.float64))])
    st = eng.read_stats(reset=False)
    assert st["table_entries"] == len(ref.model)
    assert 50 < len(ref.model) < 0.8 * len(seen)      # the filter kept a real share of the keys out
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)


def test_ftrl_reports_local_table_overflow():
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, _ = _engine(local_capacity=256, max_probe=64)
    off, keys, y = _batches(1, rows=200)[0]
    eng.step(DeviceMinibatch(off, keys, y))
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="dedup table full"):
        eng.check_status()


@pytest.mark.parametrize("rule", ["count", "sumsq"])
def test_minibatches_of_changing_size_and_one_without_repeated_keys(rule):
    """A step works in as many slots as its minibatch suggests and starts over with more when the keys do not fit;
    the accumulators of a large step are clean when a later step goes as far again."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, hy = _engine(rule=rule, table_capacity=1 << 21, local_capacity=1 << 20, max_rows=8192)
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, rule)
    small, large = _batches(1, rows=60)[0], _batches(1, rows=2000)[0]
    # all keys distinct: 2^18 slots, which three quarters of the non-zeros ask for, cannot hold 300,000
    g = torch.Generator(device="cuda").manual_seed(5)
    keys = torch.randperm(1 << 22, generator=g, device="cuda")[:300_000] * 0x9E3779B9
    off = torch.arange(0, 300_001, 60, device="cuda")
    y = torch.where(torch.rand(5000, generator=g, device="cuda") < 0.5, 1.0, -1.0)
    distinct = (off, keys, y)
    used = []
    for off, keys, y in [large, small, large, small, distinct, small, small, distinct, large]:
        eng.step(DeviceMinibatch(off, keys, y))
        eng.check_status()
        used.append(int(eng.region[0].item()))
        ref.step([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), y.cpu().numpy().astype(np.float64))])
        before = eng.stats.clone()
        xw = eng.predict(DeviceMinibatch(*small)).cpu().numpy()
        assert torch.equal(eng.stats, before)
        rxw = ref.worker_gradient(small[0].cpu().numpy(), small[1].cpu().numpy().view(np.uint64), small[2].cpu().numpy().astype(np.float64))[5]
        np.testing.assert_allclose(xw, rxw, rtol=2e-3, atol=2e-4)
    assert used[1] < used[0] < used[4] <= eng.region_log2 and used[5] == used[4], used
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)
    assert int((eng.lt_keys.local != -1).sum()) == 0
    assert eng.read_stats(reset=False)["table_entries"] == len(ref.model)


@pytest.mark.parametrize("valued", [False, True])
@pytest.mark.parametrize("rule", ["count", "sumsq"])
@pytest.mark.parametrize("launches,log2", [(1, 16), (2, 16), (2, 23)])
def test_rows_of_all_lengths(rule, valued, launches, log2):
    """Rows without non-zeros, around one warp and around what a warp keeps in registers, and far longer ones; in one
    and in two launches, and with more slots (2^23) than a packed slot reference can tell."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, hy = _engine(rule=rule, local_capacity=1 << log2, table_capacity=1 << 18)
    eng._L.two_launch_nnz = 1 if launches == 2 else 1 << 60
    eng.region[1] = log2 if log2 > 22 else 0
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, rule)
    rng = np.random.RandomState(4)
    for lens in ([0], [1], [0, 1, 31, 32, 33, 0, 127, 128, 129, 160, 1000, 0], [5] * 3000, [129] * 17):
        off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
        keys = rng.randint(0, 900, size=off[-1]).astype(np.int64) * 0x9E3779B97F
        y = np.where(rng.rand(len(lens)) < 0.4, 1.0, -1.0).astype(np.float32)
        vals = (rng.rand(off[-1]) + 0.5).astype(np.float32) if valued else None
        d = lambda a: None if a is None else torch.from_numpy(a).cuda()
        eng.step(DeviceMinibatch(d(off), d(keys), d(y), d(vals)))
        eng.check_status()
        want = ref.worker_gradient(off, keys.view(np.uint64), y.astype(np.float64), vals)[5] if off[-1] else np.zeros(len(lens))
        np.testing.assert_allclose(eng.xw[: len(lens)].cpu().numpy(), want, rtol=2e-3, atol=2e-4)
        if off[-1]:
            ref.step([(off, keys.view(np.uint64), y.astype(np.float64)) + ((vals,) if valued else ())])
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)


@pytest.mark.parametrize("impl", ["fused", "nccl"])
def test_keys_entered_by_the_update_itself_stay(impl):
    """Under the tail filter the update creates an entry and writes its sector back: every key is there once afterwards."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch, FTRLEngine, FTRLHyper
    from parameter_server_b200.parallel.peer import PeerGroup

    hyper = FTRLHyper(alpha=0.1, beta=1.0, lambda1=0.0, lambda2=0.1, rule="count", tail_feature_freq=1, countmin_n=1 << 24)
    n = 60_000
    eng = FTRLEngine(PeerGroup.single(torch.device("cuda", 0)), hyper, table_capacity=1 << 18, max_rows=4096, max_nnz=2 * n, local_capacity=1 << 18,
                     impl=impl)
    g = torch.Generator(device="cuda").manual_seed(8)
    keys = torch.arange(1, n + 1, device="cuda") * 0x9E3779B97F
    off = torch.arange(0, 2 * n + 1, 40, device="cuda")
    for _ in range(3):
        mb = torch.cat([keys, keys])[torch.randperm(2 * n, generator=g, device="cuda")]      # every key passes the filter at once
        eng.step(DeviceMinibatch(off, mb, torch.ones(off.numel() - 1, device="cuda")))
        eng.check_status()
        held = eng.tab.local[:, 0]
        assert torch.equal(held[held != -1].sort().values, keys.sort().values)
    assert eng.read_stats(reset=False)["table_entries"] == n


@pytest.mark.parametrize("threshold,launches", [(1, 2), (1 << 60, 1)])
def test_launches_of_a_step_are_counted(threshold, launches):
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, _ = _engine()
    eng._L.two_launch_nnz = threshold
    mb = DeviceMinibatch(*_batches(1)[0])
    before = eng.kernel_launches
    for _ in range(3):
        eng.step(mb)
    assert eng.kernel_launches - before == 3 * launches
    eng.predict(mb)
    assert eng.kernel_launches - before == 3 * launches + 1


@pytest.mark.parametrize("threshold", [1, 1 << 60])
def test_phase_times_tell_the_gap_between_two_launches(threshold):
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, _ = _engine()
    eng._L.two_launch_nnz = threshold
    mb = DeviceMinibatch(*_batches(1)[0])
    for _ in range(3):
        eng.step(mb)
    t = eng.phase_times_us()
    assert all(v >= 0 for v in t.values()) and t["rows"] > 0
    assert sum(v for k, v in t.items() if k != "step") == pytest.approx(t["step"], abs=0.01)
    assert t["kernel_gap"] > 0 if threshold == 1 else t["kernel_gap"] == 0


@pytest.mark.parametrize("rule", ["count", "sumsq"])
@pytest.mark.parametrize("share,log2", [(0.5, 18), (0.75, 19), (0.87, 19)])
def test_a_table_with_long_chains_is_left_for_a_larger_one(rule, share, log2):
    """300,000 non-zeros start in 2^18 slots; keys that would fill them to 0.86 fit, but at the end of long chains."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, hy = _engine(rule=rule, table_capacity=1 << 21, local_capacity=1 << 20, max_rows=8192)
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, rule)
    g = torch.Generator(device="cuda").manual_seed(6)
    n = 300_000
    for _ in range(2):
        ids = torch.cat([torch.arange(int(n * share), device="cuda"),
                         torch.randint(0, int(n * share), (n - int(n * share),), generator=g, device="cuda")])
        keys = ids[torch.randperm(n, generator=g, device="cuda")] * 0x9E3779B9
        off = torch.arange(0, n + 1, 60, device="cuda")
        y = torch.where(torch.rand(n // 60, generator=g, device="cuda") < 0.5, 1.0, -1.0)
        eng.step(DeviceMinibatch(off, keys, y))
        eng.check_status()
        assert int(eng.region[0].item()) == log2
        ref.step([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), y.cpu().numpy().astype(np.float64))])
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)
    assert eng.read_stats(reset=False)["table_entries"] == len(ref.model) == int(n * share)


@pytest.mark.parametrize("rule", ["count", "sumsq"])
def test_millions_of_distinct_keys_match_the_unfused_engine(rule):
    """Almost every slot of the largest table used: rows are walked once for the weights and once for the gradients."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    n = 6_600_000
    g = torch.Generator(device="cuda").manual_seed(9)
    off = torch.arange(0, n + 1, 60, device="cuda")
    y = torch.where(torch.rand(n // 60, generator=g, device="cuda") < 0.5, 1.0, -1.0)
    mbs = [DeviceMinibatch(off, torch.randperm(n, generator=g, device="cuda") * 0x9E3779B97F, y) for _ in range(2)]
    got = []
    for impl in ("fused", "nccl"):
        eng, _ = _engine(impl, rule, table_capacity=1 << 24, local_capacity=1 << 24, max_rows=n // 60, max_nnz=n)
        for mb in mbs:
            eng.step(mb)
        eng.check_status()
        if impl == "fused":
            assert int(eng.region[0].item()) == 24
        st = eng.read_stats(reset=False)
        got.append((*eng.dump_model(), eng.predict(mbs[0]).cpu().numpy(), st["loss_sum"], st["table_entries"]))
        del eng
        torch.cuda.empty_cache()
    (k, w, xw, loss, entries), (rk, rw, rxw, rloss, rentries) = got
    assert entries == rentries == n and len(k) > 1000 and np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=1e-4, atol=1e-6)
    np.testing.assert_allclose(xw, rxw, rtol=1e-4, atol=1e-5)
    assert loss == pytest.approx(rloss, rel=1e-6)


def test_model_text_dump(tmp_path):
    from parameter_server_b200.models.ftrl import DeviceMinibatch
    from parameter_server_b200.utils.modelio import read_model_text

    eng, _ = _engine()
    for off, keys, y in _batches(3):
        eng.step(DeviceMinibatch(off, keys, y))
    path = eng.save_model(str(tmp_path / "ftrl"))
    assert path.endswith("_S0")
    k, w = eng.dump_model()
    m = read_model_text(path)
    assert len(m) == len(k)
    for kk, ww in zip(k[:50], w[:50]):
        assert m[int(kk)] == pytest.approx(float(ww), rel=1e-5)



def test_compact_inputs_give_the_same_model():
    """32-bit feature ids hashed on the device + 32-bit row offsets == the same minibatches as uint64 keys."""
    from parameter_server_b200.models.ftrl import KEY_U32, KEY_U32_HASHED, DeviceMinibatch

    a, _ = _engine(rule="sumsq")
    b, _ = _engine(rule="sumsq")
    c, _ = _engine(rule="sumsq")
    d, _ = _engine(rule="sumsq")
    for i in range(4):
        off, keys, y, fid = ctr_minibatch(500, seed=40 + i, device="cuda", key_space_log2=13, bias=-0.5, wstar_frac=0.2,
                                          wstar_std=1.0, return_ids=True)
        a.step(DeviceMinibatch(off, keys, y))
        b.step(DeviceMinibatch(off.to(torch.int32), fid, y, None, KEY_U32_HASHED))
        c.step(DeviceMinibatch(off, fid.to(torch.int64), y))             # the ids themselves as keys, 64 bits wide
        d.step(DeviceMinibatch(off.to(torch.int32), fid, y, None, KEY_U32))
    for e in (a, b, c, d):
        e.check_status()
    (ka, wa), (kb, wb), (kc, wc), (kd, wd) = a.dump_model(), b.dump_model(), c.dump_model(), d.dump_model()
    assert len(ka) > 50 and np.array_equal(ka, kb) and np.array_equal(kc, kd)
    np.testing.assert_allclose(wa, wb, rtol=1e-5, atol=1e-7)     # same arithmetic, different summation order of atomics
    np.testing.assert_allclose(wc, wd, rtol=1e-5, atol=1e-7)
    with pytest.raises(ValueError, match="32-bit keys"):
        a.step(DeviceMinibatch(off, fid, y))


@pytest.mark.parametrize("rule", ["count", "sumsq"])
def test_shard_table_grows_instead_of_filling_up(rule):
    """A shard that starts far too small doubles between steps; the model stays the oracle's."""
    from parameter_server_b200.models.ftrl import DeviceMinibatch

    eng, hy = _engine(rule=rule, table_capacity=1 << 11, local_capacity=1 << 13)
    assert eng.cap == 1 << 14                       # room for one worst-case step from the start
    ref = FTRLRef(hy.alpha, hy.beta, hy.lambda1, hy.lambda2, rule)
    for off, keys, y in _batches(6, rows=120, log2=13):
        eng.step(DeviceMinibatch(off, keys, y))
        eng.check_status()
        eng.maybe_grow()
        ref.step([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), y.cpu().numpy().astype(np.float64))])
    assert eng.grown >= 1 and eng.cap > 1 << 14
    st = eng.read_stats(reset=False)
    assert st["table_entries"] == len(ref.model) and st["table_entries"] + eng.lcap <= eng.GROW_AT * eng.cap
    k, w = eng.dump_model()
    rk, rw = ref.nonzero()
    assert np.array_equal(k, rk)
    np.testing.assert_allclose(w, rw, rtol=2e-3, atol=2e-5)
