"""DARLIN pass kernel on one GPU against the fp64 CPU restatement of the reference."""
import numpy as np
import pytest
import torch

from baseline.cpu_ref.darlin_ref import DarlinConfig as RefConfig
from baseline.cpu_ref.darlin_ref import DarlinRef
from parameter_server_b200.data.synthetic import zipf_sparse_matrix

pytestmark = pytest.mark.gpu


def _problem(binary, rows=1500, cols=2048, nnz=16, seed=1):
    off, idx, vals, y, _ = zipf_sparse_matrix(rows, cols, nnz, seed=seed, device="cuda", binary=binary, zipf_s=0.8)
    # spread ids over a larger uint64 key space, keep order
    keys = idx * 7919 + 3
    return off, keys, vals, y


@pytest.mark.parametrize("binary", [False, True])
@pytest.mark.parametrize("impl", ["fused", "nccl"])
def test_darlin_matches_oracle(binary, impl):
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(binary)
    kw = dict(lambda1=0.3, max_pass=6, feature_block_ratio=1.0, kkt_ratio=10.0, seed=3)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(**kw), impl=impl)
    sol.preprocess(off, keys, vals, y)
    prog = sol.run()
    ref = DarlinRef([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64),
                      None if vals is None else vals.cpu().numpy(), y.cpu().numpy())], None, RefConfig(**kw))
    rprog = ref.run()
    assert sol.nblk == len(ref.blocks) and sol.nblk > 4
    assert len(prog) == len(rprog)
    for p, r in zip(prog, rprog):
        assert p.objv == pytest.approx(r.objv, rel=2e-3)
        assert abs(p.nnz_w - r.nnz_w) <= max(3, 0.03 * r.nnz_w)
        assert p.violation == pytest.approx(r.violation, rel=2e-2, abs=1e-3)
    objs = [p.objv for p in prog]
    assert all(b <= a * (1 + 1e-4) for a, b in zip(objs, objs[1:])), objs
    k, w = sol.model()
    rk, rw = ref.model()
    common = np.intersect1d(k, rk)
    assert len(common) >= 0.95 * max(len(k), len(rk))
    wd = dict(zip(k.tolist(), w.tolist()))
    rd = dict(zip(rk.tolist(), rw.tolist()))
    err = np.array([wd[c] - rd[c] for c in common.tolist()])
    assert np.abs(err).max() < 5e-2
    sol.check_status()


@pytest.mark.parametrize("tau", [0, 2])
def test_wide_block_path_matches_oracle(tau):
    """Groups with many columns fetch the owners' sums once per column and update the margins in a second step;
    forced here for every group by a threshold of one column."""
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(False)
    kw = dict(lambda1=0.3, max_pass=4, feature_block_ratio=1.0, seed=3, max_block_delay=tau)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(**kw), wide_block_cols=1)
    sol.preprocess(off, keys, vals, y)
    prog = sol.run()
    sol.check_status()
    ref = DarlinRef([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), vals.cpu().numpy(), y.cpu().numpy())], None,
                    RefConfig(**kw))
    for p, r in zip(prog, ref.run()):
        assert p.objv == pytest.approx(r.objv, rel=2e-3)
        assert abs(p.nnz_w - r.nnz_w) <= max(3, 0.03 * r.nnz_w)


@pytest.mark.parametrize("tau", [1, 3])
def test_bounded_delay_groups_match_oracle(tau):
    """max_block_delay = tau: tau+1 blocks share their synchronisation points (all gradients before any update)."""
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(False)
    kw = dict(lambda1=0.3, max_pass=4, feature_block_ratio=1.0, seed=3, max_block_delay=tau)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(**kw))
    sol.preprocess(off, keys, vals, y)
    prog = sol.run()
    ref = DarlinRef([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), vals.cpu().numpy(), y.cpu().numpy())], None,
                    RefConfig(**kw))
    rprog = ref.run()
    for p, r in zip(prog, rprog):
        assert p.objv == pytest.approx(r.objv, rel=2e-3)
    sol.check_status()


@pytest.mark.parametrize("binary", [False, True])
@pytest.mark.parametrize("rows,nnz,ratio,tau,wide", [
    (40, 3, 2.0, 0, 0),          # blocks of a few non-zeros, some of a single chunk
    (1500, 16, 1.0, 0, 0),
    (9000, 40, 0.1, 0, 0),       # 90 k non-zeros per block: more than a cluster's threads keep in registers
    (9000, 40, 0.2, 2, 0),       # the same over a bounded-delay group whose order ends in a shorter group
    (9000, 40, 0.2, 2, 1),       # ... with every column stepped once in a phase of its own
])
@pytest.mark.parametrize("variant", [1, 2])
def test_one_gpu_pass_variants_match_oracle(variant, rows, nnz, ratio, tau, wide, binary):
    """The whole-GPU and the one-cluster form of the resident one-GPU pass."""
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(binary, rows=rows, nnz=nnz)
    kw = dict(lambda1=0.3, max_pass=3, feature_block_ratio=ratio, seed=3, max_block_delay=tau)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(**kw), wide_block_cols=wide)
    sol.pass_variant = variant
    sol.preprocess(off, keys, vals, y)
    prog = sol.run()
    sol.check_status()
    ref = DarlinRef([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), None if vals is None else vals.cpu().numpy(),
                      y.cpu().numpy())], None, RefConfig(**kw))
    for p, r in zip(prog, ref.run()):
        assert p.objv == pytest.approx(r.objv, rel=2e-3)
        assert abs(p.nnz_w - r.nnz_w) <= max(3, 0.03 * r.nnz_w)
        assert p.violation == pytest.approx(r.violation, rel=2e-2, abs=1e-3)
    # the margins that were kept up to date are those of the weights
    from parameter_server_b200.models.darlin import margins_from_weights
    want = margins_from_weights(sol.col_ptr, sol.row_idx, sol.vals, sol.y, sol.w)
    assert torch.allclose(sol.margin, want, rtol=1e-4, atol=1e-4)
    assert torch.equal(sol.srv_gu.local[0], torch.zeros_like(sol.srv_gu.local[0]))


@pytest.mark.parametrize("variant", [1, 2])
def test_block_swept_twice_in_a_row_sees_its_own_update(variant):
    """A block that follows itself in the order reads the columns that were written just before."""
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(False)
    got = []
    for orders in ([[0, 0, 1, 1, 1, 0]], [[0], [0], [1], [1], [1], [0]]):
        sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(lambda1=0.3, feature_block_ratio=0.5, seed=3))
        sol.pass_variant = variant
        sol.preprocess(off, keys, vals, y)
        for o in orders:
            sol.launch_pass(np.asarray(o, dtype=np.int32))
        sol.check_status()
        got.append((sol.w.clone(), sol.margin.clone(), sol.delta.clone()))
    for a, b in zip(*got):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5)      # sums of the same terms in another order


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("variant", [1, 2])
def test_block_twice_in_one_bounded_delay_group(variant, wide):
    """A block that its group holds already ends the group: it is swept twice, and the margins are those of the weights."""
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver, margins_from_weights
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(False)
    got = []
    for orders, tau in (([[0, 1, 1, 0, 0, 1]], 2), ([[0, 1], [1, 0], [0, 1]], 1)):
        sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)),
                           DarlinConfig(lambda1=0.3, feature_block_ratio=0.5, seed=3, max_block_delay=tau), wide_block_cols=wide)
        sol.pass_variant = variant
        sol.preprocess(off, keys, vals, y)
        for o in orders:
            sol.launch_pass(torch.tensor(o, dtype=torch.int32, device="cuda") if tau == 1 else np.asarray(o, dtype=np.int32))
        sol.check_status()
        want = margins_from_weights(sol.col_ptr, sol.row_idx, sol.vals, sol.y, sol.w)
        assert torch.allclose(sol.margin, want, rtol=1e-4, atol=1e-4)
        got.append((sol.w.clone(), sol.margin.clone(), sol.delta.clone()))
    for a, b in zip(*got):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5)      # sums of the same terms in another order


def test_tail_feature_filter_drops_rare_columns():
    """Columns whose count-min estimate is <= tail_feature_freq are removed before training; the rest of the
    run equals the oracle on the data filtered by a NumPy restatement of the same sketch."""
    import math

    from baseline.cpu_ref.ftrl_ref import CountMinRef
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _problem(False, rows=1200, cols=4096, nnz=12)
    freq = 2
    kw = dict(lambda1=0.3, max_pass=3, feature_block_ratio=1.0, seed=3)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(tail_feature_freq=freq, **kw))
    sol.preprocess(off, keys, vals, y)
    hk = keys.cpu().numpy().view(np.uint64)
    uk, inv, cnt = np.unique(hk, return_inverse=True, return_counts=True)
    cm = CountMinRef(max(int(len(uk) * 2.0 / math.log(2)), 64), 2)
    cm.insert(uk, cnt)
    keep = cm.query(uk) > freq
    assert sol.tail_filter_stats["dropped"] == int((~keep).sum()) and 0 < int((~keep).sum()) < len(uk)
    assert np.array_equal(sol.lkeys.cpu().numpy().view(np.uint64), uk[keep])
    sel = keep[inv]
    ho = off.cpu().numpy()
    row_of = np.repeat(np.arange(len(ho) - 1), np.diff(ho))
    foff = np.concatenate([[0], np.cumsum(np.bincount(row_of[sel], minlength=len(ho) - 1))]).astype(np.int64)
    ref = DarlinRef([(foff, hk[sel], vals.cpu().numpy()[sel], y.cpu().numpy())], None, RefConfig(**kw))
    for p, r in zip(sol.run(), ref.run()):
        assert p.objv == pytest.approx(r.objv, rel=2e-3)
    sol.check_status()


def test_darlin_model_dump(tmp_path):
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup
    from parameter_server_b200.utils.modelio import read_model_text

    off, keys, vals, y = _problem(False, rows=600, cols=512)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(lambda1=0.2, max_pass=3))
    sol.preprocess(off, keys, vals, y)
    sol.run()
    path = sol.save_model(str(tmp_path / "m"))
    m = read_model_text(path)
    k, w = sol.model()
    assert len(m) == len(k) > 0
    assert list(m.keys()) == sorted(m.keys())


def _grouped_problem(rows=1200, seed=7):
    """TERAFEA-style keys: the top 10 bits are the feature group.  Group 3 has one feature per example (one
    block), group 5 about six, group 9 about twelve (several blocks each)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    per_group = {3: (1, 40), 5: (6, 300), 9: (12, 700)}       # group -> (features per example, vocabulary)
    cols = []
    for gid, (n, vocab) in per_group.items():
        ids = torch.randint(0, vocab, (rows, n), generator=g, device="cuda")
        cols.append((gid << 54) + ids * 1009 + 17)
    keys = torch.cat(cols, 1).sort(1).values
    keep = torch.ones_like(keys, dtype=torch.bool)
    keep[:, 1:] = keys[:, 1:] != keys[:, :-1]                  # distinct within an example
    off = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    off[1:] = keep.sum(1).cumsum(0)
    flat = keys[keep]
    w = torch.randn(1 << 12, generator=g, device="cuda")
    xw = torch.zeros(rows, device="cuda").index_add_(0, torch.repeat_interleave(torch.arange(rows, device="cuda"), keep.sum(1)),
                                                     w[(flat * 2654435761 >> 7) % (1 << 12)])
    y = torch.where(xw + 0.3 * torch.randn(rows, generator=g, device="cuda") > 0, 1.0, -1.0)
    return off, flat.contiguous(), None, y


@pytest.mark.parametrize("tau", [0, 2])
def test_feature_groups_and_prior_sweeps_match_oracle(tau):
    """Blocks cut group by group from each group's own density and key range; the important group's blocks are
    swept first, with zero delay, in the first pass (the schedule of the reference's CTR job file)."""
    from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
    from parameter_server_b200.parallel.peer import PeerGroup

    off, keys, vals, y = _grouped_problem()
    kw = dict(lambda1=0.2, max_pass=4, feature_block_ratio=0.5, seed=3, max_block_delay=tau, feature_group_bits=10,
              prior_fea_group=(9,), num_iter_for_prior_fea_group=2)
    sol = DarlinSolver(PeerGroup.single(torch.device("cuda", 0)), DarlinConfig(**kw))
    sol.preprocess(off, keys, vals, y)
    prog = sol.run()
    sol.check_status()
    ref = DarlinRef([(off.cpu().numpy(), keys.cpu().numpy().view(np.uint64), None, y.cpu().numpy())], None, RefConfig(**kw))
    rprog = ref.run()
    assert sol.block_group == ref.block_group and sol.block_keys == ref.block_keys
    assert sol.block_group.count(3) == 1 and sol.block_group.count(5) == 3 and sol.block_group.count(9) == 6
    assert len(ref.prior_order()) == 12
    for p, r in zip(prog, rprog):
        assert p.objv == pytest.approx(r.objv, rel=2e-3)
        assert abs(p.nnz_w - r.nnz_w) <= max(3, 0.03 * r.nnz_w)
        assert p.violation == pytest.approx(r.violation, rel=2e-2, abs=1e-3)
