"""What a user of the framework has it do, as cases that can be timed: the online solver, the batch solver, the
neural-network application and the key-value store, each through the entry points that the job runners call.

Kinds of cases
  ftrl    one evaluation interval of an online job on minibatches that are on the device: training steps
          (``FTRLEngine.step``), each step's predictions kept for progressive validation, then a held-out minibatch
          scored with the updated model (``FTRLEngine.predict``)
  stream  the same job as its files are read: pinned minibatches in host memory through ``FTRLTrainer.train``
  darlin  a batch job on data that is on the device: ``DarlinSolver.reset_state`` and ``run``, as a user who tries
          several settings on one preprocessed data set does
  job     the same from the loaded rows on: a new ``DarlinSolver``, ``preprocess`` and ``run``
  nn      ``SGDSolver.run`` of a small or a wide multi-layer perceptron, with the test net's AUC where the job asks for it
  kv      ``DeviceKVVector``: resolve (a worker with new keys), push, pull

Data are the synthetic streams of ``data.synthetic``: Zipf key popularity, planted models.
"""
import math

import torch

from parameter_server_b200 import config
from parameter_server_b200.data.synthetic import ctr_minibatch, mix64, zipf_sparse_matrix
from parameter_server_b200.models.darlin import DarlinConfig, DarlinSolver
from parameter_server_b200.models.ftrl import KEY_U32_HASHED, KEY_U64, DeviceMinibatch, FTRLEngine, FTRLHyper
from parameter_server_b200.models.ftrl_trainer import FTRLTrainer, HostMinibatch
from parameter_server_b200.models.nn import SGDSolver
from parameter_server_b200.parallel.kv_vector import DeviceKVVector
from parameter_server_b200.parallel.peer import PeerGroup

NNZ_CTR = 96          # non-zeros of a row of the click stream (12 groups of 6 to 10 features)


def _pow2(n):
    return 1 << max(int(n) - 1, 0).bit_length()


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # --- online
        # the smallest minibatch in real use: four steps of 500 rows, count rule (the library's default); engine sized
        # as the job runner does for this minibatch
        _ftrl("ftrl_500_rows", rows=500, steps=4),
        # a job file that leaves the solver's defaults alone: count rule, tail-feature filter with frequency 4
        _ftrl("ftrl_10k_rows_tail_filter", rows=10_000, steps=4, tail=4),
        # config/ctr_ftrl.conf: minibatches of 100,000 rows, count rule, no filter, engine sized by the job runner
        _ftrl("ftrl_100k_rows", rows=100_000, steps=2),
        # the default workload of bench.py: sum-of-squares rule, 32-bit feature ids hashed on the device, tables sized for the data
        _ftrl("ftrl_100k_rows_sumsq", rows=100_000, steps=2, rule="sumsq", keys="u32", fitted=True),
        # an ordinary stream from host memory, uint64 keys: what the file readers hand to the trainer
        {"name": "stream_8x10k_rows", "kind": "stream", "rows": 10_000, "steps": 8, "rule": "count", "keys": "u64"},
        # --- batch
        # config/rcv1_l1lr.conf on a data set of rcv1_train's size (20,242 rows): 300 small blocks, no delay
        _darlin("darlin_20k_rows", "darlin", rows=20_242, cols=47_236, per_row=90),
        # the medium batch workload of bench.py (677,399 rows)
        _darlin("darlin_677k_rows", "darlin", rows=677_399, cols=47_236, per_row=90),
        # a click log as config/ctr_l1lr.conf trains it: binary features, hashed keys, 64 wide blocks, bounded delay 8
        _darlin("darlin_clicks_delay_8", "darlin", rows=100_000, delay=8, clicks=True),
        # a whole batch job from the loaded rows on: unique keys, column-major blocks, two passes
        _darlin("job_50k_rows", "job", rows=50_000, cols=1 << 20, per_row=60, passes=2),
        # --- neural network
        # the perceptron of a small table of features: ten minibatches of 256 rows, then the test net's AUC
        _nn("nn_256_rows", rows=256, data=4096, dims=(64, 64, 1), steps=10, test=1000),
        # wide layers (the shapes of bench_gemm.py), full batch
        _nn("nn_8k_rows_wide", rows=8192, data=8192, dims=(1024, 4096, 1024, 1), steps=2),
        # --- key-value store
        # a worker with a new key list: resolve, push and pull of 8 floats a key
        _kv("kv_1m_keys_8_floats", keys=1_000_000, k=8, resolve=True),
    ]


def _ftrl(name, rows, steps, rule="count", keys="u64", tail=0, valued=False, fitted=False):
    return {"name": name, "kind": "ftrl", "rows": rows, "steps": steps, "rule": rule, "keys": keys, "tail": tail, "valued": valued,
            "fitted": fitted}


def _darlin(name, kind, rows, cols=0, per_row=0, delay=0, clicks=False, passes=3, binary=False):
    return {"name": name, "kind": kind, "rows": rows, "cols": cols, "per_row": per_row, "delay": delay, "clicks": clicks,
            "passes": passes, "binary": binary or clicks}


def _nn(name, rows, data, dims, steps, test=0, act="RELU", update="ADAGRAD"):
    return {"name": name, "kind": "nn", "rows": rows, "data": data, "dims": " ".join(map(str, dims)), "steps": steps, "test": test,
            "act": act, "update": update}


def _kv(name, keys, k, resolve):
    return {"name": name, "kind": "kv", "keys": keys, "k": k, "resolve": resolve}


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["ftrl", "ftrl", "ftrl", "stream", "darlin", "darlin", "darlin", "job", "nn", "nn", "kv"])
    if kind == "ftrl":
        rows = log(200, 100_000)
        rule = rng.choice(["count", "count", "sumsq"])
        c = _ftrl("", rows, rng.choice([1, 2, 4]) if rows < 30_000 else 2, rule, rng.choice(["u64", "u32"]),
                  rng.choice([0, 0, 4]) if rule == "count" else 0, rng.random() < 0.25, rows >= 50_000 and rng.random() < 0.5)
    elif kind == "stream":
        c = {"kind": kind, "rows": log(500, 30_000), "steps": rng.randint(4, 10), "rule": rng.choice(["count", "sumsq"]),
             "keys": rng.choice(["u64", "u32"])}
    elif kind == "darlin" and rng.random() < 0.35:
        c = _darlin("", kind, log(10_000, 150_000), delay=rng.choice([0, 4, 8]), clicks=True, passes=2)
    elif kind == "darlin":
        c = _darlin("", kind, log(5_000, 500_000), log(10_000, 200_000), rng.randint(20, 90), rng.choice([0, 0, 8]),
                    passes=rng.randint(2, 3), binary=rng.random() < 0.3)
    elif kind == "job":
        c = _darlin("", kind, log(5_000, 100_000), log(20_000, 4_000_000), rng.randint(20, 80), passes=2, binary=rng.random() < 0.3)
    elif kind == "nn":
        if rng.random() < 0.5:
            rows = rng.randint(16, 256) * 4
            c = _nn("", rows, rows * rng.randint(4, 16), (rng.randint(8, 256), rng.randint(4, 64) * 4, 1), rng.randint(5, 10),
                    rng.choice([0, log(500, 20_000)]), rng.choice(["RELU", "SIGMOID", "SCALED_TANH"]), rng.choice(["ADAGRAD", "NORMAL"]))
        else:
            rows = rng.randint(512, 2048) * 4
            c = _nn("", rows, rows, (rng.randint(256, 1024), rng.randint(64, 512) * 8, rng.randint(32, 256) * 4, 1), 2, 0,
                    rng.choice(["RELU", "SCALED_TANH"]), "ADAGRAD")
    else:
        k = rng.choice([1, 3, 8, 64])
        c = _kv("", log(1_000, 10_000_000 // max(k, 4)), k, rng.random() < 0.5)
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ what a program has in hand before the call
def prepare(case, seed):
    return {"ftrl": _prepare_ftrl, "stream": _prepare_stream, "darlin": _prepare_darlin, "job": _prepare_darlin, "nn": _prepare_nn,
            "kv": _prepare_kv}[case["kind"]](case, int(seed))


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _minibatch(rows, keys, seed, valued=False):
    off, key, y, ids = ctr_minibatch(rows, seed=seed, device=_device(), return_ids=True)
    vals = None
    if valued:
        g = torch.Generator(device=off.device).manual_seed(seed)
        vals = torch.rand(key.numel(), generator=g, device=off.device) + 0.5
    if keys == "u32":
        return DeviceMinibatch(off.to(torch.int32), ids, y, vals, KEY_U32_HASHED)
    return DeviceMinibatch(off, key, y, vals, KEY_U64)


def _engine(case):
    """An engine as the job runner sizes it for the minibatch (256 non-zeros a row at most), or fitted to the data."""
    rows = case["rows"]
    # gradients are summed over a minibatch: under the count rule a step size that suits its size, under the sum of squares the usual one
    alpha = 0.1 if case["rule"] == "sumsq" else 0.3 / rows ** 0.5
    hyper = FTRLHyper(alpha=alpha, beta=1.0, lambda1=1.0, lambda2=0.1, rule=case["rule"], tail_feature_freq=case.get("tail", 0),
                      countmin_n=10 ** 8 if rows >= 50_000 else 10 ** 7)
    max_nnz, local = rows * 256, min(rows * 256, 1 << 24)
    if case.get("fitted"):
        max_nnz, local = rows * (NNZ_CTR + 2), _pow2(rows * NNZ_CTR * 0.4)
    return FTRLEngine(PeerGroup.single(_device()), hyper, table_capacity=1 << 26 if rows >= 50_000 else 1 << 23, max_rows=rows,
                      max_nnz=max_nnz, local_capacity=local)


def _prepare_ftrl(case, seed):
    eng = _engine(case)
    make = [_minibatch(case["rows"], case["keys"], 1000 * seed + i, case["valued"]) for i in range(case["steps"] + 2)]
    held = _minibatch(max(case["rows"] // 4, 1), case["keys"], 1000 * seed + 999, case["valued"])
    for mb in make[:2]:                      # the job has been running: the model holds weights
        eng.step(mb)
    eng.check_status()
    return {"case": case, "engine": eng, "train": make[2:], "held": held}


def _prepare_stream(case, seed):
    eng = _engine(case)
    host = []
    for i in range(case["steps"]):
        b = _minibatch(case["rows"], case["keys"], 1000 * seed + i)
        host.append(HostMinibatch(b.offsets.cpu(), b.keys.cpu(), b.y.cpu(), None, b.key_mode).pin())
    trainer = FTRLTrainer(eng)
    trainer.train(host[:1])
    return {"case": case, "engine": eng, "trainer": trainer, "batches": host}


def _prepare_darlin(case, seed):
    dev = _device()
    if case["clicks"]:
        off, keys, y = ctr_minibatch(case["rows"], seed=seed, device=dev, key_space_log2=32, zipf_s=1.05, groups=12, feats_lo=8, feats_hi=12,
                                     bias=0.0, wstar_frac=0.005, wstar_std=1.0)
        vals = None
        conf = DarlinConfig(lambda1=4.0, eta=1.0, delta_init=1.0, delta_max=5.0, kkt_ratio=10.0, feature_block_ratio=63.5 / 120)
    else:
        off, keys, vals, y, _ = zipf_sparse_matrix(case["rows"], case["cols"], case["per_row"], seed=seed, device=dev, zipf_s=1.0,
                                                   wstar_frac=0.02, noise=0.3, binary=case["binary"])
        conf = DarlinConfig(lambda1=1.0, eta=1.0, delta_init=5.0, delta_max=10.0, kkt_ratio=100.0, feature_block_ratio=4.0)
    conf.max_pass, conf.epsilon, conf.max_block_delay = case["passes"], 0.0, case["delay"]
    state = {"case": case, "conf": conf, "rows": (off, keys, vals, y)}
    if case["kind"] == "darlin":
        state["solver"] = DarlinSolver(PeerGroup.single(dev), conf)
        state["solver"].preprocess(off, keys, vals, y)
        del state["rows"]
    return state


_NET = """neural_network {
  train { name: "train"
    layer { type: DATA name: "data" out: "x" out: "y" minibatch_size: %d }
%s    layer { type: LOGISTIC_LOSS name: "loss" in: "s" in: "y" }
  }
%s  solver { type: SGD update: %s lr { alpha: %g beta: 1 } max_iteration: %d display: 1000000 validation: %d }
}"""


def _prepare_nn(case, seed):
    dev, dims = _device(), [int(d) for d in case["dims"].split()]
    layers = ""
    for i, d in enumerate(dims[1:]):
        last = i == len(dims) - 2
        layers += '    layer { type: FULLY_CONNECTED name: "fc%d" in: "%s" out: "%s" size: %d activation { type: %s } }\n' % (
            i, "x" if i == 0 else "h%d" % (i - 1), "s" if last else "h%d" % i, d, "IDENTITY" if last else case["act"])
    test = ""
    if case["test"]:
        test = '  test { name: "test"\n    layer { type: DATA name: "tdata" out: "x" out: "y" }\n%s' \
               '    layer { type: AUC name: "auc" in: "s" in: "y" }\n  }\n' % layers
    batch = 0 if case["rows"] == case["data"] else case["rows"]
    text = _NET % (batch, layers, test, case["update"], (5e-3 if case["rows"] <= 1024 else 1e-3) if case["update"] == "ADAGRAD" else 1e-3, case["steps"],
                   case["steps"] if case["test"] else 0)
    solver = SGDSolver(config.parse_app_config(text).neural_network, PeerGroup.single(dev))
    g = torch.Generator(device=dev).manual_seed(seed)
    w = torch.randn(dims[0], 8, generator=g, device=dev) / dims[0] ** 0.5

    def table(n):
        x = torch.randn(n, dims[0], generator=g, device=dev)
        return x, torch.where(torch.tanh(x @ w).sum(1) > 0, 1.0, -1.0)

    solver.train.layer("data").set_data(*table(case["data"]))
    if case["test"]:
        solver.test.layer("tdata").set_data(*table(case["test"]))
    return {"case": case, "solver": solver}


def _prepare_kv(case, seed):
    dev, n = _device(), case["keys"]
    g = torch.Generator(device=dev).manual_seed(seed)
    server = mix64(torch.randperm(2 * n, generator=g, device=dev) + (seed << 33))        # distinct hashed keys
    kv = DeviceKVVector(PeerGroup.single(dev), k=case["k"])
    kv.set_keys(kv.merge_keys(server.contiguous()))
    mine = server[torch.randperm(2 * n, generator=g, device=dev)[:n]]                    # half of them are this worker's
    mine = ((mine ^ -(1 << 63)).sort().values ^ -(1 << 63)).contiguous()                 # key lists are ordered
    vals = torch.randn(n, case["k"], generator=g, device=dev)
    return {"case": case, "kv": kv, "keys": mine, "vals": vals, "where": None if case["resolve"] else kv.resolve(mine)}


# ------------------------------------------------------------------ one pass
def run(state):
    return {"ftrl": _run_ftrl, "stream": _run_stream, "darlin": _run_darlin, "job": _run_job, "nn": _run_nn,
            "kv": _run_kv}[state["case"]["kind"]](state)


def _run_ftrl(state):
    eng, margins = state["engine"], []
    for mb in state["train"]:
        eng.step(mb)
        margins.append(eng.xw[: mb.rows].clone())
    return {"margins": margins, "scores": eng.predict(state["held"]), "statistics": eng.stats}


def _run_stream(state):
    losses = state["trainer"].train(state["batches"])
    return {"losses": losses, "margins": state["engine"].xw[: state["case"]["rows"]], "statistics": state["engine"].stats}


def _whole(values, length):
    """The values of the columns that the data have, in a vector as long as the feature space (or more than it can have)."""
    if values.numel() > length:
        raise ValueError("more columns than the vector holds")
    return torch.nn.functional.pad(values, (0, length - values.numel()))


def _solver_results(solver, case):
    return {"objective": [p.objv for p in solver.progress], "violation": [p.violation for p in solver.progress],
            "w": _whole(solver.w, _columns(case)), "margin": solver.margin}


def _columns(case):
    return case["rows"] * 60 if case["clicks"] else case["cols"]


def _run_darlin(state):
    solver = state["solver"]
    solver.reset_state()
    solver.run()
    return _solver_results(solver, state["case"])


def _run_job(state):
    solver = DarlinSolver(PeerGroup.single(_device()), state["conf"])
    solver.preprocess(*state["rows"])
    solver.run()
    n = _columns(state["case"])
    return {"keys": _whole(solver.lkeys, n), "columns": _whole(solver.col_ptr, n + 1), **_solver_results(solver, state["case"])}


def _run_nn(state):
    solver, steps = state["solver"], state["case"]["steps"]
    solver.run(verbose=False)
    last = solver.history[-steps:]
    out = {"losses": [h["loss"] for h in last], "weights": [p.value for p in solver.train.models()],
           "gradients": [p.gradient for p in solver.train.models()]}
    if state["case"]["test"]:
        out["auc"] = last[-1]["test_auc"]
    return out


def _run_kv(state):
    kv = state["kv"]
    owner, slot = state["where"] or kv.resolve(state["keys"])
    kv.push(owner, slot, state["vals"])
    return {"slot": slot, "pulled": kv.pull(owner, slot), "values": kv.local_values}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("ftrl", "stream"):
        rows, steps = case["rows"], case["steps"]
        nnz = rows * NNZ_CTR
        inputs = nnz * (8 if case["keys"] == "u64" else 4) + rows * 12 + (4 * nnz if case.get("valued") else 0)
        state = 0.3 * nnz * 64        # about 0.3 distinct keys a non-zero, their 32 bytes of state read and written
        score = 0 if kind == "stream" else 0.25 * (inputs + 0.5 * state)
        return {"bytes": steps * (inputs + state + 4 * rows) + score, "flops": 4.0 * nnz * (steps + 0.25)}
    if kind in ("darlin", "job"):
        rows = case["rows"]
        nnz = rows * 120 if case["clicks"] else rows * case["per_row"] * 0.83        # repeated columns of a row are merged
        one = nnz * (4 if case["binary"] else 8) + 16 * rows                         # a pass reads the matrix once
        made = nnz * (8 + (0 if case["binary"] else 8) + 4) if kind == "job" else 0  # keys and values in, columns out
        return {"bytes": case["passes"] * one + made, "flops": 12.0 * nnz * case["passes"]}
    if kind == "nn":
        dims, rows = [int(d) for d in case["dims"].split()], case["rows"]
        weights = [a * b for a, b in zip(dims, dims[1:])]
        step = 2.0 * rows * (3 * sum(weights) - weights[0])                          # no gradient flows into the data
        data = 4.0 * (rows * (dims[0] + 2 * sum(dims[1:])) + 5 * sum(weights))
        return {"bytes": case["steps"] * data + 4.0 * case["test"] * dims[0],
                "flops": case["steps"] * step + 2.0 * case["test"] * sum(weights)}
    n, k = case["keys"], case["k"]
    # push: values in, rows read and written; pull: rows read, values out; resolve: keys in, the shard's keys once, places out
    return {"bytes": n * k * 20.0 + 8.0 * n + (n * 8.0 + 2 * n * 8.0 + 8.0 * n if case["resolve"] else 0.0), "flops": float(n * k)}


def tolerance(case):
    """About four times the largest difference seen between a pass and the same pass with its rows in another order (of the
    nn cases with minibatches: with starting weights that differ in the last bit), over several seeds.

    Online: 2e-7 of the 2-norm, 8e-7 of one value (sums in fp32).  Batch: 1.2e-5 and 3.4e-4; on the click log a feature with
    few examples may end on the other side of the filter's threshold in a few columns, 2.7e-4 and 0.7.  Networks: an
    activation that differs in the last bit may be rounded to another TF32 value, 2.9e-4 and 1.3e-3 of the small nets' last
    gradients, 2.6e-3 and 0.12 of the wide nets' second ones (the first update leaves them near zero)."""
    if case["kind"] == "nn":
        return {"rel": 1.2e-3, "max": 1e-2} if case["rows"] <= 1024 else {"rel": 1e-2, "max": 0.4}
    if case["kind"] in ("darlin", "job"):
        return {"rel": 1.2e-3, "max": 0.99} if case["clicks"] else {"rel": 5e-5, "max": 2e-3}
    return {"rel": 2e-6, "max": 2e-5} if case["kind"] in ("ftrl", "stream") else {"rel": 1e-6}
