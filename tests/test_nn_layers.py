"""Dense layers of the neural-network application on the CPU: what they hand to the operators and what they keep, with
PyTorch restatements of the operators."""
import pytest
import torch

from parameter_server_b200 import config as cfg
from parameter_server_b200.models.nn import SGDSolver
from parameter_server_b200.ops import dense
from parameter_server_b200.parallel.peer import PeerGroup

NET = '''
neural_network {
  train { name: "train"
    layer { type: DATA name: "data" out: "x" out: "y" minibatch_size: 0 }
    layer { type: FULLY_CONNECTED name: "fc1" in: "x" out: "h" size: %d activation { type: RELU } }
    layer { type: FULLY_CONNECTED name: "fc2" in: "h" out: "g" size: %d activation { type: RELU } }
    layer { type: FULLY_CONNECTED name: "fc3" in: "g" out: "s" size: 1 activation { type: IDENTITY } }
    layer { type: LOGISTIC_LOSS name: "loss" in: "s" in: "y" }
  }
  solver { type: SGD update: NORMAL lr { alpha: 0.1 beta: 1 } max_iteration: 1 display: 50 }
}
'''


@pytest.fixture
def ops(monkeypatch):
    """The operators in PyTorch, with their demands on the operands; records the transposes that a GEMM was asked for."""
    asked = []

    def gemm_tn(a, b, act="IDENTITY", out=None, pad_k=False, out_t=None, variant=0):
        assert a.stride(1) == 1 and b.stride(1) == 1 and a.dtype == b.dtype == torch.float32
        if not (pad_k and a.shape[1] % 4):
            for t in (a, b):
                if t.data_ptr() % 16 or t.stride(0) % 4:
                    raise ValueError("gemm_tn needs 16-byte aligned operands whose row strides are multiples of 4 floats")
        r = a @ b.T
        r = torch.relu(r) if act == "RELU" else r
        if out_t is not None:
            asked.append(out_t.numel() * 4)
            out_t.copy_(r.T)
        return r

    def act_backward_t(g, y, act, want_z=True):
        z = g * (y > 0) if act == "RELU" else g.clone()
        return (z if want_z else None), z.T.contiguous()

    def logistic_loss(x, y, want_grad=True):
        m = (x * y).double()
        return torch.nn.functional.softplus(-m).sum().reshape(1), (-y * torch.sigmoid(-m)).float()

    def sgd_update(w, g, h, alpha, beta, it):
        w -= alpha * g / (beta + it ** 0.5)

    for f in (gemm_tn, act_backward_t, logistic_loss, sgd_update):
        monkeypatch.setattr(dense, f.__name__, f)
    monkeypatch.setattr(dense, "transpose", lambda x: x.T.clone(memory_format=torch.contiguous_format))
    monkeypatch.setattr(dense, "check_status", lambda dev: None)
    return asked


def _net(sizes=(12, 8), rows=16, cols=6):
    sol = SGDSolver(cfg.parse_app_config(NET % sizes).neural_network, PeerGroup.single(torch.device("cpu")))
    g = torch.Generator().manual_seed(3)
    X = torch.randn(rows, cols, generator=g)
    y = torch.where(torch.rand(rows, generator=g) < 0.5, 1.0, -1.0)
    sol.train.layer("data").set_data(X, y, normalize=False)
    return sol, X, y


def _check_gradients(sol, X, y):
    ws = [sol.train.layer(n).model.value.detach().clone().double().requires_grad_(True) for n in ("fc1", "fc2", "fc3")]
    h = X.double()
    for w in ws[:2]:
        h = torch.relu(h @ w.T)
    torch.nn.functional.softplus(-(h @ ws[2].T).reshape(-1) * y).sum().backward()
    for n, w in zip(("fc1", "fc2", "fc3"), ws):
        torch.testing.assert_close(sol.train.layer(n).model.gradient.double(), w.grad, rtol=1e-4, atol=1e-5)


def test_gradients(ops):
    sol, X, y = _net()
    sol.train.forward()
    sol.train.backward()
    _check_gradients(sol, X, y)
    assert len(ops) == 2 and all(e.transposed is None for e in sol.train.edges.values()) and sol.train.kept_bytes == 0


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_one_feature_from_a_view_of_any_alignment(ops, offset):
    """A data set of one column whose rows start inside another tensor is laid out like its transpose, but not aligned."""
    sol, X, y = _net(cols=1)
    buf = torch.cat([torch.zeros(offset, 1), X])
    sol.train.layer("data").set_data(buf[offset:], y, normalize=False)
    sol.train.forward()
    sol.train.backward()
    _check_gradients(sol, X, y)


def test_training_inside_inference_mode(ops):
    """Gradients are the layers' own, so a net trains where autograd is off; such tensors have no version counter."""
    sol, X, y = _net()
    with torch.inference_mode():
        sol.train.layer("data").set_data(X.clone(), y.clone(), normalize=False)
        sol.train.forward()
        sol.train.backward()
        got = [sol.train.layer(n).model.gradient.clone() for n in ("fc1", "fc2", "fc3")]
        loss = sol.step(0)
    sol2, _, _ = _net()
    sol2.train.forward()
    sol2.train.backward()
    for n, g in zip(("fc1", "fc2", "fc3"), got):
        torch.testing.assert_close(g, sol2.train.layer(n).model.gradient)
    assert loss > 0


def test_kept_transposes_are_bounded(ops, monkeypatch):
    """Transposes wait for the backward pass up to a bound; what is beyond it is transposed when it is needed."""
    from parameter_server_b200.models import nn

    monkeypatch.setattr(nn, "KEPT_TRANSPOSE_BYTES", 16 * 8 * 4 + 100)
    sol, X, y = _net(sizes=(12, 8))
    for _ in range(2):                       # the bound holds for a step, not for the life of the net
        ops.clear()
        sol.train.forward()
        assert sum(t[2].numel() * 4 for t in (e.transposed for e in sol.train.edges.values()) if t is not None) <= 16 * 8 * 4 + 100
        assert ops == [16 * 8 * 4]           # the first hidden layer's transpose is too large, the second's fits
        sol.train.backward()
        _check_gradients(sol, X, y)
    sol.train.forward()                      # ... and holds when no backward pass came between
    sol.train.forward()
    assert ops == [16 * 8 * 4] * 3


def test_slope_and_transpose_take_float32_on_the_device_only():
    """As the transpose that they replace did; the kernel would read other data as floats."""
    g = torch.ones(4, 4)
    for a, b in ((g.double(), g.double()), (g, g.double()), (g.half(), g.half()), (g, g)):
        with pytest.raises(AssertionError):
            dense.act_backward_t(a, b, "RELU")
