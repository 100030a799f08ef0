"""Dense-layer operators of the neural-network app on the sm_100a kernels
(``csrc/gemm_tcgen05.cu``): TF32 tcgen05 GEMM with fused activation, tiled transpose,
activation backward, logistic loss, SGD / AdaGrad update, column normalisation."""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from . import _native as N

ACT = {"IDENTITY": 0, "RELU": 1, "SCALED_TANH": 2, "SIGMOID": 3}
_status = {}


def _status_for(dev) -> torch.Tensor:
    k = (dev.type, dev.index)
    if k not in _status:
        _status[k] = torch.zeros(8, dtype=torch.int32, device=dev)
    return _status[k]


def check_status(dev) -> None:
    st = _status_for(dev).tolist()
    if st[0] != 0:
        _status_for(dev).zero_()
        raise RuntimeError(f"GEMM kernel gave up waiting (code {st[0]}, tile {st[1]},{st[2] - 100})")


def _written(t: torch.Tensor) -> None:
    """A kernel wrote to a tensor of the caller's: its version counter says so, as after PyTorch's in-place operators."""
    if not t.is_inference():
        torch.autograd.graph.increment_version(t)


def gemm_tn(a: torch.Tensor, b: torch.Tensor, act: str = "IDENTITY", out: Optional[torch.Tensor] = None,
            pad_k: bool = False, out_t: Optional[torch.Tensor] = None, variant: int = 0) -> torch.Tensor:
    """``act(a @ b.T)`` for row-major fp32 ``a`` [M,K] and ``b`` [N,K] on the tcgen05 tensor cores (TF32).  ``out_t``
    (contiguous [N,M]) receives the transposed result too; ``variant``: 0 = kernel by size, 1 = one tile per thread
    block, 2 = pairs of thread blocks, 3 = a K of at most four."""
    assert a.is_cuda and a.dtype == torch.float32 and b.dtype == torch.float32 and a.shape[1] == b.shape[1]
    assert a.stride(1) == 1 and b.stride(1) == 1
    M, K = a.shape
    Nn = b.shape[0]
    if pad_k and K < 4 and variant == 0:
        variant = 3                                  # reads the operands element by element
    elif pad_k and K % 4:
        # TMA needs row strides that are multiples of 16 bytes: zero-pad the contraction dimension
        kp = (K + 3) // 4 * 4
        a = torch.nn.functional.pad(a, (0, kp - K))
        b = torch.nn.functional.pad(b, (0, kp - K))
        K = kp
    if out is None:
        out = torch.empty((M, Nn), dtype=torch.float32, device=a.device)
    else:
        _written(out)
    if out_t is not None:
        assert out_t.shape == (Nn, M) and out_t.is_contiguous() and out_t.dtype == torch.float32
    rc = N.lib().psb_gemm_tn_tf32(N.ptr(a), N.ptr(b), N.ptr(out), N.ptr(out_t), M, Nn, K, a.stride(0), b.stride(0), out.stride(0),
                                  ACT[act], variant, N.ptr(_status_for(a.device)), N.stream_ptr())
    if rc == 1:
        raise ValueError("gemm_tn needs 16-byte aligned operands whose row strides are multiples of 4 floats")
    N.check(rc, "gemm_tn_tf32")
    return out


def transpose(x: torch.Tensor) -> torch.Tensor:
    assert x.is_cuda and x.dtype == torch.float32 and x.is_contiguous() and x.dim() == 2
    out = torch.empty((x.shape[1], x.shape[0]), dtype=torch.float32, device=x.device)
    N.check(N.lib().psb_transpose(N.ptr(x), N.ptr(out), x.shape[0], x.shape[1], N.stream_ptr()), "transpose")
    return out


def act_backward(g: torch.Tensor, y: torch.Tensor, act: str) -> torch.Tensor:
    z = torch.empty_like(g)
    N.check(N.lib().psb_act_backward(N.ptr(g), N.ptr(y), N.ptr(z), C.c_size_t(g.numel()), ACT[act], N.stream_ptr()), "act_backward")
    return z


def act_backward_t(g: torch.Tensor, y: torch.Tensor, act: str, want_z: bool = True):
    """(``g ∘ act'(y)`` or None, its transpose) of two contiguous [rows, cols] matrices in one pass over them."""
    assert g.is_contiguous() and y.is_contiguous() and g.shape == y.shape and g.dim() == 2
    assert g.is_cuda and y.is_cuda and g.dtype == y.dtype == torch.float32
    z = torch.empty_like(g) if want_z else None
    zt = torch.empty((g.shape[1], g.shape[0]), dtype=torch.float32, device=g.device)
    N.check(N.lib().psb_act_backward_t(N.ptr(g), N.ptr(y), N.ptr(z), N.ptr(zt), g.shape[0], g.shape[1], ACT[act], N.stream_ptr()),
            "act_backward_t")
    return z, zt


def gather_minibatch(x: torch.Tensor, y: torch.Tensor, sel: torch.Tensor, want_t: bool):
    """(``x[sel]``, its transpose or None, ``y[sel]``) for contiguous float32 ``x`` [n, cols], ``y`` [n] and device
    int64 row numbers ``sel`` (all inside x), in one launch."""
    assert can_gather_minibatch(x, y, sel.numel()) and sel.is_cuda and sel.is_contiguous() and sel.dtype == torch.int64
    return gather_rows(x, y, sel, want_t)


def can_gather_minibatch(x: torch.Tensor, y: torch.Tensor, b: int) -> bool:
    """The data that :func:`gather_minibatch` takes: one label per row (labels of several columns are indexed)."""
    return (x.is_cuda and y.is_cuda and x.dtype == y.dtype == torch.float32 and x.dim() == 2 and y.dim() == 1
            and y.numel() == x.shape[0] and x.numel() > 0 and x.is_contiguous() and y.is_contiguous() and 0 < b <= 32 * 65535)


def gather_rows(x: torch.Tensor, y: torch.Tensor, sel: torch.Tensor, want_t: bool):
    """:func:`gather_minibatch` of data that was found fit for it."""
    b, cols = sel.numel(), x.shape[1]
    xb = torch.empty((b, cols), dtype=torch.float32, device=x.device)
    yb = torch.empty(b, dtype=torch.float32, device=x.device)
    xbt = torch.empty((cols, b), dtype=torch.float32, device=x.device) if want_t else None
    N.check(N.lib().psb_gather_minibatch(N.ptr(x), N.ptr(y), N.ptr(sel), b, cols, N.ptr(xb), N.ptr(xbt), N.ptr(yb), N.stream_ptr()),
            "gather_minibatch")
    return xb, xbt, yb


def logistic_loss(x: torch.Tensor, y: torch.Tensor, want_grad: bool = True):
    """(Σ log(1+e^{-x·y}) as a 1-element fp64 tensor, −y/(1+e^{x·y}) or None)."""
    loss = torch.zeros(1, dtype=torch.float64, device=x.device)
    grad = torch.empty_like(x) if want_grad else None
    N.check(N.lib().psb_logistic_loss(N.ptr(x), N.ptr(y), N.ptr(grad), C.c_size_t(x.numel()), N.ptr(loss), N.stream_ptr()), "logistic_loss")
    return loss, grad


def sgd_update(w: torch.Tensor, g: torch.Tensor, h: Optional[torch.Tensor], alpha: float, beta: float, it: int) -> None:
    N.check(N.lib().psb_sgd_update(N.ptr(w), N.ptr(g), N.ptr(h), C.c_size_t(w.numel()), C.c_float(alpha), C.c_float(beta),
                                   C.c_float(float(it)), 0 if h is None else 1, N.stream_ptr()), "sgd_update")


def col_normalize(x: torch.Tensor) -> None:
    assert x.is_contiguous() and x.dim() == 2
    N.check(N.lib().psb_col_normalize(N.ptr(x), x.shape[0], x.shape[1], N.stream_ptr()), "col_normalize")
    _written(x)


def sparse_fc_forward(off: torch.Tensor, idx: torch.Tensor, vals: Optional[torch.Tensor], w: torch.Tensor, act: str = "IDENTITY") -> torch.Tensor:
    """Y = act(X·W) for CSR X (int64 offsets, int32 column ids, float32 values or None = ones) and W [in, out]
    (out a multiple of 4): the embedding-bag sum of the sparse fully connected layer."""
    rows, (in_dim, out_dim) = off.numel() - 1, w.shape
    y = torch.empty((rows, out_dim), dtype=torch.float32, device=w.device)
    N.check(N.lib().psb_spfc_forward(N.ptr(off), N.ptr(idx), N.ptr(vals), N.ptr(w), N.ptr(y), rows, in_dim, out_dim, ACT[act],
                                     N.ptr(_status_for(w.device)), N.stream_ptr()), "spfc_forward")
    return y


def sparse_fc_backward(off: torch.Tensor, idx: torch.Tensor, vals: Optional[torch.Tensor], y: torch.Tensor, gy: torch.Tensor,
                       in_dim: int, act: str = "IDENTITY") -> torch.Tensor:
    """Wg = Xᵀ·(dY ∘ act'(Y)) as [in, out]."""
    rows, out_dim = y.shape
    wg = torch.zeros((in_dim, out_dim), dtype=torch.float32, device=y.device)
    N.check(N.lib().psb_spfc_backward(N.ptr(off), N.ptr(idx), N.ptr(vals), N.ptr(y), N.ptr(gy.contiguous()), N.ptr(wg), rows, in_dim,
                                      out_dim, ACT[act], N.stream_ptr()), "spfc_backward")
    return wg
