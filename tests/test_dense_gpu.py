"""tcgen05 TF32 GEMM and the NN elementwise kernels against plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref_act(x, act):
    if act == "RELU":
        return torch.relu(x)
    if act == "SCALED_TANH":
        return 1.7159 * torch.tanh(2.0 / 3.0 * x)
    if act == "SIGMOID":
        return torch.sigmoid(x)
    return x


@pytest.mark.parametrize("M,N,K", [(128, 128, 32), (128, 128, 256), (256, 384, 96), (200, 130, 72), (1000, 520, 1024), (64, 8, 4),
                                   # many tiles: persistent CTA pairs (several tiles per pair, ragged edges, short K)
                                   (2048, 4096, 512), (1925, 2563, 260), (4096, 4224, 36), (9000, 2100, 64)])
@pytest.mark.parametrize("act", ["IDENTITY", "RELU", "SCALED_TANH"])
def test_gemm_tn_matches_fp32(M, N, K, act):
    from parameter_server_b200.ops import dense

    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn(M, K, generator=g, device="cuda")
    b = torch.randn(N, K, generator=g, device="cuda") / K ** 0.5
    out = dense.gemm_tn(a, b, act)
    torch.cuda.synchronize()
    dense.check_status(a.device)
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    ref = _ref_act(a.double() @ b.double().T, act).float()
    torch.backends.cuda.matmul.allow_tf32 = prev
    err = (out - ref).abs().max().item()
    assert err < 2e-2 * max(1.0, ref.abs().max().item()), err        # TF32: 10-bit mantissa
    assert (out - ref).abs().mean().item() < 2e-3


@pytest.mark.parametrize("M,N,K,variant", [
    (256, 256, 32, 2), (257, 255, 36, 2), (5, 2000, 64, 2), (130, 120, 200, 2), (5000, 1300, 132, 2),     # CTA pairs
    (128, 128, 28, 1), (129, 127, 220, 1), (7, 9, 700, 1),                                                # one tile per CTA
    (1, 1000, 2052, 0), (8, 32, 32, 0), (9, 33, 64, 0), (3, 130, 36, 0), (8, 31, 5000, 0), (1, 1, 8, 0),       # few rows
    (100, 203, 1, 0), (37, 1, 3, 0), (1, 64, 2, 0), (1030, 5, 4, 0)])                                     # K of at most four
@pytest.mark.parametrize("act", ["IDENTITY", "SIGMOID"])
def test_gemm_kernels_and_transposed_result(M, N, K, variant, act):
    """Every kernel at the edges of its tiles against fp64: TF32 operands carry a relative error below 2^-10 each, so
    an element is off by at most 2^-9 of the sum of its terms' magnitudes (plus the fp32 sums, far below)."""
    from parameter_server_b200.ops import dense

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda") / K ** 0.5
    t = torch.full((N, M), float("nan"), device="cuda")
    out = dense.gemm_tn(a, b, act, pad_k=True, out_t=t, variant=variant)
    torch.cuda.synchronize()
    dense.check_status(a.device)
    ref, bound = a.double() @ b.double().T, (a.double().abs() @ b.double().abs().T) / 512 + 1e-5
    if act == "SIGMOID":
        ref, bound = torch.sigmoid(ref), bound / 4 + 1e-5
    assert bool(((out.double() - ref).abs() <= bound).all())
    assert torch.equal(t, out.T)


@pytest.mark.parametrize("M,N,K", [(1, 1024, 8192), (8, 96, 260), (700, 900, 520)])
def test_kernels_agree_to_the_bit(M, N, K):
    """Which kernel a product's size selects does not change its sums: the tile kernels add in the same order, and the
    outer product cuts its operands to TF32 as the tensor cores do."""
    from parameter_server_b200.ops import dense

    a, b = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda")
    assert torch.equal(dense.gemm_tn(a, b), dense.gemm_tn(a, b, variant=2))
    a, b = torch.nn.functional.pad(a[:, :1], (0, 3)), torch.nn.functional.pad(b[:, :1], (0, 3))
    assert torch.equal(dense.gemm_tn(a, b, variant=3), dense.gemm_tn(a, b, variant=2))


@pytest.mark.parametrize("rows,cols", [(1, 1), (64, 64), (63, 65), (128, 4), (70, 200), (333, 77)])
@pytest.mark.parametrize("act", ["RELU", "SCALED_TANH", "SIGMOID"])
def test_act_backward_with_transpose(rows, cols, act):
    from parameter_server_b200.ops import dense

    y, g = torch.rand(rows, cols, device="cuda") - 0.3, torch.randn(rows, cols, device="cuda")
    want = dense.act_backward(g, y, act)
    z, zt = dense.act_backward_t(g, y, act)
    assert torch.equal(z, want) and torch.equal(zt, want.T)
    z, zt = dense.act_backward_t(g, y, act, want_z=False)
    assert z is None and torch.equal(zt, want.T)


def test_gemm_strided_views_and_repeat():
    from parameter_server_b200.ops import dense

    big = torch.randn(300, 256, device="cuda")
    a, b = big[:260, :128], big[4:132, 128:]            # row stride 256, offsets keep 16-byte alignment
    o1 = dense.gemm_tn(a, b)
    o2 = dense.gemm_tn(a, b)
    torch.cuda.synchronize()
    assert torch.equal(o1, o2)
    assert (o1 - a @ b.T).abs().max().item() < 0.2
    with pytest.raises(ValueError):
        dense.gemm_tn(big[:, :127], big[:, 1:128])


def test_elementwise_kernels():
    from parameter_server_b200.ops import dense

    x = torch.randn(333, 77, device="cuda")
    assert torch.equal(dense.transpose(x), x.T.contiguous())
    g = torch.randn_like(x)
    for act in ("IDENTITY", "RELU", "SCALED_TANH", "SIGMOID"):
        xr = x.clone().requires_grad_(True)
        y = _ref_act(xr, act)
        y.backward(g)
        z = dense.act_backward(g, y.detach(), act)
        torch.testing.assert_close(z, xr.grad, rtol=1e-4, atol=1e-5)
    yl = torch.where(torch.rand(1000, device="cuda") < 0.5, 1.0, -1.0)
    s = torch.randn(1000, device="cuda")
    loss, grad = dense.logistic_loss(s, yl)
    sr = s.clone().requires_grad_(True)
    ref = torch.nn.functional.softplus(-sr * yl).sum()
    ref.backward()
    assert loss.item() == pytest.approx(ref.item(), rel=1e-5)
    torch.testing.assert_close(grad, sr.grad, rtol=1e-4, atol=1e-6)
    w, gw, h = torch.randn(500, device="cuda"), torch.randn(500, device="cuda"), torch.zeros(500, device="cuda")
    w0 = w.clone()
    dense.sgd_update(w, gw, None, 0.1, 1.0, 9)
    torch.testing.assert_close(w, w0 - 0.1 * gw / (1.0 + 3.0))
    w1 = w.clone()
    dense.sgd_update(w, gw, h, 0.1, 1.0, 9)
    torch.testing.assert_close(h, gw * gw)
    torch.testing.assert_close(w, w1 - 0.1 * gw / (1.0 + gw.abs()))
    m = torch.randn(200, 9, device="cuda") * 3 + 1
    dense.col_normalize(m)
    torch.testing.assert_close(m.mean(0), torch.zeros(9, device="cuda"), atol=1e-5, rtol=0)
    torch.testing.assert_close(m.norm(dim=0), torch.full((9,), 200 ** 0.5, device="cuda"), rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("rows,cols,b", [(1, 1, 1), (100, 3, 37), (500, 64, 256), (70, 33, 33), (4000, 129, 100)])
def test_gather_minibatch(rows, cols, b):
    from parameter_server_b200.ops import dense

    g = torch.Generator(device="cuda").manual_seed(rows)
    x, y = torch.randn(rows, cols, generator=g, device="cuda"), torch.randn(rows, generator=g, device="cuda")
    sel = torch.randint(0, rows, (b,), generator=g, device="cuda")
    for want_t in (True, False):
        xb, xbt, yb = dense.gather_minibatch(x, y, sel, want_t)
        assert torch.equal(xb, x[sel]) and torch.equal(yb, y[sel])
        assert torch.equal(xbt, x[sel].T) if want_t else xbt is None


@pytest.mark.parametrize("rows,cols", [(1, 5), (64, 64), (65, 130), (1000, 4), (2048, 512), (1023, 1026), (4, 300_000)])
def test_transpose_sizes(rows, cols):
    from parameter_server_b200.ops import dense

    x = torch.randn(rows, cols, device="cuda")
    assert torch.equal(dense.transpose(x), x.T)


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 400_001])
@pytest.mark.parametrize("adagrad", [False, True])
def test_sgd_update_is_the_same_for_any_alignment(n, adagrad):
    from parameter_server_b200.ops import dense

    w, g, h = torch.randn(3, n + 1, device="cuda").abs().unbind(0)
    out = []
    for at in (0, 1):                      # 16-byte aligned, then not
        bufs = [torch.zeros(n + 1, device="cuda")[at: at + n].copy_(t[:n]) for t in (w, g, h)]
        dense.sgd_update(bufs[0], bufs[1], bufs[2] if adagrad else None, 0.1, 1.0, 4)
        out.append((bufs[0].clone(), bufs[2].clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("M,K", [(1_048_560, 1), (1_048_561, 2), (1_100_003, 3), (2_200_000, 4)])
def test_outer_product_of_more_rows_than_a_grid_has_blocks(M, K):
    from parameter_server_b200.ops import dense

    a, b = torch.randn(M, K, device="cuda"), torch.randn(8, K, device="cuda")
    t = torch.full((8, M), float("nan"), device="cuda")
    out = dense.gemm_tn(a, b, pad_k=True, out_t=t)
    ref, bound = a.double() @ b.double().T, (a.double().abs() @ b.double().abs().T) / 512 + 1e-5      # TF32 operands
    assert bool(((out.double() - ref).abs() <= bound).all()) and torch.equal(t, out.T)
