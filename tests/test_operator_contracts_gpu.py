"""What the operators promise beside their numbers: current weights, any batch and filter size, operand types, storage of
gradients, reproducibility on request, other threads' progress."""
import gc

import pytest
import torch
import torch.nn.functional as F

from rannc_b200.ops import functional as RF

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rel(got, want):
    got, want = got.detach(), want.detach().double()
    return float((got.double() - want).norm() / want.norm().clamp_min(1e-30))


def _randn(*shape, std=1.0, dtype=BF):
    return (torch.randn(*shape, device="cuda") * std).to(dtype)


# ------------------------------------------------------------------------------------------ current weights
def _attention_ref(x, ws, bs, heads):
    B, S, _ = x.shape
    q, k, v = (F.linear(x.double(), w.double(), b.double()).view(B, S, heads, 64).transpose(1, 2) for w, b in zip(ws, bs))
    return (torch.softmax(q @ k.transpose(2, 3) / 8, -1) @ v).transpose(1, 2).reshape(B, S, heads * 64)


def _attention(x, ws, bs, heads):
    return RF.qkv_attention(x, ws[0], bs[0], ws[1], bs[1], ws[2], bs[2], num_heads=heads)


@pytest.mark.parametrize("through_data", [False, True])
def test_projections_changed_in_place_are_seen(through_data):
    """16-bit rounding of the projections, probabilities and outputs: 2^-8 each, three of them."""
    torch.manual_seed(0)
    x = _randn(2, 33, 128)
    ws, bs = [_randn(128, 128, std=128 ** -0.5) for _ in range(3)], [_randn(128, std=0.1) for _ in range(3)]
    for _ in range(3):
        assert _rel(_attention(x, ws, bs, 2), _attention_ref(x, ws, bs, 2)) < 3 * 2.0 ** -8
        for t in ws + bs:
            (t.data if through_data else t).add_(torch.randn_like(t) * 0.1)


@pytest.mark.parametrize("through_data", [False, True])
def test_filters_changed_in_place_are_seen(through_data):
    torch.manual_seed(1)
    x, w = _randn(2, 64, 12, 12), _randn(72, 64, 3, 3, std=0.05)
    for stride in (1, 2):
        for _ in range(3):
            xg = x.clone().requires_grad_(True)
            y = RF.conv2d(xg, w, None, stride, 1)
            xr = x.double().requires_grad_(True)
            ref = F.conv2d(xr, w.double(), None, stride, 1)
            assert _rel(y, ref) < 2.0 ** -8
            y.backward(torch.ones_like(y))
            ref.backward(torch.ones_like(ref))
            # the gathered path rounds each of the nine taps' shares before it sums them
            assert _rel(xg.grad, xr.grad) < 9 * 2.0 ** -9
            (w.data if through_data else w).add_(torch.randn_like(w) * 0.05)


def test_weights_at_a_freed_tensors_address_are_their_own():
    torch.manual_seed(2)
    x, xi = _randn(1, 16, 128), _randn(1, 64, 8, 8)
    for _ in range(12):
        ws, bs = [_randn(128, 128, std=128 ** -0.5) for _ in range(3)], [_randn(128, std=0.1) for _ in range(3)]
        assert _rel(_attention(x, ws, bs, 2), _attention_ref(x, ws, bs, 2)) < 3 * 2.0 ** -8
        w = _randn(64, 64, 3, 3, std=0.05)
        assert _rel(RF.conv2d(xi, w, None, 1, 1), F.conv2d(xi.double(), w.double(), None, 1, 1)) < 2.0 ** -8
        del ws, bs, w
        gc.collect()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Co,Ci", [(1, 8), (3, 264), (130, 256), (5, 72)])
@pytest.mark.parametrize("k", [2, 3, 9, 10, 18, 19, 32])
def test_filters_packed_tap_by_tap(dtype, Co, Ci, k):
    """Each channel-block width of the kernel, last blocks of a few channels; a channels-last filter is read in place."""
    torch.manual_seed(6)
    w = _randn(Co, Ci, k, k, dtype=dtype)
    want = w.permute(0, 2, 3, 1).reshape(Co, -1)
    got = RF._conv_weight(w)
    assert RF.K.pack_taps_ok(w) and torch.equal(got, want)
    cl = w.to(memory_format=torch.channels_last)
    assert RF._conv_weight(cl).data_ptr() == cl.data_ptr() and torch.equal(RF._conv_weight(cl), want)
    assert torch.equal(RF._conv_weight(w[:, :, 1:, 1:]), w[:, :, 1:, 1:].permute(0, 2, 3, 1).reshape(Co, -1))


# ------------------------------------------------------------------------------------------ filter sizes
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("k,stride,pad", [(9, 1, 4), (10, 1, 0), (11, 4, 2), (16, 16, 0)])
def test_large_filters(k, stride, pad, flat):
    torch.manual_seed(3)
    x = _randn(2, 16, 35, 34).requires_grad_(True)
    w = _randn(24, 16, k, k, std=(16 * k * k) ** -0.5).requires_grad_(True)
    if flat:
        w.main_grad = torch.full(w.shape, 2.0, device="cuda")
    y = RF.conv2d(x, w, None, stride, pad)
    xr, wr = (t.detach().double().requires_grad_(True) for t in (x, w))
    ref = F.conv2d(xr, wr, None, stride, pad)
    dy = _randn(*y.shape)
    y.backward(dy)
    ref.backward(dy.double())
    assert _rel(y, ref) < 2.0 ** -8
    assert _rel(w.main_grad - 2.0 if flat else w.grad, wr.grad) < (1e-5 if flat else 2.0 ** -8)
    assert _rel(x.grad, xr.grad) < k * 2.0 ** -8       # k * k roundings of parts that add up like a random walk


# ------------------------------------------------------------------------------------------ empty batches
@pytest.mark.parametrize("op", ["linear", "mlp", "layer_norm", "conv1x1", "attention"])
def test_an_empty_batch_has_zero_parameter_gradients(op):
    mk = lambda *s: _randn(*s).requires_grad_(True)  # noqa: E731
    poison = [torch.full((512, 512), float("nan"), device="cuda", dtype=BF) for _ in range(8)]   # noqa: F841
    del poison
    if op == "linear":
        ps = [mk(64, 128), mk(64)]
        y = RF.linear(torch.empty(0, 128, device="cuda", dtype=BF), *ps)
    elif op == "mlp":
        ps = [mk(256, 128), mk(256), mk(128, 256), mk(128)]
        y = RF.mlp(torch.empty(0, 128, device="cuda", dtype=BF), *ps)
    elif op == "layer_norm":
        ps = [mk(256), mk(256)]
        y = RF.dropout_add_layer_norm(torch.empty(0, 256, device="cuda", dtype=BF), None, *ps)
    elif op == "attention":
        ps = [mk(128, 128) for _ in range(3)] + [mk(128) for _ in range(3)]
        y = _attention(torch.empty(0, 16, 128, device="cuda", dtype=BF), ps[:3], ps[3:], 2)
    else:
        ps = [mk(64, 128, 1, 1), mk(64)]
        y = RF.conv2d(torch.empty(0, 128, 4, 4, device="cuda", dtype=BF), *ps)
    y.sum().backward()
    for p in ps:
        assert p.grad is not None and bool((p.grad == 0).all())


@pytest.mark.parametrize("out", [BF, torch.float32])
def test_a_product_over_nothing_is_zero(out):
    from rannc_b200.ops.gemm import gemm

    buf = torch.full((40, 32), 3.0, device="cuda", dtype=out)
    gemm(torch.empty(0, 40, device="cuda", dtype=BF), torch.empty(0, 24, device="cuda", dtype=BF), trans_a=True,
         trans_b=False, out=buf[:, :24])
    assert bool((buf[:, :24] == 0).all()) and bool((buf[:, 24:] == 3).all())
    if out == torch.float32:
        buf.fill_(3.0)
        gemm(torch.empty(0, 40, device="cuda", dtype=BF), torch.empty(0, 32, device="cuda", dtype=BF), trans_a=True,
             trans_b=False, out=buf, accumulate=True)
        assert bool((buf == 3).all())
    x, w, b = torch.empty(3, 0, device="cuda", dtype=BF), torch.empty(8, 0, device="cuda", dtype=BF), _randn(8)
    assert torch.equal(RF.linear(x, w, b), b.expand(3, 8))


# ------------------------------------------------------------------------------------------ operand types
@pytest.mark.parametrize("res", [False, True])
def test_layer_norm_with_parameters_of_another_type(res):
    torch.manual_seed(4)
    x = _randn(37, 512).requires_grad_(True)
    r = _randn(37, 512).requires_grad_(True) if res else None
    g, b = (torch.rand(512, device="cuda") + 0.5).requires_grad_(True), torch.randn(512, device="cuda").requires_grad_(True)
    y = RF.dropout_add_layer_norm(x, r, g, b, 0.0, 1e-5)
    dy = _randn(37, 512)
    y.backward(dy.to(y.dtype))
    xr, gr, br = (t.detach().double().requires_grad_(True) for t in (x, g, b))
    ref = F.layer_norm(xr + (r.detach().double() if res else 0.0), (512,), gr, br, 1e-5)
    ref.backward(dy.double())
    assert y.dtype == BF and _rel(y, ref) < 2 * 2.0 ** -8
    # the residual sum and the result are each rounded once
    assert _rel(x.grad, xr.grad) < 3 * 2.0 ** -8
    assert g.grad.dtype == torch.float32 and _rel(g.grad, gr.grad) < 2.0 ** -7 and _rel(b.grad, br.grad) < 2.0 ** -7


@pytest.mark.parametrize("shape", [(1, 5, 256), (256,), (3, 1, 1)])
def test_layer_norm_with_a_residual_that_broadcasts(shape):
    torch.manual_seed(7)
    x, r = _randn(3, 5, 256), _randn(*shape)
    g, b = _randn(256) + 1, _randn(256)
    y = RF.dropout_add_layer_norm(x, r, g, b, 0.0, 1e-5)
    want = F.layer_norm(x.double() + r.double(), (256,), g.double(), b.double(), 1e-5)
    assert y.shape == x.shape and _rel(y, want) < 2 * 2.0 ** -8     # the sum and the result are each rounded


def test_layer_norm_refuses_operands_its_kernels_would_misread():
    from rannc_b200.ops import _lib

    h, x, g = _lib.host(), _randn(4, 256), _randn(256)
    ln = lambda **k: h.layer_norm(k.get("x", x), k.get("r"), k.get("g", g), k.get("b", g), 0.0, 1e-5, 0, 0, None, None)  # noqa: E731
    ln()
    two = torch.stack((g, _randn(256)), 1)
    assert torch.equal(ln(g=two[:, 0], b=two[:, 0].reshape(1, 256)), ln())      # a strided parameter is read as what it is
    for bad, err in (({"g": g.float()}, TypeError), ({"b": g.half()}, TypeError), ({"r": x.float()}, TypeError),
                     ({"g": g[:128]}, ValueError), ({"r": x[:2]}, ValueError)):
        with pytest.raises(err):
            ln(**bad)


def test_operands_the_kernels_would_misread_are_refused():
    """Too short, of another type or elsewhere: ATen's own errors where a call falls back to it, the native entries' else."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm

    h, x, w, b = _lib.host(), _randn(8, 128), _randn(64, 128), _randn(64)
    w2 = _randn(128, 64)
    ids, table = torch.arange(8, device="cuda"), _randn(16, 64)
    logits, labels = _randn(8, 64), torch.arange(8, device="cuda")
    for bad in (b[:32], b.float(), b.half()):
        for call in (lambda: RF.linear(x, w, bad), lambda: RF.mlp(x, w, bad, w2, None),
                     lambda: RF.conv2d(_randn(1, 128, 4, 4), w.view(64, 128, 1, 1), bad),
                     lambda: RF.conv2d(_randn(1, 128, 4, 4), _randn(64, 128, 3, 3), bad)):
            with pytest.raises(RuntimeError):
                call()
        for call in (lambda: h.linear(x, w, bad, False, None, None, None), lambda: gemm(x, w, bias=bad)):
            with pytest.raises((TypeError, ValueError)):
                call()
    with pytest.raises(RuntimeError):
        RF.mlp(x, w, b, w2.float(), None)
    with pytest.raises(RuntimeError):
        RF.cross_entropy(logits, labels.int())
    with pytest.raises((RuntimeError, ValueError)):
        RF.cross_entropy(logits, labels[:4])
    qkv = lambda **k: RF.qkv_attention(_randn(1, 16, 128), *(k.get(n, d) for n, d in (  # noqa: E731
        ("wq", w2.new_zeros(128, 128)), ("bq", w2.new_zeros(128)), ("wk", w2.new_zeros(128, 128)), ("bk", w2.new_zeros(128)),
        ("wv", w2.new_zeros(128, 128)), ("bv", w2.new_zeros(128)))), num_heads=2)
    qkv()
    for bad in (dict(wk=torch.zeros(128, 128, device="cuda")), dict(bv=w2.new_zeros(64)), dict(bq=torch.zeros(128, device="cuda"))):
        with pytest.raises(RuntimeError):
            qkv(**bad)
    for call in (lambda: h.embedding(table, ids.int(), -1, None), lambda: h.embedding(table.t(), ids, -1, None),
                 lambda: h.cross_entropy(logits, labels, 65, -100, 1.0), lambda: h.cross_entropy(logits, labels[:4], 64, -100, 1.0),
                 lambda: gemm(x, w, out=torch.empty(8, 32, device="cuda", dtype=BF)), lambda: gemm(x, w.half()),
                 lambda: gemm(x, w, residual=_randn(8, 128)[:, :64]), lambda: gemm(x, w, gelu=True, aux_out=_randn(8, 32))):
        with pytest.raises((TypeError, ValueError)):
            call()
    wg = w.clone().requires_grad_(True)
    for mg in (torch.zeros(64, 64, device="cuda"), torch.zeros(64, 128, device="cuda", dtype=torch.float64),
               torch.zeros(64, 128)):
        wg.main_grad = mg
        with pytest.raises((TypeError, ValueError)):
            RF.linear(x, wg, b)


def test_operands_laid_out_another_way_are_read_as_they_are():
    torch.manual_seed(8)
    x, w = _randn(8, 128), _randn(64, 128)
    strided = _randn(64, 2)[:, 0]
    assert torch.equal(RF.linear(x, w, strided), RF.linear(x, w, strided.contiguous()))
    ids, table = torch.randint(0, 64, (9,), device="cuda"), _randn(64, 64).t()
    assert torch.equal(RF.embedding(table, ids), table[ids])
    logits, labels = _randn(8, 64), torch.arange(8, device="cuda")
    assert torch.allclose(RF.cross_entropy(logits.clone(), labels, num_classes=99), F.cross_entropy(logits.float(), labels))
    # running statistics that no kernel writes in place
    img = _randn(4, 16, 5, 5).to(memory_format=torch.channels_last)
    g, bt = torch.rand(16, 2, device="cuda")[:, 0], torch.rand(16, 2, device="cuda")[:, 1]
    rm, rv = torch.zeros(16, 2, device="cuda")[:, 0], torch.ones(16, 2, device="cuda")[:, 0]
    y = RF.batch_norm_act(img, g, bt, rm, rv)
    rmr, rvr = torch.zeros(16, device="cuda"), torch.ones(16, device="cuda")
    want = F.batch_norm(img.float(), rmr, rvr, g, bt, True)
    assert _rel(y, want) < 2.0 ** -8 and torch.allclose(rm, rmr, atol=1e-5) and torch.allclose(rv, rvr, atol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_a_weights_gradient_buffer_in_fp32_or_its_own_type(dtype):
    torch.manual_seed(9)
    x, dy = _randn(512, 128), _randn(512, 64)
    w = _randn(64, 128).requires_grad_(True)
    w.main_grad = torch.ones(64, 128, device="cuda", dtype=dtype)
    RF.linear(x, w).backward(dy)
    assert w.grad is None and _rel(w.main_grad, 1.0 + dy.double().t() @ x.double()) < (1e-5 if dtype == torch.float32 else 2.0 ** -8)


def _off(t):
    """The same values and strides, starting one element past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    v = buf[1:].as_strided(t.shape, t.stride())
    with torch.no_grad():
        v.copy_(t)
    assert v.data_ptr() % 16
    return v


def test_operands_that_start_at_any_element():
    """The results are those of aligned copies, bit for bit, gradients included."""
    torch.manual_seed(10)
    cl = lambda *s: _randn(*s).to(memory_format=torch.channels_last)  # noqa: E731
    ids = torch.randint(0, 33, (17,), device="cuda")
    cases = {
        "layer_norm": (lambda x, r, g, b: RF.dropout_add_layer_norm(x, r, g, b, 0.0, 1e-5),
                       [_randn(9, 512), _randn(9, 512), _randn(512), _randn(512)]),
        "gelu": (RF.gelu, [_randn(5, 24)]),
        "embedding": (lambda w: RF.embedding(w, ids), [_randn(33, 64)]),
        "linear bias": (lambda b, x=_randn(40, 64), w=_randn(96, 64): RF.linear(x, w, b, act="gelu"), [_randn(96)]),
        "conv": (lambda x: RF.conv2d(x, w3, None, 1, 1), [cl(2, 64, 12, 12)]),
        "strided conv": (lambda x: RF.conv2d(x, w3, None, 2, 1), [cl(2, 64, 12, 12)]),
        "batch_norm": (lambda x, r, g, b: RF.batch_norm_act(x, g, b, None, None, relu=True, residual=r),
                       [cl(2, 64, 5, 5), cl(2, 64, 5, 5), torch.rand(64, device="cuda"), torch.rand(64, device="cuda")]),
        "sdpa": (lambda q, k, v: RF.sdpa(q, k, v), [_randn(2, 3, 20, 64) for _ in range(3)]),
        "qkv": (lambda x, *p: RF.qkv_attention(x, *p, num_heads=2),
                [_randn(2, 20, 128), _randn(128, 128), _randn(128), _randn(128, 128), _randn(128), _randn(128, 128), _randn(128)]),
    }
    w3 = _randn(64, 64, 3, 3, std=0.05)
    for name, (fn, args) in cases.items():
        got = []
        for shift in (False, True):
            # (the first projection weight and the attention input off a boundary select another path: left aligned)
            leaves = [(_off(a) if shift and not (name == "qkv" and i in (0, 1)) else a.clone()).requires_grad_(True)
                      for i, a in enumerate(args)]
            y = fn(*leaves)
            torch.manual_seed(11)
            dy = torch.randn_like(y)
            y.backward(_off(dy) if shift else dy)
            got.append([y] + [t.grad for t in leaves])
        tol = 2.0 ** -8 if name in ("batch_norm", "embedding") else 0.0      # sums whose order is not fixed
        for a, b in zip(*got):
            assert torch.equal(a, b) if tol == 0.0 else _rel(a, b) < tol, name
    x = _randn(5, 24)
    RF.manual_seed(3)
    d0 = RF.dropout(x, 0.5)
    RF.manual_seed(3)
    assert torch.equal(RF.dropout(_off(x), 0.5), d0)


@pytest.mark.parametrize("out_dtype", [BF, torch.float32])
@pytest.mark.parametrize("M,N", [(3, 64), (150, 264)])
def test_product_outputs_that_start_at_any_element(M, N, out_dtype):
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(12)
    a, b, r = _randn(M, 72), _randn(N, 72, std=0.1), _randn(M, N)
    bias, base = _randn(N), _randn(M, N, dtype=out_dtype)
    want = gemm(a, b, bias=bias, residual=r, out=base.clone(), accumulate=True)
    assert torch.equal(gemm(a, b, bias=_off(bias), residual=_off(r), out=_off(base), accumulate=True), want)
    aux, pre = torch.empty(M, N, device="cuda", dtype=BF), _off(torch.zeros(M, N, device="cuda", dtype=BF))
    y0, y1 = gemm(a, b, bias=bias, gelu=True, aux_out=aux), gemm(a, b, bias=bias, gelu=True, aux_out=pre)
    # the two ways a result leaves the kernel evaluate GELU scalar by scalar and in pairs: a last fp32 bit apart, which 16-bit
    # rounding may turn into one of its own
    assert torch.equal(aux, pre) and _rel(y1, y0) < 2.0 ** -8
    assert _rel(gemm(a, b, dgelu=True, aux_in=pre), gemm(a, b, dgelu=True, aux_in=aux)) < 2.0 ** -8


# ------------------------------------------------------------------------------------------ weight gradients
def test_a_product_that_cannot_be_split_makes_no_fp32_copy():
    rows, K, N = 24576, 2048, 3072          # 12 x 8 tiles of 256 x 256: more than the SM pairs that run at once
    x, dy = _randn(rows, K), _randn(rows, N)
    w = _randn(N, K).requires_grad_(True)
    y = RF.linear(x, w)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    y.backward(dy)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before < 1.5 * w.numel() * 2


@pytest.mark.parametrize("op", ["linear", "conv"])
def test_weight_gradients_repeat_when_asked(op):
    """Products that add up partial sums in the order they arrive give way to one that does not."""
    torch.manual_seed(5)
    if op == "linear":
        x, w, dy = _randn(16384, 256), _randn(256, 256).requires_grad_(True), _randn(16384, 256)
        run = lambda: RF.linear(x, w)  # noqa: E731
    else:
        x, w, dy = _randn(16, 64, 28, 28), _randn(64, 64, 3, 3).requires_grad_(True), _randn(16, 64, 14, 14)
        run = lambda: RF.conv2d(x, w, None, 2, 1)  # noqa: E731
    torch.use_deterministic_algorithms(True)
    try:
        grads = []
        for _ in range(8):
            w.grad = None
            run().backward(dy)
            grads.append(w.grad)
        assert all(torch.equal(g, grads[0]) for g in grads)
    finally:
        torch.use_deterministic_algorithms(False)


@pytest.mark.parametrize("rows", [64, 4096])
def test_projection_gradients_have_their_own_storage(rows):
    x = _randn(rows // 64, 64, 128).requires_grad_(True)
    ws = [_randn(128, 128).requires_grad_(True) for _ in range(3)]
    bs = [_randn(128).requires_grad_(True) for _ in range(3)]
    _attention(x, ws, bs, 2).sum().backward()
    grads = [t.grad for t in ws + bs]
    assert len({g.untyped_storage().data_ptr() for g in grads}) == len(grads)
    assert all(g.untyped_storage().nbytes() == g.numel() * g.element_size() for g in grads)
    version = grads[1]._version
    grads[0].mul_(2)
    assert grads[1]._version == version


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,heads,hid,bias", [(37, 1, 8, True), (300, 2, 264, False), (4100, 1, 128, True), (197, 3, 72, True)])
def test_projection_gradients_leave_one_product(dtype, rows, heads, hid, bias):
    """Stored and split products, one vector per part up to many; with and without biases."""
    torch.manual_seed(13)
    n = 64 * heads
    x = _randn(1, rows, hid, dtype=dtype)
    ws = [_randn(n, hid, std=hid ** -0.5, dtype=dtype).requires_grad_(True) for _ in range(3)]
    bs = [_randn(n, dtype=dtype).requires_grad_(True) if bias else None for _ in range(3)]
    y = RF.qkv_attention(x, ws[0], bs[0], ws[1], bs[1], ws[2], bs[2], num_heads=heads)
    dy = _randn(*y.shape, dtype=dtype)
    y.backward(dy)
    wr = [w.detach().double().requires_grad_(True) for w in ws]
    br = [(b if bias else x.new_zeros(n)).detach().double().requires_grad_(True) for b in bs]
    _attention_ref(x, wr, br, heads).backward(dy.double())
    # dQ, dK and dV are rounded to 16 bits on their way, and the probabilities before them
    tol = 6 * (2.0 ** -8 if dtype == BF else 2.0 ** -11)
    for i, (got, want) in enumerate(zip(ws + (bs if bias else []), wr + br)):
        # (the key bias shifts all scores of a row: its gradient is zero but for rounding)
        assert i == 4 or _rel(got.grad, want.grad) < tol, i


# ------------------------------------------------------------------------------------------ autograd, threads
class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y):
        return y.clone()

    @staticmethod
    def backward(ctx, dy):
        return None


@pytest.mark.parametrize("op", ["linear", "layer_norm", "embedding"])
def test_a_missing_gradient_counts_as_zero_and_is_reported(op):
    """A parameter with a gradient buffer is reported although nothing flows back: a reducer counts on it."""
    w = _randn(256, 256).requires_grad_(True)
    g, b = _randn(256).requires_grad_(True), _randn(256).requires_grad_(True)
    for p in (w, g, b):
        p.main_grad = torch.zeros(p.shape, device="cuda")
    x = _randn(8, 256).requires_grad_(True)
    y = {"linear": lambda: RF.linear(x, w), "layer_norm": lambda: RF.dropout_add_layer_norm(x, None, g, b),
         "embedding": lambda: RF.embedding(w, torch.arange(8, device="cuda"))}[op]()
    seen = []
    RF.set_grad_listener(lambda ps: seen.extend(ps))
    try:
        _NoGradient.apply(y).sum().backward()
    finally:
        RF.set_grad_listener(None)
    want = [g, b] if op == "layer_norm" else [w]
    assert len(seen) == len(want) and all(any(s is p for s in seen) for p in want)
    assert all(float(p.main_grad.abs().max()) == 0.0 for p in want)
    assert op == "embedding" or (x.grad is not None and float(x.grad.abs().max()) == 0.0)


def test_other_threads_run_while_a_launch_waits():
    """The launch queue is filled behind a kernel that runs for 0.6 s; a thread that does nothing but look at the clock must
    not stand still for the time the launches wait."""
    import threading
    import time

    x, w = _randn(32, 256), _randn(256, 256)
    with torch.no_grad():
        RF.linear(x, w)
        torch.cuda.synchronize()
        stop, gap = threading.Event(), [0.0]

        def watch():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(0.001)
                now = time.perf_counter()
                gap[0] = max(gap[0], now - last)
                last = now

        th = threading.Thread(target=watch)
        th.start()
        time.sleep(0.05)
        torch.cuda._sleep(int(0.6 * 1.9e9))
        t0 = time.perf_counter()
        for _ in range(4096):
            RF.linear(x, w)
        waited = time.perf_counter() - t0
        stop.set()
        th.join()
        torch.cuda.synchronize()
    if waited < 0.4:
        pytest.skip("the launch queue took all launches")
    assert gap[0] < 0.6 * waited, (gap[0], waited)


def test_two_threads_differentiate_one_graph():
    """One keeps the graph, one releases it: each gets the gradient, or autograd's error about a released graph."""
    import threading

    torch.manual_seed(14)
    w, x = _randn(64, 64).requires_grad_(True), _randn(16, 64)
    want = torch.autograd.grad(RF.linear(x, w, act="gelu").sum(), w)[0]
    for _ in range(100):
        y, out = RF.linear(x, w, act="gelu").sum(), []

        def go(keep):
            try:
                out.append(torch.autograd.grad(y, w, retain_graph=keep)[0])
            except RuntimeError as e:
                out.append(e)

        ts = [threading.Thread(target=go, args=(k,)) for k in (True, False)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert len(out) == 2
        for o in out:
            assert torch.equal(o, want) if torch.is_tensor(o) else "second time" in str(o) or "already been freed" in str(o)


@pytest.mark.parametrize("bias", [-1e4, -1e6, -1e9, -1e15, -2e38])
def test_attention_backward_of_fully_masked_rows(bias):
    """A sequence that is all padding under a finite mask value: scores are rounded away beside it.  A single key has
    probability one, so dV is dO; of many keys none may exceed it."""
    torch.manual_seed(15)
    q, k, v, do = (_randn(1, 1, 2, 64, std=2.0) for _ in range(4))
    mask = torch.full((1, 1), bias, device="cuda")
    o, lse = RF.K.attn_fwd(q, k, v, mask)
    assert torch.equal(RF.K.attn_bwd(q, k, v, o, lse, do, mask)[2], do)
    B, S, H = 2, 160, 2
    q, k, v, do = (_randn(B, S, H, 64, std=2.0) for _ in range(4))
    mask = torch.full((B, S), bias, device="cuda")
    o, lse = RF.K.attn_fwd(q, k, v, mask)
    dv = RF.K.attn_bwd(q, k, v, o, lse, do, mask)[2]
    # each of S probabilities is at most one (a few roundings of 2^-8 above)
    assert bool((dv.abs().double() <= do.double().abs().sum(1, keepdim=True) * 1.02).all())


@pytest.mark.parametrize("first,last", [(0, 72), (8, 72), (8, 68), (3, 70), (0, 61)])
@pytest.mark.parametrize("classes", [None, 50])
def test_loss_of_a_slice_writes_only_the_slice(first, last, classes):
    """The gradient is written over the logits: not over what lies beside them in a wider matrix."""
    torch.manual_seed(16)
    whole = torch.zeros(9, 80, device="cuda", dtype=BF)
    whole[:8, :72] = _randn(8, 72)
    kept = whole.clone()
    logits = whole[:8, first:last].detach().requires_grad_(True)
    labels = torch.randint(0, 50, (8,), device="cuda")
    labels[3] = -100
    ref = kept[:8, first:last].double().requires_grad_(True)
    want = F.cross_entropy(ref[:, :classes], labels)
    want.backward()
    loss = RF.cross_entropy(logits, labels, num_classes=classes)
    loss.backward()
    assert abs(float(loss) - float(want)) < 1e-5 * abs(float(want))
    assert logits.grad.shape == ref.shape and _rel(logits.grad, ref.grad) < 2.0 ** -8
    beside = torch.ones_like(whole, dtype=torch.bool)
    beside[:8, first:last] = False
    assert torch.equal(whole[beside], kept[beside])


def test_loss_of_rows_that_share_memory():
    torch.manual_seed(17)
    row, labels = _randn(1, 40).requires_grad_(True), torch.arange(8, device="cuda")
    loss = RF.cross_entropy(row.expand(8, 40), labels)
    loss.backward()
    ref = row.detach().double().requires_grad_(True)
    F.cross_entropy(ref.expand(8, 40), labels).backward()
    assert _rel(row.grad, ref.grad) < 8 * 2.0 ** -8       # eight rows' gradients, each rounded


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k,kernel", [(1, False), (3, False), (4, True), (5, True), (9, True), (10, False)])
@pytest.mark.parametrize("Co,Ci", [(3, 8), (5, 264)])
def test_weight_gradient_folds_on_both_sides_of_the_rule(dtype, k, kernel, Co, Ci):
    """Added to an fp32 buffer or written in the filter's type, by the kernel or the strided operation."""
    dw2 = torch.randn(Co, k * k * Ci, device="cuda")
    w = torch.zeros(Co, Ci, k, k, device="cuda", dtype=BF if dtype == torch.float32 else dtype)
    want = dw2.view(Co, k, k, Ci).permute(0, 3, 1, 2)
    if dtype == torch.float32:
        mg = torch.ones(Co, Ci, k, k, device="cuda")
        assert RF.K.wgrad_fold_ok(mg) == kernel and RF._Conv2d._fold(dw2, w, mg, k) is None
        assert torch.equal(mg, 1.0 + want)
    else:
        assert RF.K.wgrad_fold_ok(w) == kernel
        got = RF._Conv2d._fold(dw2, w, None, k)
        assert got.is_contiguous() and torch.equal(got, want.to(dtype))


def test_kernel_entries_refuse_addresses_off_a_boundary():
    """An error code from the host, nothing launched: on the device it would be a fault."""
    from rannc_b200.ops import _lib

    K = RF.K
    x, v, f = _randn(8, 256), _randn(256), torch.zeros(8, device="cuda")
    img, c32 = _randn(50, 64), torch.zeros(64, device="cuda")
    q = _randn(1, 16, 2, 64)
    o, lse = K.attn_fwd(q, q, q)
    calls = [lambda: K.ln_fwd(_off(x), None, v, v, 1e-5), lambda: K.ln_fwd(x, _off(x), v, v, 1e-5),
             lambda: K.ln_fwd(x, None, _off(v), v, 1e-5), lambda: K.ln_bwd(_off(x), x, v, f, f),
             lambda: K.ln_bwd(x, x, _off(v), f, f), lambda: K.gelu(_off(x)), lambda: K.gelu_bwd(x, _off(x)),
             lambda: K.dropout(_off(x), 0.5, 1, 1), lambda: K.embed_fwd(torch.zeros(3, dtype=torch.int64, device="cuda"), _off(x)),
             lambda: K.im2col(_off(_randn(1, 5, 5, 8)), 3, 1, 1), lambda: K.col2im(_off(_randn(25, 72)), 1, 5, 5, 8, 3, 1, 1),
             lambda: K.bn_fwd(_off(img), None, c32, c32, None, None, 1e-5, 0.1, False),
             lambda: K.bn_bwd(img, img, img, _off(c32), c32, c32, False, False),
             lambda: K.bn_bwd(img, _off(img), img, c32, c32, c32, False, False),
             lambda: K.attn_bwd(q, q, q, _off(o), lse, q), lambda: K.attn_bwd(q, q, q, o, lse, q, dv=_off(q)),
             lambda: K.attn_fwd(_off(q), q, q)]
    for call in calls:
        with pytest.raises(_lib.KernelLibraryError):
            call()
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("how", ["channels_last", "contiguous", "slice", "odd", "empty"])
@pytest.mark.parametrize("flat,bias", [(True, False), (False, True)])
def test_pointwise_convolution_takes_any_layout(dtype, how, flat, bias):
    """A 1x1 convolution of images in any order, from any address, and of none: values, gradients and the layouts of both."""
    from rannc_b200.ops import functional as RF

    torch.manual_seed(3)
    N, Ci, Co, H, W = (0 if how == "empty" else 3), 24, 40, 5, 7
    x = torch.randn(N, Ci + 8, H, W, device="cuda").to(dtype)
    if how == "odd":      # an address off a 16-byte boundary
        x = torch.empty(x[:, :Ci].numel() + 1, device="cuda", dtype=dtype)[1:].view(N, H, W, Ci).normal_().permute(0, 3, 1, 2)
    elif how == "slice":
        x = x.to(memory_format=torch.channels_last)[:, 8:]
    else:
        x = x[:, :Ci].contiguous(memory_format=torch.contiguous_format if how == "contiguous" else torch.channels_last)
    x = x.detach().requires_grad_(True)
    w = torch.randn(Co, Ci, 1, 1, device="cuda").to(dtype).requires_grad_(True)
    b = torch.randn(Co, device="cuda").to(dtype).requires_grad_(True) if bias else None
    if flat:
        w.main_grad = torch.full((Co, Ci, 1, 1), 2.0, device="cuda")
    y = RF.conv2d(x, w, b)
    assert y.shape == (N, Co, H, W) and (N == 0 or y.is_contiguous(memory_format=torch.channels_last))
    dy = torch.randn(N, Co, H, W, device="cuda").to(dtype)
    y.backward(dy)
    assert x.grad.shape == x.shape and (w.grad is None) == flat
    xr, wr = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    ref = torch.nn.functional.conv2d(xr, wr, None if b is None else b.detach().double())
    ref.backward(dy.double())
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    pairs = [(y, ref, u), (x.grad, xr.grad, u), (w.main_grad - 2.0 if flat else w.grad, wr.grad, 0.0 if flat else u)]
    if b is not None:
        pairs.append((b.grad, dy.double().sum((0, 2, 3)), u))
    for got, want, rounding in pairs:      # one rounding of the result; fp32 sums (that start at 2 where they are added)
        assert ((got.double() - want).abs() <= rounding * want.abs() + 1e-5 * (want.abs().max() if N else 0) + 1e-6).all()
