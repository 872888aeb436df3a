"""Kernel variants at the sizes where their tiles, blocks and strips end, against fp32 / fp64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Largest relative error of one rounding to nearest: half the spacing of 8 (bf16) or 11 (fp16) significant bits
U = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _near(got, want, dtype, roundings, extra=0.0):
    """Every element within `roundings` storage roundings of its own value, plus fp32 accumulation error relative
    to the result's scale: 1e-5 covers sums of up to some thousand terms, `extra` what longer ones need (a product
    over K terms is accumulated in steps of 16, each of which may lose 2^-23 of the running sum)."""
    want = want.double()
    bound = roundings * U[dtype] * want.abs() + (1e-5 + extra) * want.abs().max() + 1e-7
    bad = (got.double() - want).abs() > bound
    assert not bad.any(), f"{int(bad.sum())} of {bad.numel()}, worst {float(((got.double() - want).abs() - bound).max())}"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 31, 33, 128, 257, 2305])
@pytest.mark.parametrize("N", [8, 40, 248, 264, 2312])
def test_gemm_staged_epilogue_blocks(dtype, M, N):
    """Outputs leave in 32 x 32 blocks: partial blocks in both directions, both kernel variants, every epilogue;
    columns beyond N and rows beyond M of a larger buffer stay untouched."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(0)
    K = 72
    x = torch.randn(M, K, device="cuda").to(dtype)
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).to(dtype)
    bias = torch.randn(N, device="cuda").to(dtype)
    z = x.double() @ w.double().t()
    buf = torch.full((M + 3, N + 8), 7.0, device="cuda", dtype=dtype)
    gemm(x, w, out=buf[:M, :N])
    _near(buf[:M, :N], z, dtype, 1)
    assert (buf[M:] == 7.0).all() and (buf[:, N:] == 7.0).all()
    pre = torch.empty(M, N, device="cuda", dtype=dtype)
    y = gemm(x, w, bias=bias, gelu=True, aux_out=pre)
    _near(pre, z + bias.double(), dtype, 1)
    _near(y, torch.nn.functional.gelu(z + bias.double()), dtype, 1)
    t = pre.double().requires_grad_(True)
    torch.nn.functional.gelu(t).sum().backward()
    _near(gemm(x, w, dgelu=True, aux_in=pre), z * t.grad, dtype, 1)
    # what must not be hidden from an overflow check, and signed zeros
    odd = torch.zeros(M, K, device="cuda", dtype=dtype)
    one = torch.zeros(N, K, device="cuda", dtype=dtype)
    edge = torch.tensor([float("inf"), float("nan"), 0.0, -0.0, 6e4, -6e4], device="cuda").to(dtype)
    b6 = torch.zeros(N, device="cuda", dtype=dtype)
    b6[:6] = edge
    got = gemm(odd, one, bias=b6, gelu=True)[0, :6].float()
    assert torch.isinf(got[0]) and got[0] > 0 and torch.isnan(got[1]) and (got[2:4] == 0).all()
    assert got[4] == edge[4].float() and got[5] == 0
    acc = torch.full((M + 1, N + 4), 3.0, device="cuda")
    gemm(x, w, out=acc[:M, :N], accumulate=True, alpha=0.5)
    _near(acc[:M, :N], 0.5 * z + 3.0, dtype, 0)
    assert (acc[M:] == 3.0).all() and (acc[:, N:] == 3.0).all()
    f32 = gemm(x, w, out_dtype=torch.float32)
    _near(f32, z, dtype, 0)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 3, 9, 1187, 5000])
@pytest.mark.parametrize("H", [256, 512, 768, 1024, 1536, 2048, 3072, 4096])
def test_layernorm_ring_of_rows(dtype, rows, H):
    """Every width's split of a row over warps; fewer rows than the ring is deep, and several turns of it."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(2)
    x, res, dy = (torch.randn(rows, H, device="cuda").to(dtype) for _ in range(3))
    g = (torch.randn(H, device="cuda") * 0.1 + 1).to(dtype)
    b = (torch.randn(H, device="cuda") * 0.1).to(dtype)
    for r, p in ((res, 0.0), (None, 0.0), (res, 0.25)):
        y, z, mean, rstd = K.ln_fwd(x, r, g, b, 1e-5, p=p, seed=7, offset=3)
        kept = K.dropout(x, p, 7, 3) != 0 if p else None
        xd = x.double() if kept is None else torch.where(kept, x.double() / (1 - p), 0.0 * x.double())
        _near(z, xd + (0 if r is None else r.double()), dtype, 1)
        zz = z.double().requires_grad_(True)
        gg, bb = g.double().requires_grad_(True), b.double().requires_grad_(True)
        want = torch.nn.functional.layer_norm(zz, (H,), gg, bb, 1e-5)
        _near(y, want, dtype, 1)
        want.backward(dy.double())
        dz, dx, dg, db = K.ln_bwd(dy, z, g, mean, rstd, p=p, seed=7, offset=3)
        _near(dz, zz.grad, dtype, 1)
        if kept is not None:
            _near(dx, torch.where(kept, zz.grad / (1 - p), 0.0 * zz.grad), dtype, 1)
        _near(dg, gg.grad, dtype, 0)
        _near(db, bb.grad, dtype, 0)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("N,C,Co,H,W,k", [(2, 64, 64, 28, 26, 3), (3, 192, 72, 24, 31, 3), (1, 320, 136, 25, 24, 5),
                                          (2, 1024, 2112, 24, 24, 3), (2, 40, 264, 9, 7, 3)])
def test_convolution_weight_gradient(flat, N, C, Co, H, W, k):
    """All taps in one GEMM (column blocks that straddle taps, split and unsplit K), padded operands, and the fold
    into the [Co, Ci, k, k] layout for both kinds of gradient; a gathered-matrix case last."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF

    torch.manual_seed(3)
    cl = torch.channels_last
    x = torch.randn(N, C, H, W, device="cuda").bfloat16().to(memory_format=cl).requires_grad_(True)
    w = (torch.randn(Co, C, k, k, device="cuda") * (C * k * k) ** -0.5).bfloat16().requires_grad_(True)
    if flat:
        w.main_grad = torch.full((Co, C, k, k), 2.0, device="cuda")
    y = RF.conv2d(x, w, None, 1, k // 2)
    dy = torch.randn(N, Co, H, W, device="cuda").bfloat16().to(memory_format=cl)
    y.backward(dy)
    xr, wr = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    ref = torch.nn.functional.conv2d(xr, wr, None, 1, k // 2)
    ref.backward(dy.double())
    torch.cuda.synchronize()
    assert _lib.read_error() == 0
    steps = lambda terms: terms / 16 * 2.0 ** -23  # noqa: E731
    _near(y, ref.detach(), torch.bfloat16, 1, steps(C * k * k))
    if flat:
        _near(w.main_grad - 2.0, wr.grad, torch.bfloat16, 0, steps(N * H * W) + 1e-5)
    else:
        assert w.grad.shape == w.shape
        _near(w.grad, wr.grad, torch.bfloat16, 1, steps(N * H * W))
    # the gathered path rounds every tap's contribution before it sums them
    terms = 1 if RF._Conv2d._implicit(k, 1, k // 2, C, Co, H, W) else k * k
    _near(x.grad, xr.grad, torch.bfloat16, terms, steps(Co * k * k) + (4e-3 if terms > 1 else 0.0))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 264), (17, 1024), (4099, 256), (16400, 1024)])
def test_embedding_backward_strips(dtype, rows, H):
    """Strips of rows whose ids repeat, differ, are the padding id or lie outside the table."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(1)
    V = 37
    ids = torch.randint(-2, V + 2, (rows,), device="cuda")
    ids[rows // 3:rows // 2] = 5
    dout = torch.randn(rows, H, device="cuda").to(dtype)
    table = torch.ones(V, H, device="cuda")
    K.embed_bwd(ids, dout, table, padding_idx=9)
    keep = (ids >= 0) & (ids < V) & (ids != 9)
    want = torch.ones(V, H, device="cuda", dtype=torch.float64)
    want.index_add_(0, ids[keep], dout[keep].double())
    # fp32 sums of up to `rows` terms of size one in any order: error grows like the square root of their number
    assert (table.double() - want).abs().max().item() <= 2.0 ** -23 * 8 * max(1.0, rows ** 0.5) * 4
    shifted = torch.ones(V * H + 1, device="cuda")[1:].view(V, H)     # 4-byte aligned only: the scalar kernel
    K.embed_bwd(ids, dout, shifted, padding_idx=9)
    assert (shifted.double() - want).abs().max().item() <= 2.0 ** -23 * 8 * max(1.0, rows ** 0.5) * 4


@pytest.mark.parametrize("C", [8, 64, 72, 128, 264, 2048])
@pytest.mark.parametrize("N,H,W", [(1, 1, 2), (3, 5, 7), (8, 28, 28)])
@pytest.mark.parametrize("flat", [False, True])
def test_batch_norm_channel_blocks(C, N, H, W, flat):
    from rannc_b200.ops import functional as RF

    torch.manual_seed(6)
    dt, cl = torch.bfloat16, torch.channels_last
    mk = lambda: torch.randn(N, C, H, W, device="cuda").to(dt).to(memory_format=cl)  # noqa: E731
    x, r, dy = (mk() * 2).requires_grad_(True), mk().requires_grad_(True), mk()
    g = (torch.rand(C, device="cuda") + 0.5).requires_grad_(True)
    b = torch.randn(C, device="cuda").requires_grad_(True)
    if flat:
        g.main_grad, b.main_grad = torch.full((C,), 3.0, device="cuda"), torch.full((C,), -1.0, device="cuda")
    rm, rv = torch.zeros(C, device="cuda"), torch.ones(C, device="cuda")
    y = RF.batch_norm_act(x, g, b, rm, rv, True, 0.1, 1e-5, True, r)
    y.backward(dy)
    xr, rr, gr, br = (t.detach().double().requires_grad_(True) for t in (x, r, g, b))
    rmr, rvr = torch.zeros(C, device="cuda", dtype=torch.float64), torch.ones(C, device="cuda", dtype=torch.float64)
    pre = torch.nn.functional.batch_norm(xr, rmr, rvr, gr, br, True, 0.1, 1e-5) + rr
    _near(y, torch.relu(pre).detach(), dt, 1, 1e-5)
    _near(rm, rmr, dt, 0)
    _near(rv, rvr, dt, 0, 1e-5)
    # the mask comes from the rounded output: compare with that mask
    pre.backward(dy.double() * (y > 0))
    # two samples: x - mean cancels, and rstd amplifies the 16-bit inputs' exact difference; no extra error
    _near(x.grad, xr.grad, dt, 1, 1e-4)
    _near(r.grad, rr.grad, dt, 1)
    gg, bg = (g.main_grad - 3.0, b.main_grad + 1.0) if flat else (g.grad, b.grad)
    _near(gg, gr.grad, dt, 0, 1e-5)
    _near(bg, br.grad, dt, 0, 1e-5)


@pytest.mark.parametrize("tile_n", [64, 128, 256])
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (130, 72, 200), (257, 520, 1032), (640, 1160, 72)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False), (True, True)])
def test_gemm_tile_widths(tile_n, M, N, K, trans_a, trans_b):
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(5)
    dt = torch.bfloat16
    lead = lambda n: (n + 7) // 8 * 8  # noqa: E731
    a = torch.randn((K, lead(M)) if trans_a else (M, K), device="cuda").to(dt)
    a = a[:, :M] if trans_a else a
    b = torch.randn((N, K) if trans_b else (K, N), device="cuda").to(dt)
    ref = (a.double().t() if trans_a else a.double()) @ (b.double().t() if trans_b else b.double())
    _near(gemm(a, b, trans_a=trans_a, trans_b=trans_b, tile_n=tile_n), ref, dt, 1)
    acc = torch.ones(M, N, device="cuda")
    gemm(a, b, trans_a=trans_a, trans_b=trans_b, out=acc, accumulate=True, tile_n=tile_n)
    _near(acc, ref + 1.0, dt, 0)
    # many tiles per CTA: every stage and both accumulators wrap
    few = torch.empty(M, N, device="cuda", dtype=dt)
    gemm(a, b, trans_a=trans_a, trans_b=trans_b, out=few, tile_n=tile_n, max_ctas=2)
    _near(few, ref, dt, 1)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (2, 127, 3), (5, 129, 7), (9, 200, 20), (7, 384, 16), (4, 513, 12)])
@pytest.mark.parametrize("p", [0.0, 0.25])
def test_attention_backward_blocks(B, S, H, p):
    """One, two and more query and key blocks, ragged last blocks, key bias, dropout."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import kernels as K

    torch.manual_seed(4)
    dt = torch.bfloat16
    qkv = torch.randn(B, S, 3, H, 64, device="cuda").to(dt)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    bias = torch.zeros(B, S, device="cuda")
    bias[:, S - S // 5:] = -10000.0
    drop = dict(p_drop=p, seed=5, offset=9)
    mask = torch.ones(B, H, S, S, device="cuda", dtype=torch.float64)
    if p:
        # uniform attention over one-hot values reads the mask out, 64 keys at a time
        z = torch.zeros(B, S, H, 64, device="cuda", dtype=dt)
        for w in range(0, S, 64):
            n = min(64, S - w)
            one = z.clone()
            one[:, w:w + n, :, :n] = torch.eye(n, device="cuda", dtype=dt)[None, :, None]
            mask[:, :, :, w:w + n] = (K.attn_fwd(z, z, one, **drop)[0][..., :n] > 0).permute(0, 2, 1, 3).double()
        mask /= 1 - p
    o, lse = K.attn_fwd(q, k, v, key_bias=bias, **drop)
    qr, kr, vr = (t.double().detach().requires_grad_(True) for t in (q, k, v))
    sc = torch.einsum("bqhd,bkhd->bhqk", qr, kr) / 8 + bias.double()[:, None, None]
    ref = torch.einsum("bhqk,bkhd->bqhd", sc.softmax(-1) * mask, vr)
    do = torch.randn(B, S, H, 64, device="cuda").to(dt)
    ref.backward(do.double())
    dq, dk, dv = K.attn_bwd(q, k, v, o, lse, do, key_bias=bias, **drop)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0
    # probabilities and their gradients are rounded to 16 bits before the products, O before delta: a few roundings of
    # terms as large as the largest result.  dP - delta cancels (down to nothing for a single key), so what is rounded
    # has the scale of dP, which dV's terms show and dQ itself need not.
    scale = max(t.grad.abs().max().item() for t in (qr, kr, vr)) + 1e-3
    for got, want in ((dq, qr.grad), (dk, kr.grad), (dv, vr.grad)):
        err = (got.double() - want).abs().max().item() / scale
        assert err < 6 * U[dt], err


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tile_n", [0, 64, 128])
@pytest.mark.parametrize("M,N,K", [(2, 40, 1), (72, 8, 63), (130, 520, 200), (1160, 264, 1032), (4104, 1032, 2056),
                                   (1024, 1024, 16384)])
def test_gemm_column_sums_beside_weight_gradient(dtype, tile_n, M, N, K):
    """Every row of dy is added exactly once, whichever tile, split and kernel variant does it."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(7)
    dy = torch.zeros(K, (M + 7) // 8 * 8, device="cuda", dtype=dtype)[:, :M]
    dy.copy_(torch.randn(K, M, device="cuda"))
    x = torch.randn(K, N, device="cuda").to(dtype)
    want, ref = dy.double().sum(0), dy.double().t() @ x.double()
    for kw in (dict(out=torch.ones(M, N, device="cuda"), accumulate=True), dict()):
        db = torch.full((M,), 2.0, device="cuda")
        out = gemm(dy, x, trans_a=True, trans_b=False, tile_n=tile_n, a_colsum=db, **kw)
        torch.cuda.synchronize()
        assert _lib.read_error() == 0
        steps = K / 16 * 2.0 ** -23
        _near(db - 2.0, want, dtype, 0, steps)
        _near(out, ref + (1.0 if kw else 0.0), dtype, 0 if kw else 1, steps)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,K,N", [(2047, 264, 136), (2048, 264, 136), (4500, 1032, 520), (2304, 768, 768)])
def test_linear_weight_gradient_both_sides_of_the_split(dtype, rows, K, N):
    """Weight gradients of the parameter's own type, as one product and as split sums rounded at the end."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF

    torch.manual_seed(8)
    x = torch.randn(rows, K, device="cuda").to(dtype)
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).to(dtype).requires_grad_(True)
    b = torch.randn(N, device="cuda").to(dtype).requires_grad_(True)
    dy = torch.randn(rows, N, device="cuda").to(dtype)
    RF.linear(x, w, b).backward(dy)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0
    steps = rows / 16 * 2.0 ** -23
    _near(w.grad, dy.double().t() @ x.double(), dtype, 1, steps)
    _near(b.grad, dy.double().sum(0), dtype, 1, steps)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,tile_n,max_ctas", [(160, 256, 2), (160, 0, 2), (416, 256, 3), (96, 128, 2), (32, 64, 1), (160, 0, 0)])
def test_staged_blocks_of_many_tiles(dtype, N, tile_n, max_ctas):
    """Tiles with an odd number of 32-column blocks per warp, many to a CTA and with short main loops: the two halves of the
    staging memory must keep taking turns across tiles, or a block is overwritten while the copy engine reads it.  Every
    value is a small whole number, so a block of another tile is seen exactly."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm

    M, K = 128 * 300 + 5, 64
    torch.manual_seed(9)
    a = torch.zeros(M, K, device="cuda", dtype=dtype)
    a[:, :8] = torch.randint(-3, 4, (M, 8), device="cuda").to(dtype)
    b = torch.randint(-3, 4, (N, K), device="cuda").to(dtype)
    want = (a.float() @ b.float().t()).to(dtype)
    for _ in range(5):
        assert torch.equal(gemm(a, b, tile_n=tile_n, max_ctas=max_ctas), want)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,tile_n,max_ctas", [(160, 256, 2), (416, 0, 6), (96, 128, 2), (40, 64, 1), (200, 0, 0)])
def test_activation_blocks_of_many_tiles(dtype, N, tile_n, max_ctas):
    """Sixteen epilogue warps with one staging block each: the value before the activation, the one behind it and the
    gradient's operand share the block's place, over many tiles.  The first is a small whole number and seen exactly; the
    derivative of GELU at +-30 is exactly 1 or 0, so a foreign operand block is seen exactly too."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm

    M, K = 128 * 300 + 5, 64
    torch.manual_seed(9)
    a = torch.zeros(M, K, device="cuda", dtype=dtype)
    a[:, :8] = torch.randint(-3, 4, (M, 8), device="cuda").to(dtype)
    b = torch.randint(-3, 4, (N, K), device="cuda").to(dtype)
    z = a.float() @ b.float().t()
    aux = torch.where(torch.rand(M, N, device="cuda") < 0.5, 30.0, -30.0).to(dtype)
    for _ in range(3):
        pre = torch.empty(M, N, device="cuda", dtype=dtype)
        y = gemm(a, b, gelu=True, aux_out=pre, tile_n=tile_n, max_ctas=max_ctas)
        assert torch.equal(pre, z.to(dtype))
        _near(y, torch.nn.functional.gelu(z.double()), dtype, 1)
        got = gemm(a, b, dgelu=True, aux_in=aux, tile_n=tile_n, max_ctas=max_ctas)
        assert torch.equal(got, torch.where(aux > 0, z, torch.zeros_like(z)).to(dtype))
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


# 74 pairs of SMs and 76 (2 left over), 111 (37), 112 (38: two rounds of helpers), 124 (50: three), 136 (62: six), 147 (73)
# and 150 (2) tiles; in `how` many parts the last wave is summed: see ops.gemm.last_wave
@pytest.mark.parametrize("M,N,K,how", [
    (4864, 1024, 448, 0), (4864, 1024, 600, 2), (4864, 1024, 1560, 5), (9472, 768, 1000, 0), (9472, 768, 1560, 2),
    (3500, 2048, 1560, 1), (1000, 7930, 2560, 1), (2041, 4352, 4090, 1), (5376, 1792, 1560, 0), (3833, 2552, 600, 0),
    (3833, 2552, 1560, 5)])
def test_gemm_last_wave_is_shared_out(M, N, K, how):
    """Tiles of the last wave in parts, beside whole ones: small integers, so that every order of adding is exact."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import gemm, last_wave

    assert last_wave(M, N, K) == how and last_wave(M, N, K, in_order=True) == 0
    g = torch.Generator(device="cuda").manual_seed(M + K)
    dt = torch.bfloat16
    a, b = (torch.randint(-3, 4, (K, n), generator=g, device="cuda").to(dt) for n in ((M + 7) // 8 * 8, (N + 7) // 8 * 8))
    a, b = a[:, :M], b[:, :N]
    want = a.double().t() @ b.double()
    buf = torch.full((M + 1, N + 4), 5.0, device="cuda")
    sums = torch.full((M,), 2.0, device="cuda")
    gemm(a, b, trans_a=True, trans_b=False, out=buf[:M, :N], accumulate=True, a_colsum=sums)
    assert torch.equal(buf[:M, :N].double(), want + 5.0) and (buf[M:] == 5.0).all() and (buf[:, N:] == 5.0).all()
    assert torch.equal(sums.double(), a.double().sum(0) + 2.0)
    # added whole when asked: the same bits every time
    x, y = torch.randn(K, M, device="cuda").to(dt), torch.randn(K, N, device="cuda").to(dt)
    torch.use_deterministic_algorithms(True)
    try:
        outs = []
        for _ in range(4):
            out = torch.full((M, N), 1e3, device="cuda")
            gemm(x, y, trans_a=True, trans_b=False, out=out, accumulate=True)
            outs.append(out)
        assert all(torch.equal(o, outs[0]) for o in outs)
    finally:
        torch.use_deterministic_algorithms(False)
    assert _lib.read_error() == 0


@pytest.mark.parametrize("rows,S", [(96, 48), (384, 192), (6144, 512)])
def test_kernels_in_a_row_wait_for_each_other(rows, S):
    """Kernels that begin beside the end of the one before them, over buffers that are written again and again, with a
    PyTorch kernel in between: the same bits as with the device idle before every launch."""
    from rannc_b200.ops import kernels as K
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(3)
    dt, H = torch.bfloat16, 256
    w = [(torch.randn(3 * H, H, device="cuda") * H ** -0.5).to(dt), (torch.randn(H, H, device="cuda") * H ** -0.5).to(dt)]
    g, b = torch.ones(H, device="cuda", dtype=dt), torch.zeros(H, device="cuda", dtype=dt)
    x0 = torch.randn(rows, H, device="cuda").to(dt)

    def run(idle):
        sync = torch.cuda.synchronize if idle else (lambda: None)
        x, qkv, y = x0.clone(), torch.empty(rows, 3 * H, device="cuda", dtype=dt), torch.empty_like(x0)
        out = []
        for step in range(12):
            gemm(x, w[0], out=qkv)
            sync()
            q, k, v = (qkv.view(rows // S, S, 3, 4, 64)[:, :, i] for i in range(3))
            o, lse = K.attn_fwd(q, k, v)
            sync()
            gemm(o.view(rows, H), w[1], out=y)
            sync()
            z, zin, mean, rstd = K.ln_fwd(y, x, g, b, 1e-5)
            sync()
            if step % 3 == 2:
                z = z * 0.5
                sync()
            dx, dz, dg, db = K.ln_bwd(z, zin, g, mean, rstd)
            sync()
            dq, dk, dv = K.attn_bwd(q, k, v, o, lse, dx.view(rows // S, S, 4, 64))
            sync()
            x.copy_(z) if step % 2 else gemm(z, w[1], out=x)
            sync()
            out += [x.clone(), dk.clone(), dv.clone(), dz.clone()]   # (dQ and the parameters' sums: added as they arrive)
        return out

    for a, c in zip(run(True), run(False)):
        assert torch.equal(a, c)


@pytest.mark.parametrize("how", ["captured", "two_streams"])
def test_kernels_in_a_row_under_capture_and_across_streams(how):
    """The order that a captured graph, or an event between two streams, asks for holds for kernels that begin early."""
    from rannc_b200.ops import kernels as K
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(4)
    dt, H, rows = torch.bfloat16, 512, 2048
    w = (torch.randn(H, H, device="cuda") * H ** -0.5).to(dt)
    g, b = torch.ones(H, device="cuda", dtype=dt), torch.zeros(H, device="cuda", dtype=dt)
    x0 = torch.randn(rows, H, device="cuda").to(dt)
    x, y = x0.clone(), torch.empty_like(x0)
    other = torch.cuda.Stream()

    def step(two):
        """x = layer_norm(x w^T): the product on this stream, the norm on the other one when there are two."""
        gemm(x, w, out=y)
        here = torch.cuda.current_stream()
        if two:
            other.wait_stream(here)
        with torch.cuda.stream(other if two else here):
            z = K.ln_fwd(y, None, g, b, 1e-5)[0]
            gemm(z, w, out=x)
            z.record_stream(other)
        if two:
            here.wait_stream(other)

    for _ in range(6):
        step(False)
        torch.cuda.synchronize()
    want = x.clone()
    x.copy_(x0)
    torch.cuda.synchronize()
    if how == "captured":
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            step(False)
        torch.cuda.synchronize()
        x.copy_(x0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(3):
                step(False)
        for _ in range(2):
            graph.replay()
    else:
        for _ in range(6):
            step(True)
    torch.cuda.synchronize()
    assert torch.equal(x, want)


@pytest.mark.parametrize("captured", [False, True])
def test_kernels_that_begin_early_on_streams_beside_each_other(captured):
    """Chains of such kernels on two streams at once, each over its own buffers: blocks of one stream wait on the device in
    places that kernels of the other want.  The same bits as one chain after the other; captured, the streams fork and
    join inside the graph."""
    from rannc_b200.ops import kernels as K
    from rannc_b200.ops.gemm import gemm

    torch.manual_seed(6)
    dt, H, S = torch.bfloat16, 256, 192
    w = [(torch.randn(3 * H, H, device="cuda") * H ** -0.5).to(dt), (torch.randn(H, H, device="cuda") * H ** -0.5).to(dt)]
    g, b = torch.ones(H, device="cuda", dtype=dt), torch.zeros(H, device="cuda", dtype=dt)
    start = [torch.randn(rows, H, device="cuda").to(dt) for rows in (5 * S, 24 * S)]
    sums = [torch.zeros(3 * H, H, device="cuda") for _ in start]
    xs = [x.clone() for x in start]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    kept = []

    def chain(i, steps):
        x, rows = xs[i], xs[i].shape[0]
        for _ in range(steps):
            qkv = gemm(x, w[0])
            q, k, v = (qkv.view(rows // S, S, 3, 4, 64)[:, :, j] for j in range(3))
            o, lse = K.attn_fwd(q, k, v)
            z, zin, mean, rstd = K.ln_fwd(gemm(o.view(rows, H), w[1]), x, g, b, 1e-5)
            dz = K.ln_bwd(z, zin, g, mean, rstd)[1]
            dv = K.attn_bwd(q, k, v, o, lse, dz.view(rows // S, S, 4, 64))[2]
            gemm(qkv, dv.reshape(rows, H), trans_a=True, trans_b=False, out=sums[i], accumulate=True)
            x.copy_(z)
            kept.extend((qkv, o, lse, z, zin, mean, rstd, dz, dv))

    def both(steps):
        here = torch.cuda.current_stream()
        for i, s in enumerate(streams):
            s.wait_stream(here)
            with torch.cuda.stream(s):
                chain(i, steps)
        for s in streams:
            here.wait_stream(s)

    for i in range(2):
        chain(i, 6)
    torch.cuda.synchronize()
    want, want_sums = [x.clone() for x in xs], [s.clone() for s in sums]
    for x, x0, s in zip(xs, start, sums):
        x.copy_(x0)
        s.zero_()
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            both(3)
        for _ in range(2):
            graph.replay()
    else:
        both(6)
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(xs, want))
    for s, y in zip(sums, want_sums):   # (K is split: added as it arrives)
        assert (s - y).norm() <= 1e-5 * y.norm()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H", [256, 768, 1024, 2048, 4096])
@pytest.mark.parametrize("leaf", ["both", "x", "residual", "none"])
def test_layernorm_gradients_of_two_inputs(dtype, H, leaf):
    """Without dropout both inputs have the same gradient: written twice where one of them is a leaf, else one tensor."""
    from rannc_b200.ops import functional as RF

    torch.manual_seed(4)
    x, r = (torch.randn(13, H, device="cuda").to(dtype).requires_grad_(True) for _ in range(2))
    g, b = (torch.randn(H, device="cuda").to(dtype).requires_grad_(True) for _ in range(2))
    dy = torch.randn(13, H, device="cuda").to(dtype)
    RF.dropout_add_layer_norm(x if leaf in ("both", "x") else x * 1, r if leaf in ("both", "residual") else r * 1, g, b, 0.0,
                              1e-5).backward(dy)
    z = (x.detach() + r.detach()).double().requires_grad_(True)
    torch.nn.functional.layer_norm(z, (H,), g.double(), b.double(), 1e-5).backward(dy.double())
    assert torch.equal(x.grad, r.grad)
    assert leaf != "both" or x.grad.data_ptr() != r.grad.data_ptr()
    # z is rounded to 16 bits before it is normalised: one rounding more than the result's own
    _near(x.grad, z.grad, dtype, 1, 4 * U[dtype])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 351, 3000])
def test_activation_without_a_graph(dtype, rows):
    """Under no_grad the value before the activation is not written: the result is the same."""
    from rannc_b200.ops import functional as RF

    torch.manual_seed(5)
    x = torch.randn(rows, 264, device="cuda").to(dtype)
    w, v = (torch.randn(n, m, device="cuda").mul(0.1).to(dtype).requires_grad_(True) for n, m in ((520, 264), (264, 520)))
    b, c = (torch.randn(n, device="cuda").to(dtype).requires_grad_(True) for n in (520, 264))
    with torch.no_grad():
        got = RF.linear(x, w, b, act="gelu"), RF.mlp(x, w, b, v, c)
    assert torch.equal(got[0], RF.linear(x, w, b, act="gelu")) and torch.equal(got[1], RF.mlp(x, w, b, v, c))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,S,H,p", [(20, 128, 16, 0.0), (23, 100, 16, 0.2), (11, 200, 16, 0.2), (5, 300, 16, 0.0),
                                     (7, 512, 16, 0.2), (40, 33, 16, 0.0)])
def test_attention_backward_over_many_items(dtype, B, S, H, p):
    """Several blocks of 128 keys to a CTA, one after the other: of one to five query blocks, whole and ragged.  Each (batch,
    head) by itself gives the same bits in dK and dV; dQ is added up in whichever order the key blocks come."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import kernels as K

    torch.manual_seed(11)
    q, k, v, do = (torch.randn(B, S, H, 64, device="cuda").to(dtype) for _ in range(4))
    bias = torch.where(torch.rand(B, S, device="cuda") < 0.2, -10000.0, 0.0)
    bias[:, 0] = 0.0
    o, lse = K.attn_fwd(q, k, v, bias, 0.125, p, 3, 4)
    dq, dk, dv = K.attn_bwd(q, k, v, o, lse, do, bias, 0.125, p, 3, 4)
    assert _lib.read_error() == 0
    sc = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / 8 + bias.double()[:, None, None]
    if p == 0.0:
        P = sc.softmax(-1)
        dP = torch.einsum("bqhd,bkhd->bhqk", do.double(), v.double())
        dS = P * (dP - (P * dP).sum(-1, keepdim=True))
        want = (torch.einsum("bhqk,bkhd->bqhd", dS, k.double()) / 8, torch.einsum("bhqk,bqhd->bkhd", dS, q.double()) / 8,
                torch.einsum("bhqk,bqhd->bkhd", P, do.double()))
        scale = max(w.abs().max().item() for w in want)
        for got, w in zip((dq, dk, dv), want):     # (as in test_attention_backward_blocks)
            assert (got.double() - w).abs().max().item() / scale < 6 * U[dtype]
    for b in (0, B // 2, B - 1):
        # dropout depends on a row's place in the whole batch: without it a batch row by itself is the same problem
        if p == 0.0:
            r = slice(b, b + 1)
            _, dk1, dv1 = K.attn_bwd(q[r], k[r], v[r], o[r], lse[r], do[r], bias[r].contiguous(), 0.125, p, 3, 4)
            assert torch.equal(dk1, dk[r]) and torch.equal(dv1, dv[r])
    # the same call again: no state is left behind
    dq2, dk2, dv2 = K.attn_bwd(q, k, v, o, lse, do, bias, 0.125, p, 3, 4)
    assert torch.equal(dk, dk2) and torch.equal(dv, dv2)
    assert (dq.float() - dq2.float()).abs().max().item() <= 2 * U[dtype] * dq.float().abs().max().item()
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S", [64, 200, 256, 512, 1024, 1100])
@pytest.mark.parametrize("p", [0.0, 0.25])
def test_attention_forward_bias_by_64_keys(dtype, S, p):
    """Blocks of 64 keys with, without and with nothing but padding, in every order: batch rows whose valid keys come first,
    last or between, one without a valid key, one with a bias that is no mask, and a key past which NaN and infinity hide
    behind the mask and must show."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import kernels as K

    torch.manual_seed(12)
    H = 3
    rows = torch.zeros(7, S, device="cuda")
    rows[0, S // 2:] = -10000.0
    rows[1, :S // 2] = -10000.0
    rows[2, :S // 3], rows[2, -(S // 3):] = -10000.0, torch.finfo(torch.float32).min
    rows[3] = -10000.0
    rows[4] = torch.randn(S, device="cuda")
    rows[5, -5:] = -10000.0
    B = rows.shape[0]
    q, k, v = (torch.randn(B, S, H, 64, device="cuda").to(dtype) for _ in range(3))
    keep = torch.ones(B, H, S, S, device="cuda", dtype=torch.float64)
    if p:
        z = torch.zeros_like(q)
        for w in range(0, S, 64):
            n = min(64, S - w)
            one = z.clone()
            one[:, w:w + n, :, :n] = torch.eye(n, device="cuda", dtype=dtype)[None, :, None]
            keep[:, :, :, w:w + n] = (K.attn_fwd(z, z, one, None, 0.125, p, 5, 9)[0][..., :n] > 0).permute(0, 2, 1, 3).double()
        keep /= 1 - p
    o, lse = K.attn_fwd(q, k, v, rows, 0.125, p, 5, 9)
    sc = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / 8 + rows.double()[:, None, None]
    want = torch.einsum("bhqk,bkhd->bqhd", sc.softmax(-1) * keep, v.double())
    # probabilities and the result are rounded once each; terms of the size of the largest value of v
    assert (o.double() - want).abs().max().item() <= 2 * U[dtype] * v.double().abs().max().item() / (1 - p) + 1e-4
    # (a row whose scores are all rounded away under the bias: 10000 log2(e) holds eleven binary places)
    assert (lse.double() - torch.logsumexp(sc, -1)).abs().max().item() <= 2.0 ** -9
    k2 = k.clone()
    k2[0, S - 1, 0] = float("nan")
    k2[1, 0, 1, 5] = float("inf")
    o2, _ = K.attn_fwd(q, k2, v, rows, 0.125, 0.0, 5, 9)
    o1, _ = K.attn_fwd(q, k, v, rows, 0.125, 0.0, 5, 9)
    assert o2[0, :, 0].isnan().all()
    assert o2[1, :, 1].isnan().any()     # (an infinite score beats the bias where it is positive)
    same = torch.ones(B, S, H, dtype=torch.bool, device="cuda")
    same[0, :, 0] = same[1, :, 1] = False
    assert torch.equal(o1[same], o2[same])
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 1031])
def test_vectors_moved_four_at_a_time(dtype, n):
    """n vectors of 16 bytes a row in the kernels that fetch four per thread before they store one: an embedding row, a
    padded row of an image, a row of the loss gradient (written over the logits and beside them)."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(13)
    table = torch.randn(9, 8 * n, device="cuda").to(dtype)
    ids = torch.tensor([0, 8, 3, 3, 7], device="cuda")
    assert torch.equal(K.embed_fwd(ids, table), table[ids])

    x = torch.randn(2, 3, n, 8, device="cuda").to(dtype)
    for pad in (0, 1, 2):
        assert torch.equal(K.pad_nhwc(x, pad), torch.nn.functional.pad(x, (0, 0, 0, pad, 0, pad)))

    V = 8 * n - 3     # padding inside the last vector
    logits = torch.randn(5, 8 * n, device="cuda").to(dtype)
    labels = torch.tensor([0, V - 1, -100, V // 2, -100], device="cuda")
    _, lse, acc = K.xent_fwd(logits, labels, V)
    gout = torch.full((), 1.5, device="cuda")
    apart = K.xent_bwd(logits, labels, lse, acc, gout, V, inplace=False)
    p = logits[:, :V].double().softmax(-1)
    p[torch.arange(5), labels.clamp(min=0)] -= 1
    want = torch.nn.functional.pad(p * (labels >= 0).double()[:, None] * (1.5 / 3), (0, 3))
    _near(apart, want, dtype, 1)
    assert torch.equal(K.xent_bwd(logits, labels, lse, acc, gout, V), apart)


@pytest.mark.parametrize("R,C", [(1, 8), (3, 24), (37, 72), (4 * 148 + 1, 2048), (5003, 264)])
@pytest.mark.parametrize("relu,res", [(False, False), (True, True)])
def test_batch_norm_rows_two_at_a_time(R, C, relu, res):
    """Odd numbers of rows per thread, in a chain of launches whose sums start from memory that held NaN."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(14)
    dtype = torch.bfloat16
    x, dy = (torch.randn(R, C, device="cuda").to(dtype) for _ in range(2))
    r = torch.randn(R, C, device="cuda").to(dtype) if res else None
    g, b = torch.rand(C, device="cuda") + 0.5, torch.randn(C, device="cuda")
    for _ in range(2):
        junk = [torch.full((n, C), float("nan"), device="cuda") for n in (2, 4, 6) for _ in range(3)]
        del junk   # (the next allocations of this size get that memory)
        y, mean, rstd = K.bn_fwd(x, r, g, b, None, None, 1e-5, 0.1, relu)
    xd = x.double()
    var = xd.var(0, unbiased=False)
    xhat = (xd - xd.mean(0)) / (var + 1e-5).sqrt()
    want = xhat * g + b + (r.double() if res else 0)
    want = want.relu() if relu else want
    # sums of squares in fp32: the variance of rows that hardly differ (R = 1: exactly none) loses 2^-22 of the mean square
    slack = 0.0 if R == 1 else 1e-4
    if R > 1:
        _near(y, want, dtype, 1, slack)
    else:
        _near(y, (b.double() + (r.double() if res else 0)).relu() if relu else b.double().expand(1, C), dtype, 1, 1e-4)
    dx, dres, dgamma, dbeta = K.bn_bwd(x, dy, y, mean, rstd, g, relu, res)
    gd = torch.where(y > 0, dy, torch.zeros_like(dy)).double() if relu else dy.double()
    _near(dbeta, gd.sum(0), dtype, 0, 1e-5)
    if res:
        assert torch.equal(dres.double(), gd)
    if R > 30:
        _near(dgamma, (gd * xhat).sum(0), dtype, 0, 1e-4)
        _near(dx, (gd - gd.mean(0) - xhat * (gd * xhat).mean(0)) * g / (var + 1e-5).sqrt(), dtype, 1, 1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("Co,Ci", [(1, 8), (5, 72), (3, 256), (2, 264), (7, 1032)])
def test_weight_gradient_of_small_filters_folded(dtype, k, Co, Ci):
    """Chunks of 256 channels and what is left of them, to the bit; a destination off a 16-byte boundary and a channel count
    that is no multiple of 8 take the strided operation."""
    from rannc_b200.ops import functional as RF

    torch.manual_seed(15)
    for ci, off in ((Ci, 0), (Ci, 1), (Ci + 4, 0)):
        n = Co * ci * k * k
        dw2 = torch.randn(Co, k * k * ci, device="cuda")
        want = dw2.view(Co, k, k, ci).permute(0, 3, 1, 2)
        mg = torch.full((n + 9,), 0.5, device="cuda", dtype=dtype)
        dst = mg[off:off + n].view(Co, ci, k, k)
        fast = off == 0 and ci % 8 == 0
        assert RF.K.wgrad_fold_few_ok(dst) == fast
        if dtype == torch.float32:
            assert RF._Conv2d._fold(dw2, dst, dst, k) is None
            assert torch.equal(dst, 0.5 + want)
        else:
            assert torch.equal(RF._Conv2d._fold(dw2, dst, None, k), want.to(dtype))
            if fast:
                RF.K.wgrad_fold_few(dw2, dst, k * k)
                assert torch.equal(dst, want.to(dtype))
        assert (mg[:off] == 0.5).all() and (mg[off + n:] == 0.5).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k", [2, 3, 5])
@pytest.mark.parametrize("Co,Ci", [(1, 8), (5, 72), (3, 256), (2, 264), (7, 1032)])
def test_filters_packed_by_tap(dtype, k, Co, Ci):
    """Chunks of 256 channels and what is left of them, to the bit."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(16)
    w = torch.randn(Co, Ci, k, k, device="cuda").to(dtype)
    assert torch.equal(K.pack_taps(w), w.permute(0, 2, 3, 1).reshape(Co, -1))


@pytest.mark.parametrize("how", ["captured", "two_streams"])
def test_small_kernels_in_a_row_under_capture_and_across_streams(how):
    """Lookup, batch norm, loss and their gradients, each of which begins beside the end of the one before, in a captured
    graph and with every other kernel on a second stream: what came before is complete."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(17)
    dt, C, rows = torch.bfloat16, 1024, 3001
    table = torch.randn(64, C, device="cuda").to(dt)
    ids, labels = (torch.randint(0, n, (rows,), device="cuda") for n in (64, C))
    g, b, gout = torch.rand(C, device="cuda") + 0.5, torch.randn(C, device="cuda"), torch.ones((), device="cuda")
    dtable = torch.zeros(64, C, device="cuda")
    other = torch.cuda.Stream()

    def step(two):
        here = torch.cuda.current_stream()
        kept = []

        def on_other(f):
            if two:
                other.wait_stream(here)
            with torch.cuda.stream(other if two else here):
                out = f()
            if two:
                here.wait_stream(other)
            kept.append(out)   # (alive until both streams are done)
            return out

        dtable.zero_()
        e = K.embed_fwd(ids, table)
        y, mean, rstd = on_other(lambda: K.bn_fwd(e, None, g, b, None, None, 1e-5, 0.1, False))
        loss, lse, acc = K.xent_fwd(y, labels, C)
        dy = on_other(lambda: K.xent_bwd(y, labels, lse, acc, gout, C, inplace=False))
        dx = K.bn_bwd(e, dy, y, mean, rstd, g, False, False)[0]
        on_other(lambda: K.embed_bwd(ids, dx, dtable))
        kept.append((e, lse, acc, dx))
        return loss, kept

    t = table.double().requires_grad_(True)
    e = t[ids]
    y = torch.nn.functional.batch_norm(e, None, None, g.double(), b.double(), True, 0.1, 1e-5)
    want = torch.nn.functional.cross_entropy(y, labels)
    want.backward()
    if how == "captured":
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            step(False)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            loss, kept = step(False)
        for _ in range(3):
            graph.replay()
    else:
        for _ in range(3):
            loss, kept = step(True)
    torch.cuda.synchronize()
    # y, dy and dx are rounded once each, and alike for all tokens of one id: rounding y by U |y| changes its probability by
    # that factor, dy and dx add U each, and one more covers the sums
    assert abs(float(loss) - want.item()) <= U[dt] * want.item()
    scale = t.grad.abs().max()
    assert (dtable.double() - t.grad).abs().max() <= (y.abs().max() + 3) * U[dt] * scale


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S", [1, 31, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("B,H", [(75, 2), (80, 3), (40, 7), (20, 16)])
def test_attention_forward_two_heads_a_block(dtype, S, B, H):
    """Short sequences with more heads than SMs: two heads to a block (an odd number leaves one alone), to the bit what each
    batch row gives by itself, where a block has one head."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import kernels as K

    torch.manual_seed(18)
    q, k, v = (t for t in torch.randn(B, S, 3, H, 64, device="cuda").to(dtype).unbind(2))
    bias = torch.zeros(B, S, device="cuda")
    bias[1::2, S // 2 + 1:] = -10000.0
    for kb, p in ((None, 0.0), (bias, 0.0), (bias, 0.25)):
        o, lse = K.attn_fwd(q, k, v, kb, 0.125, p, 3, 4)
        for b in range(B) if p == 0 else (0,):   # (a row's dropout depends on its place in the batch)
            one = slice(b, b + 1)
            o1, lse1 = K.attn_fwd(q[one], k[one], v[one], None if kb is None else kb[one].contiguous(), 0.125, p, 3, 4)
            assert torch.equal(o1, o[one]) and torch.equal(lse1, lse[one])
    sc = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / 8 + bias.double()[:, None, None]
    o, _ = K.attn_fwd(q, k, v, bias, 0.125, 0.0, 3, 4)
    want = torch.einsum("bhqk,bkhd->bqhd", sc.softmax(-1), v.double())
    # probabilities and the result are rounded once each
    assert (o.double() - want).abs().max().item() <= 2 * U[dtype] * v.double().abs().max().item() + 1e-4
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("S", [1, 33, 64, 100, 127, 128, 129])
@pytest.mark.parametrize("B,H", [(1, 1), (3, 4), (40, 7)])
def test_attention_backward_of_one_key_block(dtype, S, B, H):
    """dQ of a sequence of one key block is stored as it is made: into a part of a packed gradient whose other parts stay as
    they are, and with strides of its own.  One key more goes by way of the sums."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import kernels as K

    torch.manual_seed(19)
    q, k, v = (t for t in torch.randn(B, S, 3, H, 64, device="cuda").to(dtype).unbind(2))
    do = torch.randn(B, S, H, 64, device="cuda").to(dtype)
    bias = torch.zeros(B, S, device="cuda")
    bias[::2, S // 2 + 1:] = -10000.0
    o, lse = K.attn_fwd(q, k, v, bias, 0.125)
    packed = torch.full((B, S, 4, H, 64), 3.0, device="cuda", dtype=dtype)
    K.attn_bwd(q, k, v, o, lse, do, bias, 0.125, dq=packed[:, :, 0], dk=packed[:, :, 1], dv=packed[:, :, 2])
    assert (packed[:, :, 3] == 3.0).all()
    flipped = torch.full((H, B, S + 1, 72), 3.0, device="cuda", dtype=dtype)   # heads outermost, rows 72 apart
    dq = flipped.permute(1, 2, 0, 3)[:, :S, :, :64]
    K.attn_bwd(q, k, v, o, lse, do, bias, 0.125, dq=dq)
    assert (flipped[:, :, S] == 3.0).all() and (flipped[..., 64:] == 3.0).all()
    if S <= 128:
        assert torch.equal(dq, packed[:, :, 0])
    qd, kd, vd = (t.double().requires_grad_(True) for t in (q, k, v))
    sc = torch.einsum("bqhd,bkhd->bhqk", qd, kd) / 8 + bias.double()[:, None, None]
    torch.einsum("bhqk,bkhd->bqhd", sc.softmax(-1), vd).backward(do.double())
    for got, want in zip(packed.unbind(2), (qd.grad, kd.grad, vd.grad)):
        # o, the probabilities and the gradients of the scores are rounded, each sum's terms with errors of both signs
        bound = 6 * U[dtype] * max(1.0, want.abs().max().item())
        assert (got.double() - want).abs().max().item() <= bound
    torch.cuda.synchronize()
    assert _lib.read_error() == 0


@pytest.mark.parametrize("H", [256, 768, 2048])
@pytest.mark.parametrize("std,scale,eps", [(1.0, 1.0, 1e-5), (2.0 ** 58, 1e-4, 1e-5), (2.0 ** -58, 2.0 ** 20, 0.0)])
def test_layer_norm_backward_of_rows_far_from_one(H, std, scale, eps):
    """Rows whose reciprocal deviation is in fp32's range and its square, times a gradient, is not."""
    from rannc_b200.ops import kernels as K

    torch.manual_seed(31)
    z = (torch.randn(37, H, device="cuda") * std).bfloat16()
    dy = (torch.randn(37, H, device="cuda") * scale).bfloat16()
    g = (torch.rand(H, device="cuda") + 0.5).bfloat16()
    b = torch.zeros_like(g)
    y, _, mean, rstd = K.ln_fwd(z, None, g, b, eps)
    dz, _, dgamma, dbeta = K.ln_bwd(dy, z, g, mean, rstd)
    zd, w = z.double(), dy.double() * g.double()
    r = 1.0 / (zd.var(1, unbiased=False, keepdim=True) + eps).sqrt()
    xh = (zd - zd.mean(1, keepdim=True)) * r
    want = r * (w - w.mean(1, keepdim=True) - xh * (w * xh).mean(1, keepdim=True))
    # one rounding to 16 bits, and fp32 sums of H terms
    bound = 2.0 ** -8 * want.abs() + 1e-5 * (r * w.abs().amax(1, keepdim=True))
    assert ((dz.double() - want).abs() <= bound).all()
    _near(dgamma, (dy.double() * xh).sum(0), torch.bfloat16, 0, 1e-4)
    _near(dbeta, dy.double().sum(0), torch.bfloat16, 0, 1e-4)


@pytest.mark.parametrize("native", [True, False])
def test_launches_are_counted_as_they_are(native):
    """Batch norm and attention backward, of one key block and of two, through the operators' host side and past it: what
    the library says it launched, and the kernels of its that the device ran."""
    from torch.profiler import ProfilerActivity, profile

    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF
    from rannc_b200.ops import kernels as K

    torch.manual_seed(32)
    img = torch.randn(2, 64, 8, 8, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    rows = torch.randn(128, 64, device="cuda").bfloat16()
    g = torch.ones(64, device="cuda", requires_grad=True)
    ws = [torch.randn(128, 128, device="cuda").bfloat16().requires_grad_(True) for _ in range(3)]
    qkv = [torch.randn(2, s, 2, 64, device="cuda").bfloat16() for s in (100, 200)]

    def work():
        if native:
            RF.batch_norm_act(img.clone().requires_grad_(True), g, torch.zeros_like(g), None, None).sum().backward()
            for s in (100, 200):
                x = torch.randn(2, s, 128, device="cuda").bfloat16()
                RF.qkv_attention(x, ws[0], None, ws[1], None, ws[2], None, num_heads=2).sum().backward()
        else:
            y, mean, rstd = K.bn_fwd(rows, None, g.detach(), g.detach(), None, None, 1e-5, 0.1, True)
            K.bn_bwd(rows, rows, y, mean, rstd, g.detach(), True, False)
            for t in qkv:
                o, lse = K.attn_fwd(t, t, t)
                K.attn_bwd(t, t, t, o, lse, t)

    work()
    torch.cuda.synchronize()
    before = _lib.launch_count()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        work()
        torch.cuda.synchronize()
    ran = sum(e.count for e in p.key_averages() if "rb::" in e.key)
    assert ran > 0 and _lib.launch_count() - before == ran


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_layernorm_of_one_leaf_twice(dtype):
    """Both inputs the same leaf: its gradient is twice that of either, whose one tensor the backward writes."""
    from rannc_b200.ops import functional as RF
    from rannc_b200.ops import kernels as K

    torch.manual_seed(33)
    x = torch.randn(37, 1024, device="cuda").to(dtype).requires_grad_(True)
    g, b = torch.randn(1024, device="cuda").to(dtype), torch.randn(1024, device="cuda").to(dtype)
    dy = torch.randn(37, 1024, device="cuda").to(dtype)
    RF.dropout_add_layer_norm(x, x, g, b, 0.0, 1e-5).backward(dy)
    y, z, mean, rstd = K.ln_fwd(x.detach(), x.detach(), g, b, 1e-5)
    dz = K.ln_bwd(dy, z, g, mean, rstd)[0]
    assert torch.equal(x.grad, dz + dz)
