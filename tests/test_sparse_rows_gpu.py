"""Backward of a wide output layer whose gradient has rows of zeros: found, gathered and put back on the device."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan(dy, x, room):
    from rannc_b200.ops import _lib

    R = dy.shape[0]
    i32 = dict(dtype=torch.int32, device="cuda")
    live, idx, pos, ctl = torch.empty(R, dtype=torch.uint8, device="cuda"), torch.full((room,), -7, **i32), \
        torch.full((R,), -7, **i32), torch.empty(2, **i32)
    code = 1 if dy.dtype == torch.bfloat16 else 0
    L = ctypes.c_longlong
    rc = _lib.lib().rb_rows_plan(_lib.vp(dy), L(dy.stride(0)), _lib.vp(x), L(x.stride(0)), R, dy.shape[1], x.shape[1], room,
                                 _lib.vp(live), _lib.vp(idx), _lib.vp(pos), _lib.vp(ctl), code, _lib.stream_ptr())
    assert rc == 0
    return idx, pos, ctl


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("R,V,H,room,count", [
    (1, 8, 8, 64, 1), (7, 264, 8, 64, 0), (130, 1304, 72, 64, 63), (130, 1304, 72, 64, 64), (1500, 264, 40, 1024, 1023),
    (3001, 1288, 264, 1024, 700), (5000, 520, 16, 4096, 5000)])
def test_rows_are_found_gathered_and_put_back(dtype, R, V, H, room, count):
    """Numbers of rows on both sides of a block, of the room and of a padded step; a row whose only value is its last; the
    matrix a slice of a wider one; a row of zeros whose input is not finite."""
    from rannc_b200.ops import _lib

    torch.manual_seed(R + count)
    wide = torch.randn(R, V + 16, device="cuda").to(dtype)
    dy, x = wide[:, 8:8 + V], torch.randn(R, H, device="cuda").to(dtype)
    on = torch.zeros(R, dtype=torch.bool, device="cuda")
    on[torch.randperm(R, device="cuda")[:count]] = True
    dy[~on] = 0
    rows = on.nonzero().flatten()
    if count > 2:
        dy[rows[0], :-1] = 0
        dy[rows[1]] = 0
        x[rows[1], H - 1] = float("nan")
        dy[rows[2]] = 0
        x[rows[2], 0] = float("-inf")
    idx, pos, ctl = _plan(dy, x, room)
    use = 0 < count < room
    assert ctl.tolist() == [count, int(use)]
    L = ctypes.c_longlong
    dyc, xc = torch.full((room, V), 3.0, device="cuda", dtype=dtype), torch.full((room, H), 3.0, device="cuda", dtype=dtype)
    d32 = torch.full((room, H), 3.0, device="cuda")
    assert _lib.lib().rb_rows_gather(_lib.vp(dy), L(dy.stride(0)), _lib.vp(x), L(H), V, H, _lib.vp(idx), _lib.vp(ctl),
                                     _lib.vp(dyc), _lib.vp(xc), _lib.vp(d32), _lib.stream_ptr()) == 0
    out = torch.full((R, H), 5.0, device="cuda", dtype=dtype)
    if use:
        assert torch.equal(idx[:count].long(), rows)
        want = torch.full((R,), -1, device="cuda")
        want[rows] = torch.arange(count, device="cuda")
        assert torch.equal(pos.long(), want)
        pad = (count + 64) // 64 * 64
        assert torch.equal(dyc[:count], dy[rows]) and torch.equal(xc[:count].nan_to_num(9.0), x[rows].nan_to_num(9.0))
        assert (dyc[count:pad] == 0).all() and (xc[count:pad] == 0).all() and (d32[:count + 1] == 0).all()
        assert (dyc[pad:] == 3.0).all() and (xc[pad:] == 3.0).all() and (d32[count + 1:] == 3.0).all()
        d32[:count + 1] = torch.randn(count + 1, H, device="cuda")
    assert _lib.lib().rb_rows_scatter(_lib.vp(d32), _lib.vp(out), R, H, _lib.vp(pos), _lib.vp(ctl),
                                      1 if dtype == torch.bfloat16 else 0, _lib.stream_ptr()) == 0
    if use:
        want = d32[count].to(dtype).expand(R, H).clone()
        want[rows] = d32[:count].to(dtype)
        assert torch.equal(out, want)
    else:
        assert (out == 5.0).all() and (dyc == 3.0).all() and (d32 == 3.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("share", [0.0, 0.0003, 0.15, 0.749, 0.9, 1.0])
@pytest.mark.parametrize("flat", [True, False])
def test_wide_layer_backward(dtype, share, flat):
    """Gradients against fp64, whichever form runs, at the smallest size that looks at the rows; sums added to what is there."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF

    R, H, V = 4099, 776, 28680
    torch.manual_seed(7)
    x = torch.randn(R, H, device="cuda").to(dtype).requires_grad_(True)
    w = (torch.randn(V, H, device="cuda") * 0.05).to(dtype).requires_grad_(True)
    b = torch.randn(V, device="cuda").to(dtype).requires_grad_(True)
    if flat:
        w.main_grad, b.main_grad = torch.full((V, H), 2.0, device="cuda"), torch.full((V,), -1.0, device="cuda")
    dy = torch.randn(R, V, device="cuda").to(dtype)
    on = torch.rand(R, device="cuda") < share
    on[-1] = share > 0
    dy[~on] = 0
    y = RF.linear(x, w, b)
    before = _lib.launch_count()
    y.backward(dy)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0
    # the look at the rows (three kernels), each product in two forms, and the one that puts rows back
    assert _lib.launch_count() - before == 8
    gw, gb = (w.main_grad - 2.0, b.main_grad + 1.0) if flat else (w.grad, b.grad)
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    n = int(on.sum())
    for got, want, terms, rounded in ((x.grad, dy.double() @ w.detach().double(), V, True),
                                      (gw, dy.double().t() @ x.detach().double(), n, not flat), (gb, dy.double().sum(0), n, not flat)):
        # one rounding of the result, a sum in steps of 16 terms that may lose 2^-23 of the running sum each, and (sums that
        # start at 2) the rounding of the sum so far
        bound = (u if rounded else 0.0) * want.abs() + (1e-5 + terms / 16 * 2.0 ** -23) * want.abs().max() + 1e-6
        assert ((got.double() - want).abs() <= bound).all()
    assert (x.grad[~on] == 0).all()


def test_infinities_and_nan_reach_the_gradients_of_rows_of_zeros():
    """0 * inf is NaN: a weight that is not finite shows in its column of every row's gradient, an input that is not finite in
    its column of the weight's, as in the product over all rows."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF

    R, H, V = 4096, 768, 30528
    torch.manual_seed(8)
    x, w, dy = (torch.randn(*s, device="cuda").bfloat16() for s in ((R, H), (V, H), (R, V)))
    dy[100:] = 0
    w[17, 5], w[400, 9] = float("inf"), float("nan")
    x[4000, 11] = float("inf")
    got = {}
    for all_rows in (False, True):
        xg, wg = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
        y = RF.linear(xg, wg)
        before = _lib.launch_count()
        torch.use_deterministic_algorithms(all_rows)     # (its products go over all rows)
        try:
            y.backward(dy)
        finally:
            torch.use_deterministic_algorithms(False)
        assert _lib.launch_count() - before == (2 if all_rows else 8)
        got[all_rows] = (xg.grad, wg.grad)
    for a, b in zip(got[False], got[True]):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    assert got[False][0][200].isnan().nonzero().flatten().tolist() == [5, 9]
    assert got[False][1][:, 11].isnan().all() and not got[False][1][:, 12].isnan().any()


def test_few_rows_of_many_inputs():
    """Less room than a step of 64 rows: the layer's backward goes over all of them."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF

    R, H, V = 85, 16384, 65536
    torch.manual_seed(9)
    x = torch.randn(R, H, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    w = torch.empty(V, H, device="cuda", dtype=torch.bfloat16).normal_(std=0.01).requires_grad_(True)
    dy = torch.randn(R, V, device="cuda", dtype=torch.bfloat16)
    dy[10:80] = 0
    RF.linear(x, w).backward(dy)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0
    u = 2.0 ** -8
    for got, a, b, terms in ((x.grad, dy, w.detach(), V), (w.grad[::97], dy.t()[::97], x.detach(), R)):
        want = a.double() @ b.double()
        bound = u * want.abs() + (1e-5 + terms / 16 * 2.0 ** -23) * want.abs().max() + 1e-6   # (as above)
        assert ((got.double() - want).abs() <= bound).all()
    assert (x.grad[10:80] == 0).all()


def _product(a, b, out, ctl, mode, flags, M, N, K, a_major, colsum=None, rows_out=0):
    """rb_gemm over gathered rows; returns its code."""
    from rannc_b200.ops import _lib
    from rannc_b200.ops.gemm import _Args

    g = _Args()
    g.A, g.B, g.D = a.data_ptr(), b.data_ptr(), out.data_ptr()
    g.M, g.N, g.K, g.batch = M, N, K, 1
    g.lda, g.ldb, g.ldd = a.stride(0), b.stride(0), out.stride(0)
    g.a_major, g.b_major = a_major, 1
    g.in_dtype = 1 if a.dtype == torch.bfloat16 else 0
    g.out_dtype = 1 if out.dtype == torch.float32 else 0
    g.flags, g.alpha = flags, 1.0
    g.a_colsum = None if colsum is None else colsum.data_ptr()
    g.rows_ctl, g.rows_mode, g.rows_out = ctl.data_ptr(), mode, rows_out
    return _lib.lib().rb_gemm(ctypes.byref(g), _lib.stream_ptr())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("V,H,room,count", [(264, 72, 64, 1), (520, 264, 128, 63), (520, 264, 128, 64), (264, 72, 128, 65),
                                            (1288, 520, 4096, 4095), (1288, 520, 4096, 2113)])
def test_weight_gradient_over_gathered_rows(dtype, fp32, V, H, room, count):
    """K counted on the device: the number of rows on both sides of a step, up to the room.  Few tiles, which an ordinary
    product added to fp32 would share out; the form that is not in use leaves everything as it is."""
    from rannc_b200.ops import _lib

    torch.manual_seed(room + count)
    dy, x = torch.randn(room, V, device="cuda").to(dtype), torch.randn(room, H, device="cuda").to(dtype)
    pad = (count + 64) // 64 * 64
    dy[count:pad] = 0
    x[count:pad] = 0
    dy[pad:] = float("nan")
    x[pad:] = float("nan")
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for use in (1, 0):
        ctl = torch.tensor([count, use], dtype=torch.int32, device="cuda")
        out = torch.full((V, H), 3.0, dtype=torch.float32 if fp32 else dtype, device="cuda")
        sums = torch.full((V,), 3.0, device="cuda")
        assert _product(dy, x, out, ctl, 2, 16 if fp32 else 0, V, H, room, 1, sums) == 0
        torch.cuda.synchronize()
        assert _lib.read_error() == 0
        if not use:
            assert (out == 3.0).all() and (sums == 3.0).all()
            continue
        d, e = dy[:count].double(), x[:count].double()
        for got, want in ((out.double() - (3.0 if fp32 else 0.0), d.t() @ e), (sums.double() - 3.0, d.sum(0))):
            # (as above; a column sum has no rounding of its own)
            bound = (0.0 if fp32 or got.dim() == 1 else u) * want.abs() + (1e-5 + count / 16 * 2.0 ** -23) * want.abs().max() + 1e-6
            assert ((got - want).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("V,H,room,count,rows_out", [(64, 8, 64, 1, 256), (1096, 264, 320, 255, 512), (1096, 264, 320, 256, 2048),
                                                     (4104, 520, 320, 319, 4096), (30528, 136, 704, 511, 16 * 512)])
def test_input_gradient_over_gathered_rows(dtype, V, H, room, count, rows_out):
    """M counted on the device: rows on both sides of a tile, with room for one part of K and for many; the parts, added up,
    are the gathered rows' gradients and that of a row of zeros, and the same to the bit every time."""
    from rannc_b200.ops import _lib

    torch.manual_seed(room + count)
    dy, w = torch.randn(room, V, device="cuda").to(dtype), torch.randn(V, H, device="cuda").to(dtype)
    dy[count:(count + 64) // 64 * 64] = 0
    dy[(count + 64) // 64 * 64:] = float("nan")
    rows = count + 5
    pos = torch.arange(rows, dtype=torch.int32, device="cuda") - 5        # (five rows that were left out)
    pos[:5] = -1
    code = 1 if dtype == torch.bfloat16 else 0
    first = None
    for use in (1, 1, 1, 0):
        ctl = torch.tensor([count, use, -9, -9], dtype=torch.int32, device="cuda")
        parts = torch.full((rows_out, H), 3.0, device="cuda")
        out = torch.full((rows, H), 5.0, dtype=dtype, device="cuda")
        assert _product(dy, w, parts, ctl, 3, 0, room, H, V, 0, rows_out=rows_out) == 0
        assert _lib.lib().rb_rows_scatter_parts(_lib.vp(parts), _lib.vp(out), rows, H, _lib.vp(pos), _lib.vp(ctl), code,
                                                _lib.stream_ptr()) == 0
        torch.cuda.synchronize()
        assert _lib.read_error() == 0
        if not use:
            assert (parts == 3.0).all() and (out == 5.0).all() and ctl.tolist() == [count, 0, -9, -9]
            continue
        n, apart = ctl[2:].tolist()
        assert apart == (count + 256) // 256 * 256 and 1 <= n * apart <= rows_out
        assert n > 1 or rows_out < 2 * apart or V < 512
        want = dy[:count].double() @ w.double()
        u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        bound = u * want.abs() + (1e-5 + V / 16 * 2.0 ** -23) * want.abs().max() + 1e-6   # (as above)
        assert ((out[5:].double() - want).abs() <= bound).all() and (out[:5] == 0).all()
        first = out.clone() if first is None else first
        assert torch.equal(out, first)
    assert _product(dy, w, parts, ctl, 3, 0, room, H, V, 0, rows_out=256 * ((room - 1) // 256)) == -10
    assert _product(dy, w, parts, ctl, 3, 16, room, H, V, 0, rows_out=rows_out) == -10


def test_wide_layer_backward_repeats_to_the_bit():
    from rannc_b200.ops import _lib
    from rannc_b200.ops import functional as RF

    R, H, V = 4099, 776, 28680
    torch.manual_seed(10)
    x = torch.randn(R, H, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    w = torch.randn(V, H, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    dy = torch.randn(R, V, device="cuda", dtype=torch.bfloat16)
    dy[torch.rand(R, device="cuda") >= 0.15] = 0
    first = None
    for _ in range(30):
        y = RF.linear(x, w)
        before = _lib.launch_count()
        got = torch.autograd.grad(y, (x, w), dy)
        assert _lib.launch_count() - before == 8        # (over the gathered rows)
        first = got if first is None else first
        assert torch.equal(got[0], first[0]) and torch.equal(got[1], first[1])


@pytest.mark.parametrize("flat", [True, False])
def test_backward_without_memory_for_the_gathered_rows(flat):
    """An allocator with room for the gradients alone: the products go over all rows, as under deterministic algorithms."""
    from rannc_b200.ops import functional as RF

    R, H, V = 4099, 776, 28680
    torch.manual_seed(11)
    x = torch.randn(R, H, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    w = torch.randn(V, H, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    dy = torch.randn(R, V, device="cuda", dtype=torch.bfloat16)
    dy[500:] = 0
    want = None
    for short in (False, True):
        if flat:
            w.main_grad = torch.zeros(V, H, device="cuda")
        x.grad = w.grad = None
        y = RF.linear(x, w)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        try:
            if short:
                reserved = torch.cuda.memory_reserved()
                torch.cuda.set_per_process_memory_fraction(reserved / total)
                kept = []
                try:                                        # (what other tests left free in blocks of theirs)
                    while True:
                        kept.append(torch.empty(32 << 20, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    pass
                torch.cuda.set_per_process_memory_fraction((reserved + (96 << 20)) / total)
                failed = torch.cuda.memory_stats()["num_ooms"]
            else:
                torch.use_deterministic_algorithms(True)
            y.backward(dy)
        finally:
            torch.use_deterministic_algorithms(False)
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert not short or torch.cuda.memory_stats()["num_ooms"] > failed
        got = (x.grad, w.main_grad if flat else w.grad)
        want = want or got
        for a, b in zip(got, want):
            assert torch.equal(a, b) or (flat and (a - b).abs().max() <= 1e-4 * b.abs().max())   # (fp32: last wave in parts)
