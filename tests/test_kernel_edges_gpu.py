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
    acc = torch.full((M + 1, N + 4), 3.0, device="cuda")
    gemm(x, w, out=acc[:M, :N], accumulate=True, alpha=0.5)
    _near(acc[:M, :N], 0.5 * z + 3.0, dtype, 0)
    assert (acc[M:] == 3.0).all() and (acc[:, N:] == 3.0).all()
    f32 = gemm(x, w, out_dtype=torch.float32)
    _near(f32, z, dtype, 0)
    torch.cuda.synchronize()
    assert _lib.read_error() == 0
