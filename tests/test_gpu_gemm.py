"""tcgen05 GEMM against an fp32 PyTorch product, every operand-major combination."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b):
    return a.float() @ b.float().t()


@pytest.mark.parametrize("a_mn", [False, True])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("shape", [(128, 256, 64), (200, 328, 136), (1024, 768, 512)])
def test_gemm_majors(a_mn, b_mn, shape):
    from ringattention_b200.ops import _lib, kernels as K

    M, N, Kd = shape
    torch.manual_seed(0)
    a = torch.randn(M, Kd, device="cuda").bfloat16()
    b = torch.randn(N, Kd, device="cuda").bfloat16()
    A = a.t().contiguous() if a_mn else a
    B = b.t().contiguous() if b_mn else b
    c = K.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = _ref(a, b)
    assert (c.float() - ref).abs().max() <= 0.01 * ref.abs().max() + 1e-3


def test_gemm_residual_and_fp32_accumulate():
    from ringattention_b200.ops import kernels as K

    torch.manual_seed(1)
    a = torch.randn(256, 320, device="cuda").bfloat16()
    b = torch.randn(512, 320, device="cuda").bfloat16()
    r = torch.randn(256, 512, device="cuda").bfloat16()
    c = K.gemm(a, b, residual=r)
    ref = _ref(a, b) + r.float()
    assert (c.float() - ref).abs().max() <= 0.01 * ref.abs().max()
    acc = torch.randn(256, 512, device="cuda")
    acc0 = acc.clone()
    K.gemm(a, b, out=acc, residual=acc)
    assert torch.allclose(acc, acc0 + _ref(a, b), atol=2e-3, rtol=1e-4)


def test_linear_fwd_dgrad_wgrad_match_autograd():
    from ringattention_b200.ops import kernels as K

    torch.manual_seed(2)
    x = torch.randn(384, 256, device="cuda").bfloat16()
    w = torch.randn(512, 256, device="cuda").bfloat16()
    dy = torch.randn(384, 512, device="cuda").bfloat16()
    xf, wf = x.float().requires_grad_(True), w.float().requires_grad_(True)
    (xf @ wf.t()).backward(dy.float())
    y = K.linear_fwd(x, w)
    dx = K.linear_dgrad(dy, w)
    dw = torch.zeros(512, 256, device="cuda")
    K.linear_wgrad(dy, x, dw)
    assert (y.float() - (xf @ wf.t())).abs().max() <= 0.01 * (xf @ wf.t()).abs().max()
    assert (dx.float() - xf.grad).abs().max() <= 0.01 * xf.grad.abs().max()
    assert torch.allclose(dw, wf.grad, atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,Kd", [(1, 8, 8), (128, 64, 640), (100, 72, 200), (257, 200, 1000), (2048, 1024, 328), (1100, 3000, 72), (4000, 1544, 136)])
def test_gemm_at_every_tile_width(M, N, Kd, a_mn, b_mn):
    """Products that get tiles of 64, 128 and 256 columns, ragged in every direction, with and without an fp32 addend. The
    products of bf16 numbers are exact in fp32: tolerance 2e-6 of the sum of their magnitudes, plus bf16 rounding (2^-8)."""
    from ringattention_b200.ops import _lib, kernels as K

    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("a leading dimension that is no multiple of eight is refused")
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    A, B = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    want = a.double() @ b.double().t()
    slack = 2e-6 * (a.double().abs() @ b.double().abs().t())
    wide = torch.full((M, N + 24), 3.0, device="cuda")
    acc = wide[:, :N]
    K.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=acc, residual=acc)
    assert ((acc.double() - 3.0 - want).abs() <= slack + 1e-6).all() and (wide[:, N:] == 3.0).all()
    c = K.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
    assert ((c.double() - want).abs() <= slack + 2**-8 * want.abs()).all()
    _lib.check_status()


@pytest.mark.parametrize("M,F,Kd", [(5, 8, 64), (128, 72, 200), (300, 1000, 1024), (2048, 2816, 512), (2100, 5504, 136)])
def test_swiglu_epilogue_at_every_tile_width(M, F, Kd):
    """Gate and up columns of a tile come from two places of the weight: ragged widths at each tile width. The result equals
    the two-pass path, up to the last bit of a bf16 (2^-8) where a sum lies on a rounding border."""
    from ringattention_b200.ops import kernels as K

    g = torch.Generator(device="cuda").manual_seed(F)
    x = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * F, Kd, device="cuda", generator=g) / Kd ** 0.5).bfloat16()
    got = K.linear_swiglu(x, w)
    gu = K.linear_fwd(x, w).float()
    want = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    assert ((got.float() - want).abs() <= 2**-7 * want.abs() + 1e-4).all()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True)])
@pytest.mark.parametrize("M,N,Kd", [(8, 8, 8), (104, 72, 200), (2048, 1024, 328), (4000, 1544, 136)])
def test_gemm_fp32_addend_bf16_result(M, N, Kd, a_mn, b_mn):
    """The last part of a sum kept in fp32, at tiles of 64, 128 and 256 columns: one rounding to bf16 (2^-8 of the value at most)
    beside 2e-6 of the sum of the magnitudes."""
    from ringattention_b200.ops import kernels as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = torch.randn(M, Kd, device="cuda", generator=g).bfloat16(), torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    r = torch.randn(M, N + 12, device="cuda", generator=g)[:, :N]
    A, B = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    got = K.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=torch.empty(M, N, device="cuda", dtype=torch.bfloat16), residual=r)
    want = a.double() @ b.double().t() + r.double()
    slack = 2e-6 * (a.double().abs() @ b.double().abs().t() + r.double().abs())
    assert ((got.double() - want).abs() <= slack + 2**-8 * want.abs()).all()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,Kd", [(512, 4104, 2056), (520, 2056, 2056), (1030, 4104, 2056), (1000, 4104, 1000), (1030, 6000, 2056), (3900, 4104, 1000)])
def test_gemm_on_cta_pairs(M, N, Kd, a_mn, b_mn):
    """Products that get pairs of CTAs at both widths: an odd number of 128-row tiles, rows that end in either CTA's half, ragged columns
    and K, a strided result, and results in bf16, bf16 with an addend and accumulated in fp32. Tolerances as above."""
    from ringattention_b200.ops import _lib, kernels as K

    M = (M + 7) // 8 * 8 if a_mn else M
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    A, B = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    want = a.double() @ b.double().t()
    slack = 2e-6 * (a.double().abs() @ b.double().abs().t())
    wide = torch.full((M + 1, N + 24), 3.0, device="cuda")
    acc = wide[:M, :N]
    K.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=acc, residual=acc)
    assert ((acc.double() - 3.0 - want).abs() <= slack + 1e-6).all() and (wide[:, N:] == 3.0).all() and (wide[M:] == 3.0).all()
    c = K.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
    assert ((c.double() - want).abs() <= slack + 2**-8 * want.abs()).all()
    r = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    c = K.gemm(A, B, a_mn=a_mn, b_mn=b_mn, residual=r)
    assert ((c.double() - want - r.double()).abs() <= slack + 2e-6 * r.double().abs() + 2**-8 * (want + r.double()).abs()).all()
    _lib.check_status()


@pytest.mark.parametrize("M,F,Kd", [(520, 2816, 1000), (1030, 5000, 1000), (2048, 2816, 512)])
def test_swiglu_epilogue_on_cta_pairs(M, F, Kd):
    """One CTA of a pair holds the gate's columns, the other the matching ones of up. Tolerance as above."""
    test_swiglu_epilogue_at_every_tile_width(M, F, Kd)
