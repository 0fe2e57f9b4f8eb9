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
    """Products that get tiles of several widths (of each form: test_every_form), ragged in every direction, with and without an fp32 addend. The
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
    """Gate and up columns of a tile come from two places of the weight: ragged widths (at every form: test_every_form). The result equals
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
    """The last part of a sum kept in fp32 (at every form: test_every_form): one rounding to bf16 (2^-8 of the value at most)
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
    """Products that get pairs of CTAs at both widths (1000 x 4104 x 1000 with an addend only): an odd number of 128-row tiles, rows that end in either CTA's half, ragged columns
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


# (CTAs a tile, columns) -> M, N, K that get it with and without an addend and with SwiGLU on 148 SMs; M ends in either half of a pair's rows
FORMS = {(1, 64): (104, 208, 200), (1, 128): (104, 11024, 520), (1, 256): (264, 11024, 2056), (2, 128): (648, 1552, 2056), (2, 256): (520, 16400, 520)}


def _operands(M, N, Kd):
    from ringattention_b200.ops import kernels as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = torch.randn(M, Kd, device="cuda", generator=g).bfloat16(), torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    want = a.double() @ b.double().t()
    return K, g, a, b, want, 2e-6 * (a.double().abs() @ b.double().abs().t())


def _form_is(form, M, N, Kd, **kw):
    from ringattention_b200.ops import kernels as K

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shapes are chosen for 148 SMs")
    assert K.gemm_form(M, N, Kd, **kw) == form


@pytest.mark.parametrize("form", FORMS)
def test_every_form(form):
    """Each form of the kernel by its name, with each kind of result: bf16, bf16 with an addend in bf16 or fp32, accumulated in fp32, SwiGLU. Tolerances as
    above; SwiGLU as the two-pass path."""
    M, N, Kd = FORMS[form]
    K, g, a, b, want, slack = _operands(M, N, Kd)
    _form_is(form, M, N, Kd)
    c = K.gemm(a, b)
    assert ((c.double() - want).abs() <= slack + 2**-8 * want.abs()).all()
    _form_is(form, M, N, Kd, addend=True)
    r = torch.randn(M, N + 8, device="cuda", generator=g)[:, :N]
    for rr in (r, r.bfloat16()):
        c = K.gemm(a, b, out=torch.empty(M, N, device="cuda", dtype=torch.bfloat16), residual=rr)
        assert ((c.double() - want - rr.double()).abs() <= slack + 2e-6 * rr.double().abs() + 2**-8 * (want + rr.double()).abs()).all()
    acc = r.clone()
    K.gemm(a, b, out=acc, residual=acc)
    assert ((acc.double() - want - r.double()).abs() <= slack + 2e-6 * r.double().abs()).all()
    _form_is(form, M, N, Kd, swiglu=True)
    w = (b * Kd ** -0.5).bfloat16()
    gu = K.linear_fwd(a, w).float()
    h = torch.nn.functional.silu(gu[:, :N // 2]) * gu[:, N // 2:]
    assert ((K.linear_swiglu(a, w).float() - h).abs() <= 2**-7 * h.abs() + 1e-4).all()


@pytest.mark.parametrize("form", FORMS)
def test_layer_epilogues_at_every_form(form):
    """Bias with a factor, the squared relu into a strided view, and an fp32 tail that begins at a tile's start and inside either half of one."""
    from ringattention_b200.ops import _lib

    M, N, Kd = FORMS[form]
    K, g, a, b, want, slack = _operands(M, N, Kd)
    _form_is(form, M, N, Kd)
    bias = torch.randn((N + 31) // 32 * 32, device="cuda", generator=g)
    c = K.linear_ex(a, b, torch.empty(M, N, device="cuda"), bias=bias, alpha=0.37)
    assert ((c.double() - 0.37 * want - bias[:N].double()).abs() <= slack + 1e-6 * (want.abs() + 10)).all()
    wide = torch.full((M, N + 16), 3.0, device="cuda", dtype=torch.bfloat16)
    K.linear_ex(a, b, wide[:, 8:8 + N], relu2=True)
    sq = want.clamp_min(0).square()
    assert ((wide[:, 8:8 + N].double() - sq).abs() <= 2 * want.abs() * slack + slack ** 2 + 2**-8 * sq).all()
    assert (wide[:, :8] == 3).all() and (wide[:, 8 + N:] == 3).all()
    at = N // (2 * form[1]) * form[1]  # where a tile begins
    for cut in {at, at + 32, at + form[1] // 2 + form[1] // 4 // 32 * 32} - {0}:
        main, tail = torch.empty(M, cut, device="cuda", dtype=torch.bfloat16), torch.empty(M, N - cut, device="cuda")
        K.linear_ex(a, b, main, tail=tail, n_split=cut)
        assert ((main.double() - want[:, :cut]).abs() <= slack[:, :cut] + 2**-8 * want[:, :cut].abs()).all()
        assert ((tail.double() - want[:, cut:]).abs() <= slack[:, cut:]).all()
    _lib.check_status()


@pytest.mark.parametrize("M", [16, 128])
@pytest.mark.parametrize("addend", [False, True])
def test_a_pair_whose_second_cta_has_no_row(M, addend):
    N, Kd = 1032, 4104
    K, g, a, b, want, slack = _operands(M, N, Kd)
    _form_is((2, 128), M, N, Kd, addend=addend)
    r = torch.randn(M, N, device="cuda", generator=g).bfloat16() if addend else torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    room = torch.full((M + 256, N), 3.0, device="cuda", dtype=torch.bfloat16)
    K.gemm(a, b, out=room[:M], residual=r if addend else None)
    want = want + r.double()
    assert ((room[:M].double() - want).abs() <= slack + 2e-6 * r.double().abs() + 2**-8 * want.abs()).all() and (room[M:] == 3.0).all()
