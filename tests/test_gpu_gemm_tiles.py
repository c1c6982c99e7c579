"""The GEMM's tile kinds (128 x 256, 256 x 256 on a CTA pair, 128 x 128) and K-slices against fp64
products.  Which kind a shape gets is asked of the library, for the chip the test runs on."""
import pytest
import torch

from ceo_b200.ops import _lib, fp8, matmul

pytestmark = pytest.mark.gpu
WIDE, PAIR, NARROW = 0, 1, 2
STORE, MORE, SWIGLU_BWD, ACCUMULATE, GENERAL = range(5)  # epilogues


def _kind(M, N, K, epi, batch=1, fp8=0):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r = _lib.lib().ceo_gemm_pick(M, N, K, batch, fp8, epi, sms)
    return r & 3, r >> 2


# last tiles that are ragged in M, N and K, a last CTA of a pair with no row at all (M = 264, 520,
# 2312), whole 64-column panels (320, 1216, 192), rows that are no multiple of 16 bytes (N = 11270 ...)
SHAPES = [(WIDE, 264, 264, 520, 20), (WIDE, 264, 11272, 520, 1), (WIDE, 2312, 1032, 520, 3),
          (WIDE, 320, 11264, 512, 1), (WIDE, 264, 11270, 520, 1), (PAIR, 200, 11264, 1032, 1),
          (PAIR, 1160, 2056, 1032, 1), (PAIR, 2312, 1032, 1032, 1), (PAIR, 264, 2056, 1032, 3),
          (PAIR, 520, 4104, 1032, 1), (PAIR, 200, 520, 1032, 20), (PAIR, 1216, 2112, 1032, 1),
          (PAIR, 520, 4102, 4104, 1), (NARROW, 264, 520, 520, 1), (NARROW, 1000, 264, 520, 1),
          (NARROW, 200, 264, 520, 3), (NARROW, 192, 320, 520, 1), (NARROW, 264, 518, 520, 1)]


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("kind,M,N,K,batch", SHAPES)
def test_every_tile_kind(kind, M, N, K, batch, a_mn, b_mn):
    for epi in (GENERAL,) if N % 8 else (STORE, MORE, ACCUMULATE):
        assert _kind(M, N, K, epi, batch) == (kind, 1)
    if b_mn and N % 8:
        pytest.skip("a TMA row stride is a multiple of 16 bytes")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    new = lambda *s: torch.randn(*((batch, *s) if batch > 1 else s), device="cuda", generator=g)
    a = new(*((K, M) if a_mn else (M, K))).bfloat16()
    b = new(*((N, K) if b_mn else (K, N))[::-1]).bfloat16()
    tr = lambda t: t.transpose(-1, -2)
    want = (tr(a) if a_mn else a).double() @ (b if b_mn else tr(b)).double()
    near = lambda got, w: (got.double() - w).abs() <= w.abs() * 2 ** -8 + 2 ** -15 * K ** 0.5
    assert near(matmul.gemm(a, b, a_mn=a_mn, b_mn=b_mn), want).all()
    res = new(M, N).bfloat16()
    got = matmul.gemm(a, b, a_mn=a_mn, b_mn=b_mn, residual=res, alpha=0.5)
    assert near(got, 0.5 * want + res.double()).all()
    # fp32 sums of K unit-normal products in any order
    acc = new(M, N)
    w = want + acc.double()
    matmul.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=acc, accumulate=True)
    assert (acc.double() - w).abs().max() <= 2 ** -16 * K ** 0.5 * 4


@pytest.mark.parametrize("kind,M,N,K", [(WIDE, 520, 2056, 4104), (WIDE, 1032, 1032, 8200),
                                        (PAIR, 2056, 264, 4104), (PAIR, 520, 520, 16392),
                                        (NARROW, 264, 1032, 4104), (NARROW, 2056, 36, 4104)])
def test_k_slices_of_every_tile_kind(kind, M, N, K):
    got, slices = _kind(M, N, K, ACCUMULATE)
    assert got == kind and slices > 1
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randn(K, n, device="cuda", generator=g).bfloat16() for n in (M, N + N % 8))
    b = b[:, :N]
    acc = torch.randn(M, N, device="cuda", generator=g)
    w = a.double().t() @ b.double() + acc.double()
    matmul.gemm(a, b, a_mn=True, b_mn=True, out=acc, accumulate=True)
    # the tensor core drops what lies below its accumulator, at most 2^-22 of a sum of at most 6
    # standard deviations, at each of its K / 16 steps; a slice's sums are shorter by its share
    assert (acc.double() - w).abs().max() <= K / 16 * 2 ** -22 * 6 * (K / slices) ** 0.5


@pytest.mark.parametrize("kind,M,N,K", [
    (WIDE, 264, 11272, 528), (WIDE, 320, 11264, 528), (PAIR, 1160, 2064, 2064),
    (PAIR, 2312, 1040, 2064), (PAIR, 4360, 2064, 4112), (NARROW, 200, 528, 528)])
def test_every_tile_kind_on_8_bit_operands(kind, M, N, K):
    assert _kind(M, N, K, STORE, fp8=1)[0] == _kind(M, N, K, ACCUMULATE, fp8=1)[0] == kind
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randn(n, K, device="cuda", generator=g).to(torch.float8_e4m3fn) for n in (M, N))
    want = a.float().double() @ b.float().double().t()
    got = fp8.gemm_fp8(a.view(torch.uint8), b.view(torch.uint8))
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + 2 ** -15 * K ** 0.5).all()
    acc = torch.ones(M, N, device="cuda")
    fp8.gemm_fp8(a.view(torch.uint8), b.view(torch.uint8), out=acc, accumulate=True)
    assert (acc.double() - want - 1).abs().max() <= 2 ** -16 * K ** 0.5 * 4


# both SwiGLU epilogues: (kind of the gate / up product, kind of the data gradient)
@pytest.mark.parametrize("up,down,M,F,D", [
    (PAIR, PAIR, 2312, 1376, 1032), (PAIR, PAIR, 1160, 2816, 1032), (PAIR, WIDE, 4360, 2816, 1032),
    (PAIR, NARROW, 1160, 1376, 1032), (WIDE, WIDE, 8456, 1376, 72), (WIDE, WIDE, 264, 11296, 136),
    (NARROW, NARROW, 576, 1376, 136)])
def test_swiglu_epilogues_of_every_tile_kind(up, down, M, F, D):
    assert _kind(M, 2 * F, D, MORE) == (up, 1) and _kind(M, F, D, SWIGLU_BWD) == (down, 1)
    _swiglu_case(M, F, D)


def _swiglu_case(M, F, D):
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, D, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * F, D, device="cuda", generator=g) * D ** -0.5).bfloat16()
    gu = torch.empty(M, 2 * F, dtype=torch.bfloat16, device="cuda")
    act = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
    matmul._gemm_swiglu(x, w, gu, M, 2 * F, D, False, 1, act)
    z = x.double() @ w.double().t()
    ref = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
    # one bf16 rounding (2^-8 relative) of fp32 results; the exponential's own error stays below
    assert ((gu.double() - z).abs() <= z.abs() * 2 ** -8 + 1e-5).all()
    assert ((act.double() - ref).abs() <= ref.abs() * 2 ** -8 + 1e-4).all()
    dy = torch.randn(M, D, device="cuda", generator=g).bfloat16()
    wd = (torch.randn(D, F, device="cuda", generator=g) * D ** -0.5).bfloat16()
    dgu = torch.empty_like(gu)
    matmul._gemm_swiglu(dy, wd, dgu, M, F, D, True, 2, gu)
    zz = gu.double().requires_grad_(True)
    (torch.nn.functional.silu(zz[:, 0::2]) * zz[:, 1::2]).backward(dy.double() @ wd.double())
    assert ((dgu.double() - zz.grad).abs() <= zz.grad.abs() * 2 ** -7 + 1e-3).all()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(576, 2048, 520), (136, 136, 64), (1024, 1024, 4096),
                                   (5632, 1024, 640), (264, 4104, 1000), (2048, 40, 2048)])
def test_tile_widths(M, N, K, a_mn, b_mn):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", generator=g).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", generator=g).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    got = matmul.gemm(a, b, a_mn=a_mn, b_mn=b_mn, residual=res)
    w = want + res.double()
    assert ((got.double() - w).abs() <= w.abs() * 2 ** -8 + 2 ** -15 * K ** 0.5).all()
    acc = torch.randn(M, N, device="cuda", generator=g)
    w = want + acc.double()
    matmul.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=acc, accumulate=True)
    # fp32 sums of K unit-normal products in any order
    assert (acc.double() - w).abs().max() <= 2 ** -16 * K ** 0.5 * 4


@pytest.mark.parametrize("M,F,D", [(576, 1376, 512), (200, 96, 136)])
def test_swiglu_epilogues_on_narrow_tiles(M, F, D):
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, D, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * F, D, device="cuda", generator=g) * D ** -0.5).bfloat16()
    gu = torch.empty(M, 2 * F, dtype=torch.bfloat16, device="cuda")
    act = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
    matmul._gemm_swiglu(x, w, gu, M, 2 * F, D, False, 1, act)
    z = x.double() @ w.double().t()
    ref = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
    assert ((gu.double() - z).abs() <= z.abs() * 2 ** -8 + 1e-5).all()
    assert ((act.double() - ref).abs() <= ref.abs() * 2 ** -8 + 1e-4).all()
    dy = torch.randn(M, D, device="cuda", generator=g).bfloat16()
    wd = (torch.randn(D, F, device="cuda", generator=g) * D ** -0.5).bfloat16()
    dgu = torch.empty_like(gu)
    matmul._gemm_swiglu(dy, wd, dgu, M, F, D, True, 2, gu)
    zz = gu.double().requires_grad_(True)
    (torch.nn.functional.silu(zz[:, 0::2]) * zz[:, 1::2]).backward(dy.double() @ wd.double())
    assert ((dgu.double() - zz.grad).abs() <= zz.grad.abs() * 2 ** -7 + 1e-3).all()
