"""The GEMM over shapes whose tile counts pick the 128-wide tiles, the 256-wide ones and the
K-slices, against fp64 products."""
import pytest
import torch

from ceo_b200.ops import matmul

pytestmark = pytest.mark.gpu


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
