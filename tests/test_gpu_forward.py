"""The native no-gradient forward pass, the beta logits inside the normalisation kernels and the
RMSNorm widths of the rows kernel."""
import pytest
import torch

from ceo_b200.models.model import EflaLM
from ceo_b200.ops import _lib, decode, nn as K
from ceo_b200.utils.config import Config

pytestmark = pytest.mark.gpu


def _model(d, per_token, use_query):
    cfg = Config.parse_from_file("configs/efla_340m.yaml").model
    cfg.num_layers, cfg.vocab_size = 2, 1000
    cfg.hidden_dim, cfg.intermediate_dim = 512, 1376
    cfg.num_heads, cfg.head_dim = 512 // d, d
    cfg.efla.per_token_beta, cfg.efla.use_query = per_token, use_query
    return EflaLM(cfg, "cuda", seed=3).eval()


@pytest.mark.parametrize("d,per_token,use_query", [(64, True, True), (128, False, False)])
@pytest.mark.parametrize("B,T", [(1, 64), (3, 192), (1, 2048)])
def test_native_forward_matches_layers(d, per_token, use_query, B, T, monkeypatch):
    m = _model(d, per_token, use_query)
    g = torch.Generator(device="cuda").manual_seed(T)
    tok = torch.randint(0, 1000, (B, T), device="cuda", generator=g)
    states = [torch.randn(B, 512 // d, d, d, device="cuda", generator=g) for _ in m.blocks]
    resets = (torch.rand(B, T // 64, device="cuda", generator=g) < 0.3) if B == 3 else None
    with torch.no_grad():
        assert decode.forward_hidden(m, tok, states, resets) is not None
        a, sa = m(tok, states=states, resets=resets, return_states=True)
        la = m(tok, tok)
        monkeypatch.setattr(decode, "forward_hidden", lambda *x, **k: None)
        b, sb = m(tok, states=states, resets=resets, return_states=True)
        lb = m(tok, tok)
    # the same kernels on the same operands
    assert torch.equal(a, b) and torch.equal(la, lb)
    assert all(torch.equal(x, y) for x, y in zip(sa, sb))


def _kernels(f):
    """(kernels of this library that ran in f(), what the launch counter added)."""
    from torch.profiler import ProfilerActivity, profile
    f()
    torch.cuda.synchronize()
    n = _lib.launch_count
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        f()
        torch.cuda.synchronize()
    n = _lib.launch_count - n
    return sum(e.device_type == torch.autograd.DeviceType.CUDA and "ceo::" in e.name
               for e in prof.events()), n


@pytest.mark.parametrize("T", [64, 2048])  # the plain recurrence and spans
def test_launches_are_counted(T):
    m = _model(128, True, True)
    tok = torch.zeros(1, T, dtype=torch.int64, device="cuda")
    assert (_lib.lib().ceo_efla_fwd_segments(1, T, 4, 128) > 1) == (T == 2048)
    with torch.no_grad():
        ran, counted = _kernels(lambda: decode.forward_hidden(m, tok))
        assert ran == counted > 0
        st = m.new_states(1)
        for logits in (True, False):
            ran, counted = _kernels(lambda: decode.decode_tokens(m, tok[:, :5], st, logits))
            assert ran == counted > 0


def test_native_forward_hands_back_other_forms():
    m = _model(64, True, True)
    tok = torch.zeros(1, 64, dtype=torch.int64, device="cuda")
    with torch.no_grad():
        assert decode.forward_hidden(m, tok) is not None
        assert decode.forward_hidden(m, tok[:, :63]) is None
        h = m.blocks[0].efla.register_forward_hook(lambda *a: None)
        assert decode.forward_hidden(m, tok) is None
        h.remove()
        m.blocks[0].mlp.forward = lambda x, r: r
        assert decode.forward_hidden(m, tok) is None
        del m.blocks[0].mlp.forward
        with pytest.raises(ValueError):
            m(tok[:, :63])
    m.train()
    loss = m(tok, tok)
    loss.backward()
    assert m.blocks[0].mlp.w_up.grad is not None


def test_loss_without_gradients_leaves_main_grad_alone():
    w = torch.randn(256, 64, device="cuda").bfloat16().requires_grad_(True)
    w.main_grad = torch.zeros(256, 64, device="cuda")
    x = torch.randn(32, 64, device="cuda").bfloat16().requires_grad_(True)
    t = torch.randint(0, 256, (32,), device="cuda")
    with torch.no_grad():
        a = K.linear_cross_entropy(x, w, t)
    assert not w.main_grad.any()
    b = K.linear_cross_entropy(x, w, t)
    assert torch.equal(a, b.detach()) and w.main_grad.any()


@pytest.mark.parametrize("H,d,P,pad,rows", [(1, 64, 3, 7, 1), (5, 64, 3, 59, 70), (3, 128, 2, 13, 333)])
def test_beta_logits_in_prep(H, d, P, pad, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    N = P * H * d + H + pad
    N += -N % 8
    pad = N - P * H * d - H
    proj = torch.randn(rows, N, device="cuda", generator=g).bfloat16()
    L, st = _lib.lib(), _lib.stream()
    new = lambda *s, dt=torch.float32: torch.empty(*s, dtype=dt, device="cuda")
    q, k = proj.data_ptr(), proj.data_ptr() + 2 * (P - 2) * H * d
    outs = []
    beta = torch.sigmoid(proj[:, P * H * d:P * H * d + H].float()).contiguous()
    for fused in (True, False):
        qn, kn = new(rows, H, d, dt=torch.bfloat16), new(rows, H, d, dt=torch.bfloat16)
        rq, rk, al, bo = new(rows, H), new(rows, H), new(rows, H), new(rows, H)
        if fused:
            _lib.check(L.ceo_efla_prep_fwd_logits(
                q, k, proj.data_ptr() + 2 * P * H * d, N, bo.data_ptr(), qn.data_ptr(),
                kn.data_ptr(), rq.data_ptr(), rk.data_ptr(), al.data_ptr(), rows, H, d, N, N, 1, st),
                "prep")
            assert (bo - beta).abs().max() < 1e-6
        else:
            _lib.check(L.ceo_efla_prep_fwd(q, k, beta.data_ptr(), 0, qn.data_ptr(), kn.data_ptr(),
                                           rq.data_ptr(), rk.data_ptr(), al.data_ptr(), rows, H, d,
                                           N, N, 1, st), "prep")
        outs.append((qn, kn, rq, rk, al))
    for a, b in zip(*outs):
        assert torch.allclose(a.float(), b.float(), rtol=1e-5, atol=1e-6)
    qn, kn, rq, rk, al = outs[1]
    dqn, dkn = (torch.randn(rows, H, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    da = torch.randn(rows, H, device="cuda", generator=g)
    dq, dk = new(rows, H, d, dt=torch.bfloat16), new(rows, H, d, dt=torch.bfloat16)
    dq2, dk2, db = torch.empty_like(dq), torch.empty_like(dk), new(rows, H)
    dl = torch.full((rows, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    off = 2 * P * H * d
    _lib.check(L.ceo_efla_prep_bwd_logits(
        dqn.data_ptr(), dkn.data_ptr(), qn.data_ptr(), kn.data_ptr(), rq.data_ptr(), rk.data_ptr(),
        beta.data_ptr(), da.data_ptr(), dq.data_ptr(), dk.data_ptr(), dl.data_ptr() + off, N, pad,
        rows, H, d, H * d, H * d, 1, st), "prep_bwd")
    _lib.check(L.ceo_efla_prep_bwd(
        dqn.data_ptr(), dkn.data_ptr(), qn.data_ptr(), kn.data_ptr(), rq.data_ptr(), rk.data_ptr(),
        beta.data_ptr(), 0, da.data_ptr(), dq2.data_ptr(), dk2.data_ptr(), db.data_ptr(), rows, H, d,
        H * d, H * d, 1, st), "prep_bwd")
    assert torch.equal(dq, dq2) and torch.equal(dk, dk2)
    want = (db * beta * (1 - beta)).bfloat16().float()
    got = dl[:, P * H * d:].float()
    assert (got[:, :H] - want).abs().max() <= 2 ** -8 * want.abs().max() and not got[:, H:].any()
    assert dl[:, :P * H * d].isnan().all()


@pytest.mark.parametrize("d,normalize", [(64, 1), (128, 0)])
def test_beta_and_its_gradient_are_those_of_torch_sigmoid(d, normalize):
    # every finite bf16 logit whose exponential is a normal fp32 number, bit for bit: a last bit
    # of beta decides roundings in all layers behind it
    x = torch.arange(-2 ** 15, 2 ** 15, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = x[x.isfinite() & (x.float().abs() < 87)].cuda()
    H = 8
    x = x[:x.numel() // H * H].view(-1, H)
    rows = x.shape[0]
    g = torch.Generator(device="cuda").manual_seed(d)
    q = torch.randn(rows, H, d, device="cuda", generator=g).bfloat16()
    dqn, dkn = (torch.randn(rows, H, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    da = torch.randn(rows, H, device="cuda", generator=g)
    beta = torch.sigmoid(x.float())
    L, st = _lib.lib(), _lib.stream()
    new = lambda *s, dt=torch.float32: torch.empty(*s, dtype=dt, device="cuda")
    half = lambda: new(rows, H, d, dt=torch.bfloat16)
    qn, kn, rq, rk, al, al2, bo = half(), half(), *(new(rows, H) for _ in range(5))
    _lib.check(L.ceo_efla_prep_fwd_logits(
        q.data_ptr(), q.data_ptr(), x.data_ptr(), H, bo.data_ptr(), qn.data_ptr(), kn.data_ptr(),
        rq.data_ptr(), rk.data_ptr(), al.data_ptr(), rows, H, d, H * d, H * d, normalize, st), "prep")
    assert torch.equal(bo, beta)
    _lib.check(L.ceo_efla_prep_fwd(
        q.data_ptr(), q.data_ptr(), beta.data_ptr(), 0, qn.data_ptr(), kn.data_ptr(), rq.data_ptr(),
        rk.data_ptr(), al2.data_ptr(), rows, H, d, H * d, H * d, normalize, st), "prep")
    assert torch.equal(al, al2)
    dq, dk, db, dl = half(), half(), new(rows, H), torch.empty_like(x)
    _lib.check(L.ceo_efla_prep_bwd_logits(
        dqn.data_ptr(), dkn.data_ptr(), qn.data_ptr(), kn.data_ptr(), rq.data_ptr(), rk.data_ptr(),
        beta.data_ptr(), da.data_ptr(), dq.data_ptr(), dk.data_ptr(), dl.data_ptr(), H, 0, rows, H, d,
        H * d, H * d, normalize, st), "prep_bwd")
    _lib.check(L.ceo_efla_prep_bwd(
        dqn.data_ptr(), dkn.data_ptr(), qn.data_ptr(), kn.data_ptr(), rq.data_ptr(), rk.data_ptr(),
        beta.data_ptr(), 0, da.data_ptr(), dq.data_ptr(), dk.data_ptr(), db.data_ptr(), rows, H, d,
        H * d, H * d, normalize, st), "prep_bwd")
    want = db * beta * (1.0 - beta)
    sure = want.abs() > 1e-30  # (the kernels flush denormals)
    assert torch.equal(dl[sure], want.bfloat16()[sure]) and not dl[~sure].float().abs().gt(2e-30).any()


@pytest.mark.parametrize("D", [512, 1024, 2048, 4096, 768])
@pytest.mark.parametrize("rows", [1, 3, 4, 5, 2500])
def test_rmsnorm_rows(D, rows):
    g = torch.Generator(device="cuda").manual_seed(D + rows)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, r, w, dy, dh = rn(rows, D), rn(rows, D), rn(D), rn(rows, D), rn(rows, D)
    for res in (None, r):
        xs = x.clone().requires_grad_(True)
        ws = w.clone().requires_grad_(True)
        rs = None if res is None else res.clone().requires_grad_(True)
        y, h = K.rmsnorm(xs, ws, 1e-6, rs, skip=res is None)
        torch.autograd.backward([y, h], [dy, dh])
        hd = (x.double() if res is None else (x.float() + r.float()).bfloat16().double()) \
            .requires_grad_(True)
        wd = w.double().requires_grad_(True)
        yd = hd * torch.rsqrt(hd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
        torch.autograd.backward([yd, hd * 1.0], [dy.double(), dh.double()])
        # one bf16 rounding of an fp32 result
        assert ((y.double() - yd).abs() <= yd.abs() * 2 ** -8 + 1e-5).all()
        assert ((xs.grad.double() - hd.grad).abs() <= hd.grad.abs() * 2 ** -8 + 1e-4).all()
        assert ((ws.grad.double() - wd.grad).abs()
                <= wd.grad.abs() * 2 ** -8 + 1e-5 * rows ** 0.5).all()


@pytest.mark.parametrize("D", [512, 768, 1024])
def test_rmsnorm_of_a_sum_that_is_not_stored(D):
    # without an h to store, x + residual is normalised in fp32 at these widths
    g = torch.Generator(device="cuda").manual_seed(D)
    x, r, w = (torch.randn(n, D, device="cuda", generator=g).bfloat16() for n in (300, 300, 1))
    y, rstd = torch.empty_like(x), torch.empty(300, device="cuda")
    _lib.check(_lib.lib().ceo_rmsnorm_fwd(
        x.data_ptr(), r.data_ptr(), w.data_ptr(), y.data_ptr(), None, rstd.data_ptr(), 300, D, 1e-6,
        _lib.stream()), "ceo_rmsnorm_fwd")
    h = x.double() + r.double()
    want = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    # one rounding to bf16 (half an ulp: 2^-8 of the power of two below) of an fp32 result
    half_ulp = torch.ldexp(torch.ones_like(want), torch.frexp(want).exponent - 9)
    assert ((y.double() - want).abs() <= half_ulp + want.abs() * 2 ** -20).all()
