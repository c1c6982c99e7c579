"""The weight-streaming GEMM for up to 128 rows and the native token loop built on it, against
fp32 PyTorch products and the layer-by-layer path."""
import pytest
import torch

from ceo_b200.models.model import EflaLM
from ceo_b200.ops import decode, matmul
from ceo_b200.utils.config import Config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128, 129])
@pytest.mark.parametrize("N,K", [(4, 8), (100, 72), (128, 64), (2048, 2048), (6208, 1024),
                                 (1024, 2816), (130, 200)])
def test_few_rows_gemm(M, N, K):
    # edges: row counts around each MMA width, a partial weight tile, a K tail, every cluster cut
    g = torch.Generator(device="cuda").manual_seed(M * 7919 + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    want = a.double() @ w.double().t()
    # fp32 sums of K products of unit normals: error far below K^0.5 * 2^-20
    got = matmul.gemm(a, w, out_dtype=torch.float32, alpha=0.5)
    assert (got.double() - 0.5 * want).abs().max() <= 2 ** -18 * K ** 0.5 * 8
    got = matmul.gemm(a, w, residual=res)
    want = want + res.double()
    # one rounding to bf16 (half an ulp, 2^-8 relative) plus the fp32 error
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + 2 ** -15 * K ** 0.5).all()


@pytest.mark.parametrize("M", [1, 40, 128])
@pytest.mark.parametrize("F,K", [(32, 64), (96, 200), (2816, 1024)])
def test_few_rows_swiglu(M, F, K):
    g = torch.Generator(device="cuda").manual_seed(M + F + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * F, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    act = torch.empty(M, F, dtype=torch.bfloat16, device="cuda")
    gu = torch.empty(M, 2 * F, dtype=torch.bfloat16, device="cuda")
    matmul._gemm_swiglu(x, w, gu, M, 2 * F, K, False, 1, act)
    want = x.double() @ w.double().t()
    assert ((gu.double() - want).abs() <= want.abs() * 2 ** -8 + 1e-5).all()
    ref = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    assert ((act.double() - ref).abs() <= ref.abs() * 2 ** -8 + 1e-4).all()


def _model(d, per_token, use_query, normalize, layers=3):
    cfg = Config.parse_from_file("configs/efla_340m.yaml").model
    cfg.num_layers, cfg.vocab_size = layers, 1000
    cfg.hidden_dim, cfg.intermediate_dim = 512, 1376
    cfg.num_heads, cfg.head_dim = 512 // d, d
    cfg.efla.per_token_beta, cfg.efla.use_query = per_token, use_query
    cfg.efla.normalize_qk = normalize
    m = EflaLM(cfg, "cuda", seed=3).eval()
    with torch.no_grad():
        m.embed_tokens.normal_(0.0, 1.0, generator=torch.Generator(device="cuda").manual_seed(1))
    return m


@pytest.mark.parametrize("d,per_token,use_query,normalize", [
    (64, True, True, True), (128, True, True, True), (128, False, False, True),
    (64, False, True, False)])
def test_native_decode_matches_layers(d, per_token, use_query, normalize, monkeypatch):
    m = _model(d, per_token, use_query, normalize)
    tok = torch.randint(0, 1000, (5, 21), device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(9))
    calls = []
    real = decode.decode_tokens
    monkeypatch.setattr(decode, "decode_tokens", lambda *a, **k: (calls.append(0), real(*a, **k))[1])
    for B in (1, 5):
        st = m.new_states(B)
        calls.clear()
        native = [m.decode_step(tok[:B, t], st) for t in range(21)]
        assert len(calls) == 21 and real(m, tok[:B, :1], m.new_states(B)) is not None
        with monkeypatch.context() as mp:
            mp.setattr(decode, "decode_tokens", lambda *a, **k: None)
            st2 = m.new_states(B)
            layers = [m.decode_step(tok[:B, t], st2) for t in range(21)]
        # bf16 activations: roundings that fall the other way after a different summation order
        for a, b in zip(native, layers):
            assert (a - b).norm() / b.norm() < 2e-2
        for a, b in zip(st, st2):
            assert (a - b).norm() / b.norm() < 2e-2
    # a prompt in one pass (16 tokens are staged at a time: 21 leaves a remainder)
    sp = m.new_states(1)
    lp = m.prefill_tokens(tok[0].tolist(), sp)
    st = m.new_states(1)
    for t in range(21):
        ls = m.decode_step(tok[:1, t], st)
    assert (lp - ls).norm() / ls.norm() < 2e-2
    for a, b in zip(sp, st):
        assert (a - b).norm() / b.norm() < 2e-2


def test_decode_beta_is_torch_sigmoid():
    # one head whose key and value are the first unit vector and ones, so that row 0 of the state
    # after one token is alpha itself, bit for bit; 128 tokens spell 128 logits in binary
    cfg = Config.parse_from_file("configs/efla_340m.yaml").model
    cfg.num_layers, cfg.vocab_size, cfg.hidden_dim, cfg.intermediate_dim = 1, 128, 64, 32
    cfg.num_heads, cfg.head_dim = 1, 64
    cfg.efla.per_token_beta = cfg.efla.use_query = cfg.efla.normalize_qk = True
    m = EflaLM(cfg, "cuda").eval()
    bits = torch.tensor([[1.0 if t >> i & 1 else -1.0 for i in range(7)] for t in range(128)],
                        device="cuda")
    step = torch.tensor([4.0 / 2 ** i for i in range(7)], device="cuda")
    with torch.no_grad():
        m.embed_tokens.fill_(1.0)
        m.embed_tokens[:, 1:8] = bits.bfloat16()
        w = m.blocks[0].efla.w_qkv
        w.zero_()
        w[64, 0] = 1.0        # k = e_0
        w[128:192, 0] = 1.0   # v = 1
        w[192, 1:8] = step.bfloat16()
    st = m.new_states(128)
    assert decode.decode_tokens(m, torch.arange(128, device="cuda")[:, None], st) is not None
    alpha = -torch.expm1(-torch.sigmoid(bits @ step))
    assert torch.equal(st[0][:, 0, 0], alpha[:, None].expand(128, 64))


def test_native_decode_hands_back_other_forms():
    m = _model(64, True, True, True)
    tok = torch.zeros(1, 1, dtype=torch.int64, device="cuda")
    st = m.new_states(1)
    assert decode.decode_tokens(m, tok, [s.double() for s in st]) is None
    assert decode.decode_tokens(m, tok, [s.transpose(2, 3) for s in st]) is None
    assert decode.decode_tokens(m, torch.zeros(129, 1, dtype=torch.int64, device="cuda"),
                                m.new_states(129)) is None
    h = m.blocks[1].mlp.register_forward_hook(lambda *a: None)
    assert decode.decode_tokens(m, tok, st) is None
    h.remove()
    # a prompt longer than one pass
    ids = [i % 1000 for i in range(150)]
    a, b = m.new_states(1), m.new_states(1)
    la = m.prefill_tokens(ids, a)
    for i in ids:
        lb = m.decode_step(torch.tensor([i], device="cuda"), b)
    assert (la - lb).norm() / lb.norm() < 2e-2


class _Wrapped(torch.nn.Module):
    """A block behind another module, as a checkpointing or logging wrapper puts it."""

    def __init__(self, blk):
        super().__init__()
        self.inner = blk

    def forward(self, *a, **k):
        return self.inner(*a, **k)

    @property
    def prism(self):
        return self.inner.prism

    @property
    def dropout(self):
        return self.inner.dropout

    def decode_step(self, *a, **k):
        return self.inner.decode_step(*a, **k)


@pytest.mark.parametrize("how", ["wrapped block", "weight as attribute", "decode_step replaced"])
def test_models_with_replaced_parts_run_layer_by_layer(how):
    m, plain = _model(64, True, True, True), _model(64, True, True, True)
    if how == "wrapped block":
        m.blocks[1] = _Wrapped(m.blocks[1])
    elif how == "weight as attribute":
        w = m.blocks[1].efla.w_qkv.detach().clone()
        del m.blocks[1].efla.w_qkv
        m.blocks[1].efla.w_qkv = w
    else:
        calls = []
        real = m.blocks[1].efla.decode_step
        m.blocks[1].efla.decode_step = lambda *a: (calls.append(0), real(*a))[1]
    tok = torch.randint(0, 1000, (2, 64), device="cuda",
                        generator=torch.Generator(device="cuda").manual_seed(4))
    with torch.no_grad():
        a, b = m(tok), plain(tok)
    assert (a - b).norm() < 2e-2 * b.norm()
    sa, sb = m.new_states(2), plain.new_states(2)
    a, b = m.decode_step(tok[:, 0], sa), plain.decode_step(tok[:, 0], sb)
    assert (a - b).norm() < 2e-2 * b.norm()
    if how == "decode_step replaced":
        assert len(calls) == 1
