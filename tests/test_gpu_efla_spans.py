"""The forward state recurrence in spans (few chains, many chunks) against the fp64 recurrence and
against the plain kernels."""
import pytest
import torch

from ceo_b200.ops import _lib, efla

pytestmark = pytest.mark.gpu


def _run(q, k, v, a, s0, resets, segs):
    B, T, H, d = k.shape
    n = T // 64
    new = lambda *s, dt=torch.bfloat16: torch.empty(*s, dtype=dt, device="cuda")
    w, up, o = new(B, T, H, d), new(B, T, H, d), new(B, T, H, d)
    states, xinv = new(B, H, n, d, d), new(B, H, n, 64, 64)
    sf = new(B, H, d, d, dt=torch.float32)
    ws = torch.full((3 * B * H * segs * d * d,), float("nan"), device="cuda")
    _lib.check(_lib.lib().ceo_efla_fwd_seg(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), a.data_ptr(), _lib.ptr(s0), w.data_ptr(),
        up.data_ptr(), states.data_ptr(), xinv.data_ptr(), o.data_ptr(), sf.data_ptr(),
        _lib.ptr(resets), segs, ws.data_ptr(), B, T, H, d, H * d, H * d, H * d,
        _lib.status_word(q.device).data_ptr(), _lib.stream()), "ceo_efla_fwd_seg")
    return o, sf, states


def _exact(q, k, v, a, s0, resets):
    B, T, H, d = k.shape
    q, k, v, a = (t.double() for t in (q, k, v, a))
    S = torch.zeros(B, H, d, d, dtype=torch.float64, device="cuda") if s0 is None else s0.double()
    out = []
    for t in range(T):
        if resets is not None and t % 64 == 0:
            S = S * (1 - resets[:, t // 64].double())[:, None, None, None]
        u = v[:, t] - torch.einsum("bhkv,bhk->bhv", S, k[:, t])
        S = S + a[:, t][..., None, None] * k[:, t][..., :, None] * u[..., None, :]
        out.append(torch.einsum("bhkv,bhk->bhv", S, q[:, t]))
    return torch.stack(out, 1), S


# n chunks that do not divide by the spans, spans of one chunk, slowly forgotten states (small
# alpha: the transfer matrices matter), a carried state, document starts in and between spans
@pytest.mark.parametrize("d,n,segs,scale,with_s0,with_resets", [
    (64, 11, 3, 0.9, False, False), (64, 4, 4, 0.02, True, False), (128, 13, 5, 0.02, True, False),
    (128, 7, 3, 0.5, False, True), (64, 10, 4, 0.05, True, True)])
def test_spans_match_the_recurrence(d, n, segs, scale, with_s0, with_resets):
    g = torch.Generator(device="cuda").manual_seed(d + n + segs)
    B, H, T = 2, 3, 64 * n
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = (efla.l2norm(rn(B, T, H, d).bfloat16()) for _ in range(2))
    v = rn(B, T, H, d).bfloat16()
    a = torch.rand(B, T, H, device="cuda", generator=g) * scale
    s0 = rn(B, H, d, d) if with_s0 else None
    resets = None
    if with_resets:
        resets = (torch.rand(B, n, device="cuda", generator=g) < 0.3).to(torch.uint8)
    o1, s1, st1 = _run(q, k, v, a, s0, resets, 1)
    o2, s2, st2 = _run(q, k, v, a, s0, resets, segs)
    want_o, want_s = _exact(q, k, v, a, s0, resets)
    err = lambda x, y: float((x.double() - y).norm() / y.norm())
    # bf16 operands bound both; the spans' fold is fp32, so it may not add to the plain error by
    # more than the scatter of a different rounding (10 %)
    assert err(o2, want_o) <= 1.1 * err(o1, want_o) + 1e-4 and err(o2, want_o) < 1e-2
    assert err(s2, want_s) <= 1.1 * err(s1, want_s) + 1e-4 and err(s2, want_s) < 1e-2
    assert err(st2, st1.double()) < 1e-2


# an overflow in one document: chunk 1 (span 0) holds an infinite or NaN value, or the carried
# state does; documents start at the given chunks (inside spans, at a span's first and last chunk,
# in the same span as the overflow)
@pytest.mark.parametrize("starts", [(5,), (3,), (2, 9), (8,), (2, 4, 5)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("d,where", [(64, "v"), (128, "s0")])
def test_documents_stay_apart_when_one_overflows(starts, bad, d, where):
    g = torch.Generator(device="cuda").manual_seed(sum(starts))
    B, H, n, segs = 2, 2, 12, 4  # spans of three chunks
    T = 64 * n
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k = (efla.l2norm(rn(B, T, H, d).bfloat16()) for _ in range(2))
    v, s0 = rn(B, T, H, d).bfloat16(), rn(B, H, d, d)
    a = torch.rand(B, T, H, device="cuda", generator=g) * 0.1
    resets = torch.zeros(B, n, dtype=torch.uint8, device="cuda")
    resets[0, list(starts)] = 1  # the second sequence has no document start and no overflow
    if where == "v":
        v[0, 70, 1] = bad
    else:
        s0[0, 1] = bad
    o1, s1, st1 = _run(q, k, v, a, s0, resets, 1)
    o2, s2, st2 = _run(q, k, v, a, s0, resets, segs)
    first = 64 * min(c for c in starts if where == "s0" or c > 1)
    assert o1[0, first:].isfinite().all() and s1.isfinite().all()  # what a reset promises
    for x, y in ((o2, o1), (s2, s1), (st2, st1)):
        x, y = x.float(), y.float()
        assert torch.equal(x.isfinite(), y.isfinite())
        ok = y.isfinite()
        # spans and the plain kernel round the same bf16 operands differently: as above
        assert (x[ok] - y[ok]).norm() < 1e-2 * y[ok].norm()


def test_span_rule_and_public_path():
    L = _lib.lib()
    assert L.ceo_efla_fwd_segments(8, 4096, 16, 128) == 1   # enough chains
    assert L.ceo_efla_fwd_segments(1, 512, 16, 64) == 1     # too few chunks
    assert L.ceo_efla_fwd_segments(1, 100, 16, 64) == 0     # refused as before
    assert L.ceo_efla_fwd_segments(1, 8192, 2, 64) >= 3
    g = torch.Generator(device="cuda").manual_seed(0)
    q = efla.l2norm(torch.randn(1, 2048, 2, 64, device="cuda", generator=g).bfloat16())
    v = torch.randn(1, 2048, 2, 64, device="cuda", generator=g).bfloat16()
    a = torch.full((1, 2048, 2), 0.1, device="cuda")
    o, s = efla.delta_rule(q, q, v, a)
    o1, s1, _ = _run(q, q, v, a, None, None, 1)
    assert (o.float() - o1.float()).norm() / o1.float().norm() < 5e-3
    assert (s - s1).norm() / s1.norm() < 5e-3
