"""Equally shaped Muon matrices in batched products against the update of one matrix at a time."""
import pytest
import torch

from ceo_b200.ops.matmul import gemm
from ceo_b200.optim.flat import FlatParams
from ceo_b200.optim.optimizers import ShardedOptimizer

pytestmark = pytest.mark.gpu


class _Mats(torch.nn.Module):
    def __init__(self, shapes, seed):
        super().__init__()
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.w = torch.nn.ParameterList(
            torch.nn.Parameter(torch.randn(s, device="cuda", generator=g).bfloat16())
            for s in shapes)


# wide, tall and square groups, one of them larger than the kernels' 32-entry table
@pytest.mark.parametrize("shapes", [[(64, 192)] * 3 + [(192, 64)] * 2 + [(8, 8)],
                                    [(72, 40)] * 35, [(256, 136)]])
@pytest.mark.parametrize("ns", ["cubic", "quintic"])
def test_groups_match_single_matrices(shapes, ns):
    opts = []
    for grouped in (True, False):
        m = _Mats(shapes, 5)
        flat = FlatParams(m)
        opt = ShardedOptimizer(flat, "lion_muon", max_grad_norm=1.0, muon_ns=ns)
        if not grouped:
            opt._muon_update = lambda segs, lr, gs, o=opt, f=flat: [
                o._muon_matrix(s, f.grads, lr, gs) for s in segs]
        for step in range(2):
            g = torch.Generator(device="cuda").manual_seed(step)
            flat.grads.copy_(torch.randn(flat.total, device="cuda", generator=g))
            opt.step(0.1)
        opts.append((flat, opt))
    (fa, a), (fb, b) = opts
    assert a._muon_state.keys() == b._muon_state.keys() and len(a._muon_state) == len(shapes)
    for n, st in a._muon_state.items():
        # the momentum is elementwise fp32; the update is bf16 Newton-Schulz from a Frobenius
        # norm summed in another order: an entry may round the other way (2^-8 relative)
        assert torch.allclose(st["momentum"], b._muon_state[n]["momentum"], rtol=1e-6, atol=1e-7)
        d = (st["master"] - b._muon_state[n]["master"]).norm()
        assert d <= 2 ** -7 * 0.1 * len(st["master"]) ** 0.5
    assert (fa.params.float() - fb.params.float()).abs().max() <= 2 ** -6


def test_newton_schulz_product_with_scaled_residual():
    g = torch.Generator(device="cuda").manual_seed(1)
    for M, N, K, nb in ((64, 64, 64, 1), (200, 136, 72, 3), (130, 24, 40, 2)):
        a = torch.randn(nb, M, K, device="cuda", generator=g).bfloat16()
        b = torch.randn(nb, N, K, device="cuda", generator=g).bfloat16()
        r = torch.randn(nb, M, N, device="cuda", generator=g).bfloat16()
        want = -0.5 * (a.double() @ b.double().transpose(1, 2)) + 1.5 * r.double()
        got = gemm(a, b, alpha=-0.5, residual=r, residual_scale=1.5)
        assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + 1e-4).all()
        got = gemm(a[0], b[0], alpha=-0.5, residual=r[0], residual_scale=1.5)
        assert ((got.double() - want[0]).abs() <= want[0].abs() * 2 ** -8 + 1e-4).all()


def test_skipped_step_leaves_groups_alone():
    m = _Mats([(64, 64)] * 2, 3)
    flat = FlatParams(m)
    opt = ShardedOptimizer(flat, "lion_muon", max_grad_norm=1.0)
    flat.grads.normal_()
    opt.step(0.1)
    before = {n: {k: v.clone() for k, v in st.items()} for n, st in opt._muon_state.items()}
    p = flat.params.clone()
    flat.grads.fill_(float("inf"))
    opt.step(0.1)
    assert torch.equal(p, flat.params)
    for n, st in opt._muon_state.items():
        for k, v in st.items():
            assert torch.equal(v, before[n][k])


def test_groups_are_bounded_in_memory():
    # 16 matrices of 2^24 elements: four at a time, three bf16 copies of them and four Gram matrices
    m = _Mats([(4096, 4096)] * 16, 2)
    flat = FlatParams(m)
    opt = ShardedOptimizer(flat, "lion_muon", max_grad_norm=1.0)
    flat.grads.normal_()
    opt.step(0.1)  # momentum and masters exist from here on
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    opt.step(0.1)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - held < 4 * 2 * 2 ** 26 + 2 ** 24


def test_state_loaded_from_slices_of_a_buffer():
    # tensors of a state already on the device are taken as they are, whatever their alignment
    shapes = [(64, 192)] * 3
    out = []
    for shift in (0, 1):
        flat = FlatParams(_Mats(shapes, 5))
        opt = ShardedOptimizer(flat, "lion_muon", max_grad_norm=1.0)
        flat.grads.copy_(torch.sin(torch.arange(flat.total, device="cuda").float()))
        opt.step(0.1)
        st = opt.state_dict()
        for one in st["muon"].values():
            for k, t in one.items():
                buf = torch.empty(t.numel() + 4, device="cuda")
                one[k] = buf[shift:shift + t.numel()].copy_(t)
        opt.load_state_dict(st)
        flat.grads.copy_(torch.cos(torch.arange(flat.total, device="cuda").float()))
        opt.step(0.1)
        out.append(flat.params.float())
    assert (out[0] - out[1]).abs().max() <= 2 ** -6
