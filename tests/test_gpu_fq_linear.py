"""QLinear's product on integer codes (fp32, PACT+ activations, per-channel SAWB+ weights) against 64-bit products of the same
fake-quantised operands, and the rule that chooses it.

Bounds.  Forward: the integer sums are exact; step, weight scale and bias contribute one fp32 rounding each (3 * 2^-24),
and the symmetric quantiser's values differ from (q - cv / step) * step by one rounding of the clip value.  Gradients:
31-bit fixed point per row (column) and one rounding at the end.  4e-7 relative Frobenius covers both; an fp32 GEMM of these
sizes shows 4e-7 to 1e-6."""

import pytest
import torch

from fms_model_optimizer_b200 import ops
from fms_model_optimizer_b200.modules import QLinear
from fms_model_optimizer_b200.modules import linear as ML

pytestmark = pytest.mark.gpu


def _make(dev, M, K, N, mode="pact+", bits=8, bias=True, seed=0):
    g = torch.Generator().manual_seed(seed)
    lin = QLinear(K, N, bias=bias, num_bits_feature=bits, qa_mode="pact+" if mode == "one-sided" else mode, num_bits_weight=8, qw_mode="sawb+perCh",
                  act_clip_init_val=3.0, act_clip_init_valn=-2.5, non_neg=mode == "one-sided", device=dev).train()  # fmt: skip
    with torch.no_grad():
        lin.weight.copy_(torch.randn(N, K, generator=g) * 0.02)
    return lin, torch.randn(M, K, generator=g).to(dev), torch.randn(M, N, generator=g).to(dev)


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("mode,bits", [("pact+", 8), ("pact+", 4), ("pactsym+", 8), ("one-sided", 8)])
@pytest.mark.parametrize("M,K,N", [(1, 16, 16), (130, 48, 272), (517, 768, 80), (2049, 1008, 528)])
def test_product_and_gradients(cuda_dev, monkeypatch, mode, bits, M, K, N):
    monkeypatch.setattr(ML, "_FQ_MIN_MACS", 0)
    lin, x, go = _make(cuda_dev, M, K, N, mode, bits)
    go *= torch.logspace(-6, 3, M, device=cuda_dev).view(-1, 1)  # rows of very different size
    qx, qw = lin.quantize_feature(x).detach().requires_grad_(True), lin.quantize_weight(lin.weight).detach().requires_grad_(True)
    act = lin._codes_route(qx, qw)
    assert act is not None
    out = ML._FakeQuantMatmul.apply(qx, qw, lin.bias, act, lin.quantize_weight.clip_val.detach().clone(), 8)
    gx, gw, gb = torch.autograd.grad(out, [qx, qw, lin.bias], go)
    xd, wd, gd = qx.detach().double(), qw.detach().double(), go.double()
    assert _rel(out.detach(), xd @ wd.t() + lin.bias.detach().double()) < 4e-7
    assert _rel(gw, gd.t() @ xd) < 4e-7
    assert _rel(gb, gd.sum(0)) < 4e-7
    want = gd @ wd
    err = (gx.double() - want).norm(dim=1) / want.norm(dim=1)  # every row on its own scale
    assert err.max().item() < 4e-7
    ops.check_status(cuda_dev)


def test_through_the_module_and_again(cuda_dev, monkeypatch):
    """The whole layer against itself on the library GEMM: same quantizer gradients, partial gradient requests, no bias, leading
    dimensions, and a backward pass that is differentiated."""
    monkeypatch.setattr(ML, "_FQ_MIN_MACS", 0)
    lin, x, go = _make(cuda_dev, 96, 64, 48, bias=False)
    x3, g3 = x.view(4, 24, 64).requires_grad_(True), go.view(4, 24, 48)
    params = [lin.weight, lin.quantize_feature.clip_val, lin.quantize_feature.clip_valn]
    got = torch.autograd.grad(lin(x3), [x3, *params], g3)
    monkeypatch.setattr(ML, "_FQ_MIN_MACS", 1 << 60)
    want = torch.autograd.grad(lin(x3), [x3, *params], g3)
    for a, b in zip(got, want):
        assert a.shape == b.shape and torch.allclose(a, b, rtol=2e-5, atol=2e-5)
    monkeypatch.setattr(ML, "_FQ_MIN_MACS", 0)
    (only_w,) = torch.autograd.grad(lin(x3.detach()), [lin.weight], g3)
    assert torch.equal(only_w, got[1])
    gg = g3.clone().requires_grad_(True)
    qx, qw = lin.quantize_feature(x3).detach().requires_grad_(True), lin.quantize_weight(lin.weight).detach().requires_grad_(True)
    out = ML._FakeQuantMatmul.apply(qx, qw, None, lin._codes_route(qx, qw), lin.quantize_weight.clip_val.detach().clone(), 8)
    gx, gw = torch.autograd.grad(out, [qx, qw], gg, create_graph=True)
    (twice,) = torch.autograd.grad(gx.sum() + (gw * gw).sum(), [gg])
    assert twice.shape == gg.shape and bool(torch.isfinite(twice).all())


def test_infinities_reach_the_gradients(cuda_dev, monkeypatch):
    monkeypatch.setattr(ML, "_FQ_MIN_MACS", 0)
    lin, x, go = _make(cuda_dev, 64, 32, 48)
    go[5, 7] = float("inf")
    go[9, 11] = float("nan")
    go[20] = 0
    x.requires_grad_(True)
    gx, gw, gb = torch.autograd.grad(lin(x), [x, lin.weight, lin.bias], go)
    assert not torch.isfinite(gw[7]).any() and not torch.isfinite(gw[11]).any() and not torch.isfinite(gb[[7, 11]]).any()
    rows = torch.tensor([i for i in range(48) if i not in (7, 11)], device=cuda_dev)
    assert bool(torch.isfinite(gw[rows]).all()) and bool((gx[20] == 0).all())
    inside = (x[5] > -2.5) & (x[5] < 3.0)
    assert not torch.isfinite(gx[5][inside]).any()
    keep = torch.tensor([i for i in range(64) if i not in (5, 9)], device=cuda_dev)
    assert bool(torch.isfinite(gx[keep]).all())


def test_rule(cuda_dev, monkeypatch):
    lin, x, _ = _make(cuda_dev, 64, 64, 48)
    qx, qw = lin.quantize_feature(x), lin.quantize_weight(lin.weight)
    assert lin._codes_route(qx, qw) is None  # too small
    monkeypatch.setattr(ML, "_FQ_MIN_MACS", 0)
    assert lin._codes_route(qx, qw) is not None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert lin._codes_route(qx, qw) is None
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        assert lin._codes_route(qx, qw) is None
    finally:
        torch.backends.cuda.matmul.allow_tf32 = False
    handle = lin.quantize_feature.register_forward_hook(lambda m, i, o: o * 1.5)
    assert lin._codes_route(qx, qw) is None
    handle.remove()
    assert lin._codes_route(qx.bfloat16(), qw.bfloat16()) is None
    odd = _make(cuda_dev, 64, 72, 48)[0]
    assert odd._codes_route(odd.quantize_feature(torch.randn(4, 72, device=cuda_dev)), odd.quantize_weight(odd.weight)) is None
    per_tensor = QLinear(64, 48, num_bits_feature=8, qa_mode="pact+", num_bits_weight=8, qw_mode="sawb+", device=cuda_dev)
    assert per_tensor._codes_route(qx, qw) is None
    with torch.no_grad():
        y = torch.func.vmap(lambda v: torch.nn.functional.linear(v, qw))(qx)  # a transform around the call keeps the library product
        assert torch.func.vmap(lambda v: torch.zeros(()) if lin._codes_route(qx, qw) is None else torch.ones(()))(qx).sum().item() == 0
    assert y.shape == (64, 48)
