"""QLinear's product in fp32 at sizes of 2^32 multiply-adds and more, for every PACT+ quantizer, clip values whose codes
reach one beyond [0, 255] (symmetric pairs, zero points on a half), sparse activations, NaN, and gradients of a wide range: output and
gradients against 64-bit products of the same fake-quantised operands, element by element.

Bound: a sum of n fp32 products in any order, each product and addition rounded once, is within 8 sqrt(n) 2^-24 of the sum of
the terms' absolute values, element by element (Higham and Mary's probabilistic bound; with the factor 8 it fails for one
element in 10^13).  An element whose large terms meet a zero is held to the size of the terms that are left."""

import pytest
import torch

from fms_model_optimizer_b200.modules import QLinear

pytestmark = pytest.mark.gpu

M, K, N = 2048, 1024, 2048


def _make(dev, mode="pact+", clips=(8.0, -8.0), shape=(M, K, N)):
    m, k, n = shape
    g = torch.Generator(device=dev).manual_seed(0)
    lin = QLinear(k, n, num_bits_feature=8, qa_mode="pact+" if mode == "one-sided" else mode, num_bits_weight=8, qw_mode="sawb+perCh",
                  act_clip_init_val=clips[0], act_clip_init_valn=clips[1], non_neg=mode == "one-sided", device=dev).train()  # fmt: skip
    with torch.no_grad():
        lin.weight.copy_(torch.randn(n, k, generator=g, device=dev) * 0.02)
    x = torch.randn(m, k, generator=g, device=dev) * clips[0] * 0.7  # about 8 % of the values beyond each clip
    return lin, x, torch.randn(m, n, generator=g, device=dev)


def _operands(lin, x):
    with torch.no_grad():
        return lin.quantize_feature(x).double(), lin.quantize_weight(lin.weight).double()


def _within(got, want, terms, n):
    return bool(((got.double() - want).abs() <= 8 * n**0.5 * 2.0**-24 * terms + 1e-38).all())


def _check(lin, x, go, gradients=True):
    qx, qw = _operands(lin, x)
    out = lin(x.requires_grad_(True))
    bias = lin.bias.detach().double()
    assert _within(out.detach(), qx @ qw.t() + bias, qx.abs() @ qw.abs().t() + bias.abs(), qx.shape[1] + 1)
    if not gradients:
        return
    gx, gw, gb = torch.autograd.grad(out, [x, lin.weight, lin.bias], go)
    gd = go.double()
    assert _within(gw, gd.t() @ qx, gd.abs().t() @ qx.abs(), qx.shape[0])
    assert _within(gb, gd.sum(0), gd.abs().sum(0), qx.shape[0])
    # the quantizer passes the product's gradient on inside the clips and stops it at and outside them
    Qa = lin.quantize_feature
    hi = Qa.clip_val.detach()
    lo = Qa.clip_valn.detach() if hasattr(Qa, "clip_valn") else (-hi if type(Qa).__name__ == "PACTplusSym" else 0.0)
    want = torch.where((x > lo) & (x < hi), gd @ qw, 0.0)
    assert _within(gx, want, gd.abs() @ qw.abs(), qw.shape[0])


# 8.0 / -8.0 are the module's defaults.  With an 8-bit code of 256 at the upper clip (symmetric pairs, 8.7 / -1.5), of -1 at
# the lower one (5.01 / -1.002), and within [0, 255]
@pytest.mark.parametrize("clips", [(8.0, -8.0), (6.0, -6.0), (3.0, -3.0), (8.7, -1.5), (5.01, -1.002), (3.0, -2.5)])
def test_two_sided(cuda_dev, clips):
    _check(*_make(cuda_dev, clips=clips))


@pytest.mark.parametrize("mode", ["pactsym+", "one-sided"])
def test_other_quantizers(cuda_dev, mode):
    _check(*_make(cuda_dev, mode, (4.0, -4.0)))


@pytest.mark.parametrize("mode,clips", [("one-sided", (4.0, -4.0)), ("pact+", (8.0, -1.0))])
def test_sparse_activations(cuda_dev, mode, clips):
    """One value in a thousand is not zero, as behind a gate or a ReLU; weights with a mean."""
    lin, x, go = _make(cuda_dev, mode, clips)
    with torch.no_grad():
        lin.weight += 0.02
        lin.bias.zero_()
    x *= torch.rand(M, K, generator=torch.Generator(device=cuda_dev).manual_seed(1), device=cuda_dev) < 1e-3
    _check(lin, x, go, gradients=False)


@pytest.mark.parametrize("ratio", [2.0**16, 2.0**24, 2.0**40])
def test_gradient_with_one_large_element_a_row(cuda_dev, ratio):
    lin, x, go = _make(cuda_dev, clips=(3.0, -2.5))
    go[torch.arange(M, device=cuda_dev), torch.arange(M, device=cuda_dev) % N] *= ratio
    _check(lin, x, go)


def test_nan_activation(cuda_dev):
    lin, x, go = _make(cuda_dev, "pactsym+", (4.0, -4.0))
    x[3, 5] = float("nan")
    qx, _ = _operands(lin, x)
    assert bool(torch.isnan(qx[3, 5])) and int(torch.isnan(qx).sum()) == 1  # the symmetric quantizer keeps it
    out = lin(x.requires_grad_(True))
    (gw,) = torch.autograd.grad(out, [lin.weight], go)
    assert bool(torch.isnan(out[3]).all()) and int(torch.isnan(out).sum()) == N
    assert bool(torch.isnan(gw[:, 5]).all()) and int(torch.isnan(gw).sum()) == N


def test_gradient_that_starts_off_a_16_byte_boundary(cuda_dev):
    lin, x, go = _make(cuda_dev)
    leaf = [x.requires_grad_(True), lin.weight, lin.bias]
    want = torch.autograd.grad(lin(x), leaf, go)
    aux = torch.zeros(3, device=cuda_dev, requires_grad=True)
    joined = torch.cat([aux, lin(x).flatten()])  # the gradient of the output is a slice that starts at element 3
    got = torch.autograd.grad(joined, leaf, torch.cat([torch.zeros(3, device=cuda_dev), go.flatten()]))
    for a, b in zip(got, want):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max()))


@pytest.mark.parametrize("where", ["matmul", "all"])
def test_tf32_by_the_current_switch(cuda_dev, where):
    lin, x, _ = _make(cuda_dev)
    owner = torch.backends.cuda.matmul if where == "matmul" else torch.backends
    before = owner.fp32_precision
    owner.fp32_precision = "tf32"
    try:
        out = lin(x).detach()
    finally:
        owner.fp32_precision = before
    qx, qw = _operands(lin, x)
    assert ((out.double() - lin.bias.detach().double() - qx @ qw.t()).norm() / out.double().norm()).item() < 1e-2


def test_memory_of_the_backward_pass(cuda_dev):
    """Gradients of a call with few outputs need the gradients and an operand's size, not several times that."""
    m, k, n = 16384, 4096, 64
    lin, x, go = _make(cuda_dev, shape=(m, k, n))
    x.requires_grad_(True)
    peak = []
    for _ in range(2):  # the first pass takes the library's workspace
        out = lin(x)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        grads = torch.autograd.grad(out, [x, lin.weight], go)
        peak.append(torch.cuda.max_memory_allocated() - before)
        del out, grads
    assert peak[-1] <= 2.5 * (m * k + n * k) * 4  # the product's input gradient, the quantizer's, and half of one to spare


def test_infinities_reach_the_gradients(cuda_dev):
    lin, x, go = _make(cuda_dev)
    go[5, 7] = float("inf")
    go[9, 11] = float("nan")
    go[20] = 0
    gx, gw, gb = torch.autograd.grad(lin(x.requires_grad_(True)), [x, lin.weight, lin.bias], go)
    hit = torch.zeros(N, dtype=torch.bool, device=cuda_dev)
    hit[[7, 11]] = True
    assert not torch.isfinite(gw[hit]).any() and not torch.isfinite(gb[hit]).any() and bool(torch.isfinite(gw[~hit]).all())
    assert bool((gx[20] == 0).all())
    inside = (x[5] > -8) & (x[5] < 8)
    assert not torch.isfinite(gx[5][inside]).any()
    rows = torch.ones(M, dtype=torch.bool, device=cuda_dev)
    rows[[5, 9]] = False
    assert bool(torch.isfinite(gx[rows]).all())
