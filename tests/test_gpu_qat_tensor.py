"""The QAT product on the tensor cores (csrc/qlin_qat.cu) at the sizes and values where it can go wrong: edges of its 256 x 128 / 192 / 256
tiles and 64-term stages, operands that it must hand to fp32, a clip value that changes between forward and backward, gradients
that are differentiated again, and the rule that leaves a call to the library.

Bound: a product of n terms summed in fp32 in any order is within 8 sqrt(n) 2^-24 of the sum of the terms' absolute values."""

import ctypes as C

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200.modules import QLinear
from fms_model_optimizer_b200.modules.linear import _ordinary_call

gpu = pytest.mark.gpu


MODES = {"two-sided": L.PACT_TWO_SIDED, "one-sided": L.PACT_ONE_SIDED, "symmetric": L.PACT_SYMMETRIC}


def _operands(t, k, n, clips=(3.0, -2.5), mode="two-sided"):
    g = torch.Generator(device="cuda").manual_seed(t + k + n)
    lin = QLinear(k, n, num_bits_feature=8, qa_mode="pactsym+" if mode == "symmetric" else "pact+", num_bits_weight=8, qw_mode="sawb+perCh",
                  act_clip_init_val=clips[0], act_clip_init_valn=clips[1], non_neg=mode == "one-sided", device="cuda").train()  # fmt: skip
    with torch.no_grad():
        lin.weight.copy_(torch.randn(n, k, generator=g, device="cuda") * 0.02)
        x = lin.quantize_feature(torch.randn(t, k, generator=g, device="cuda")).detach().requires_grad_(True)
        w = lin.quantize_weight(lin.weight).detach().requires_grad_(True)
    return lin, x, w, torch.randn(t, n, generator=g, device="cuda")


def _run(lin, x, w, mode="two-sided"):
    Qa, Qw = lin.quantize_feature, lin.quantize_weight
    return L.host().qat_linear(x, w, lin.bias, Qa.clip_val, getattr(Qa, "clip_valn", None), Qw.clip_val, 8, 8, MODES[mode])


class _Args(C.Structure):  # qlin_qat_args
    _fields_ = [(f, C.c_void_p) for f in ("x", "w", "g", "bias", "clip_x", "clipn_x", "clip_w", "step", "scale", "rcp", "x_codes", "w_codes", "g_planes", "d", "colsum",
                                          "workspace", "flags", "status")]  # fmt: skip
    _fields_ += [(f, C.c_int32) for f in ("tokens", "inp", "out", "num_bits_x", "num_bits_w", "variant")] + [("clip_kept", C.c_void_p)]


def _passes(lin, x, w, go, mode="two-sided", left_out=(), between=lambda: None):
    """Both passes through the C entry points: (flags of x and w in the forward pass, of x, w and the gradient in the backward pass) and
    (whether out, gx and gw were computed again in fp32).  The second is seen by putting zeros in the operands' place once their codes are
    made.  The flags start as memory that nobody cleared.  ``between`` is called between the passes."""
    lib, t, k, n = L.load(), x.shape[0], x.shape[1], w.shape[0]
    Qa, Qw = lin.quantize_feature, lin.quantize_weight
    dev = dict(device="cuda")
    f32 = {"step": torch.empty(1, **dev), "scale": torch.empty(n, **dev), "rcp": torch.empty(n, **dev), "clip_kept": torch.empty(1, **dev), "x": x.detach(), "w": w.detach(),
           "g": go, "clip_x": Qa.clip_val.detach(), "clip_w": Qw.clip_val, "d": None}  # fmt: skip
    if mode == "two-sided":
        f32["clipn_x"] = Qa.clip_valn.detach()
    codes = {"x_codes": t * k, "w_codes": n * k, "g_planes": 3 * t * n}
    codes = {f: torch.empty(c, dtype=torch.bfloat16, **dev) for f, c in codes.items()}
    kept = {f: v for f, v in codes.items() if f not in left_out}
    zeros = torch.zeros(max(t * k, n * k, t * n), **dev)
    flags = torch.ones(lib.qlin_qat_flag_count(), dtype=torch.int32, **dev)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def args(**other):
        ptr = {f: v.data_ptr() for f, v in {**f32, **codes, **other}.items() if v is not None}
        return C.byref(_Args(flags=flags.data_ptr(), tokens=t, inp=k, out=n, num_bits_x=8, num_bits_w=8, variant=MODES[mode], **ptr))

    raised, again = [], []
    for backward in (0, 1):
        if left_out and backward:
            codes = kept
            flags.fill_(1)
        L.check(lib.qlin_qat_codes(args(), C.c_int32(backward), stream), "qlin_qat_codes")
        if backward:
            L.check(lib.qlin_qat_split(args(), stream), "qlin_qat_split")
        if not left_out:
            counts = flags.view(3, -1)[: 2 + backward].clone()
            used = [((t * k // 8 + 255) // 256), ((n + 63) // 64) * ((k + 63) // 64), ((t + 15) // 16) * ((n + 1023) // 1024)]
            raised += [bool((counts[i, : used[i]] != 0).any()) for i in range(2 + backward)]
        for which in (1, 2) if backward else (0,):
            if left_out and (not backward or {1: "w_codes", 2: "x_codes"}[which] in left_out):
                continue
            d = torch.full((max(t * k, n * k, t * n),), float("nan"), **dev)
            L.check(lib.qlin_qat_product(args(d=d, x=zeros, w=zeros, g=zeros), C.c_int32(which), stream), "qlin_qat_product")
            again.append(bool((d.nan_to_num(1.0)[: (t * n, t * k, n * k)[which]] == 0).all()))
        between()
    return tuple(raised), tuple(again)


def _check(lin, x, w, go, out, grads):
    xd, wd, gd = x.detach().double(), w.detach().double(), go.double()
    bd = lin.bias.detach().double()
    for got, want, terms, n in (
        (out.detach(), xd @ wd.t() + bd, xd.abs() @ wd.abs().t() + bd.abs(), x.shape[1] + 1),
        (grads[0], gd @ wd, gd.abs() @ wd.abs(), w.shape[0]),
        (grads[1], gd.t() @ xd, gd.abs().t() @ xd.abs(), x.shape[0]),
        (grads[2], gd.sum(0), gd.abs().sum(0), x.shape[0]),
    ):
        assert bool(((got.double() - want).abs() <= 8 * n**0.5 * 2.0**-24 * terms + 1e-38).all())


@gpu
@pytest.mark.parametrize("t,k,n", [(1, 8, 8), (65, 64, 136), (257, 128, 264), (256, 72, 384), (1000, 200, 392), (63, 1032, 8), (3001, 520, 1048), (130, 4104, 776)])
def test_edges(cuda_dev, t, k, n):
    lin, x, w, go = _operands(t, k, n)
    out = _run(lin, x, w)
    _check(lin, x, w, go, out, torch.autograd.grad(out, [x, w, lin.bias], go))


@gpu
@pytest.mark.parametrize("t,k,n", [(1, 8, 8), (65, 64, 136), (257, 128, 264), (127, 72, 384), (1000, 200, 392), (129, 1032, 56), (63, 1032, 8), (3001, 520, 1048)])
def test_edges_of_the_product_in_fp32(cuda_dev, t, k, n):
    """Operands off the steps: every product is the fp32 one, with edges of its 128 x 64 tiles and 16-term stages, and once with a
    gradient off a 16-byte boundary."""
    lin, x, w, go = _operands(t, k, n)
    with torch.no_grad():
        x[t // 2, k // 2] += 0.003
        w[n // 2, k // 2] += 0.0007
    buf = torch.empty(t * n + 1, device="cuda")
    buf[1:] = go.flatten()
    out = _run(lin, x, w)
    for g in (go, buf[1:].view(t, n)):
        assert _passes(lin, x, w, g)[1] == (True, True, True)
        _check(lin, x, w, g, out, torch.autograd.grad(out, [x, w, lin.bias], g, retain_graph=True))


@gpu
@pytest.mark.parametrize("what", ["tiny gradient", "activation off the steps", "weight off the steps", "scales replaced", "gradient off 16 bytes"])
def test_operands_the_codes_cannot_carry(cuda_dev, what):
    t, k, n = 300, 264, 200
    lin, x, w, go = _operands(t, k, n)
    with torch.no_grad():
        if what == "tiny gradient":
            go *= 1e-34
        elif what == "activation off the steps":
            x[7, 9] += 0.003
        elif what == "weight off the steps":
            w[11, 13] *= 1.01
    out = _run(lin, x, w)
    if what == "scales replaced":  # as by another forward pass with new weights before this one's backward
        lin.quantize_weight.clip_val.mul_(1.5)
        with torch.no_grad():
            lin.quantize_feature.clip_val.mul_(0.5)
    if what == "gradient off 16 bytes":
        buf = torch.empty(t * n + 1, device="cuda")
        buf[1:] = go.flatten()
        go = buf[1:].view(t, n)
    _check(lin, x, w, go, out, torch.autograd.grad(out, [x, w, lin.bias], go))


@gpu
@pytest.mark.parametrize("mode", list(MODES))
def test_operands_that_a_hook_changed(cuda_dev, mode):
    """An operand scaled far below a step, and one element a single place off, are multiplied as they are."""
    t, k, n = 300, 264, 200
    lin, x, w, go = _operands(t, k, n, mode=mode)
    assert _passes(lin, x, w, go, mode) == ((False,) * 5, (False,) * 3)
    with torch.no_grad():
        lin.bias.zero_()
    for what in ("x", "w"):
        sx, sw = (1e-7, 1.0) if what == "x" else (1.0, 1e-7)
        xs, ws = (x.detach() * sx).requires_grad_(True), (w.detach() * sw).requires_grad_(True)
        flags = (what == "x", what == "w", what == "x", what == "w", False)
        again = (True, what == "w", what == "x")
        assert _passes(lin, xs, ws, go, mode) == (flags, again)
        out = _run(lin, xs, ws, mode)
        _check(lin, xs, ws, go, out, torch.autograd.grad(out, [xs, ws, lin.bias], go))
        x1, w1 = x.detach().clone(), w.detach().clone()
        e = (x1 if what == "x" else w1).view(-1)
        i = int(e.abs().argmax())
        e[i] = torch.nextafter(e[i], torch.zeros((), device="cuda"))
        assert _passes(lin, x1, w1, go, mode) == (flags, again)


@gpu
def test_large_gradients_stay_finite(cuda_dev):
    """Gradients whose product with the operand is an fp32 number, but not with the operand's codes or as g times a scale of 1."""
    t, k, n = 300, 264, 200
    lin, x, w, go = _operands(t, k, n)
    with torch.no_grad():
        w[5] = 0  # its scale counts as 1
        big = go.clone()
        big[:, 5] *= 1.4e36
        all_big = go * (2.0**122 / float(go.abs().max()))
        large = go * (2.0**36 / float((go * lin.quantize_weight.clip_val.view(1, -1) / 127).abs().max()))
        large[:, 5] = 0
        lin.quantize_weight.clip_val[5] = 0
    for g, flag in ((big, True), (all_big, True), (large, False)):
        assert _passes(lin, x, w, g) == ((False,) * 4 + (flag,), (False, flag, flag))
        out = _run(lin, x, w)
        grads = torch.autograd.grad(out, [x, w, lin.bias], g)
        assert all(bool(torch.isfinite(v).all()) for v in grads)
        _check(lin, x, w, g, out, grads)


@gpu
@pytest.mark.parametrize("what", ["a few", "a row and a column", "all", "subnormal", "beside a tiny scale"])
def test_tiny_gradients(cuda_dev, what):
    """Elements down to the smallest fp32 number, as in the tails of a GELU: the tensor cores carry them, to the last place that
    fp32 has, unless the weight's scale is so small beside the activations' that lost digits could show."""
    t, k, n = 300, 264, 200
    lin, x, w, go = _operands(t, k, n)
    g = torch.Generator(device="cuda").manual_seed(1)
    with torch.no_grad():
        if what in ("a few", "beside a tiny scale"):
            go[torch.rand(t, n, generator=g, device="cuda") < 0.02] = 1e-35
            go[:, ::7] *= 1e-12
            go[1::3, 1::9], go[2, 3] = 1e-42, 2.0**-149
        elif what == "a row and a column":
            go[5], go[:, 7] = go[5] * 1e-36, go[:, 7] * 1e-38
        elif what == "all":
            go *= 1e-33
        else:
            go *= 1e-40
        if what == "beside a tiny scale":
            w[3] *= 2.0**-40
            lin.quantize_weight.clip_val.view(-1)[3] *= 2.0**-40
    flag = what == "beside a tiny scale"
    assert _passes(lin, x, w, go) == ((False,) * 4 + (flag,), (False, flag, flag))
    got = torch.autograd.grad(_run(lin, x, w), [x, w], go)
    gd, xd, wd = go.double(), x.detach().double(), w.detach().double()
    for a, want, terms, m in ((got[0], gd @ wd, gd.abs() @ wd.abs(), n), (got[1], gd.t() @ xd, gd.abs().t() @ xd.abs(), t)):
        # in fp32 each product is rounded to a multiple of 2^-149
        assert bool(((a.double() - want).abs() <= 8 * m**0.5 * 2.0**-24 * terms + (m if flag else 1) * 2.0**-149).all())


@gpu
def test_operand_that_is_left_out(cuda_dev):
    """A caller of the C entry points that wants one gradient makes the codes of one operand; the other's flags are not looked at."""
    lin, x, w, go = _operands(300, 264, 200)
    for left_out in ("x_codes", "w_codes"):
        assert _passes(lin, x, w, go, left_out=(left_out,))[1] == (False,)


@gpu
def test_infinite_operands_give_what_fp32_gives(cuda_dev):
    lin, x, w, go = _operands(300, 264, 200)
    go[3, 5], go[8, 9], go[11] = float("inf"), float("nan"), 0
    out = _run(lin, x, w)
    got = torch.autograd.grad(out, [x, w], go)
    want = torch.autograd.grad(torch.nn.functional.linear(x, w, lin.bias), [x, w], go)
    for a, b in zip(got, want):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
        ok = torch.isfinite(b)
        assert torch.allclose(a[ok], b[ok], rtol=1e-4, atol=1e-5)


@gpu
def test_gradients_of_gradients_and_single_gradients(cuda_dev):
    lin, x, w, go = _operands(200, 136, 144)
    for leaf in (x, w, lin.bias):  # one gradient at a time
        (a,) = torch.autograd.grad(_run(lin, x, w), [leaf], go)
        (b,) = torch.autograd.grad(torch.nn.functional.linear(x, w, lin.bias), [leaf], go)
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max()))
    res = []
    for f in (lambda: _run(lin, x, w), lambda: torch.nn.functional.linear(x, w, lin.bias)):
        gx, gw = torch.autograd.grad(f(), [x, w], go, create_graph=True)
        res.append(torch.autograd.grad((gx * gx).sum() + (gw * gw).sum(), [x, w]))
    for a, b in zip(*res):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max()))


@gpu
def test_batched_gradients_and_modes_in_the_backward_pass(cuda_dev):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Watch(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    lin, x, w, go = _operands(200, 136, 144)
    gos = torch.stack([go, -2 * go, go.flip(0)])
    got = torch.autograd.grad(_run(lin, x, w), [x, w, lin.bias], gos, is_grads_batched=True)
    for i in range(3):
        want = torch.autograd.grad(torch.nn.functional.linear(x, w, lin.bias), [x, w, lin.bias], gos[i])
        for a, b in zip(got, want):
            assert torch.allclose(a[i], b, rtol=1e-4, atol=1e-4 * float(b.abs().max()))
    lin, x, _, go = _operands(1024, 512, 512)  # through the module, where its product is this one
    x = x.detach()
    assert type(lin._product(x, lin.weight).grad_fn).__name__ != "AddmmBackward0"
    (got,) = torch.autograd.grad(lin(x), [lin.weight], torch.stack([go, go * 2]), is_grads_batched=True)
    (want,) = torch.autograd.grad(lin(x), [lin.weight], go)
    assert torch.allclose(got[0], want, rtol=1e-4, atol=1e-3) and torch.allclose(got[1], 2 * want, rtol=1e-4, atol=1e-3)
    out = lin(x)
    with Watch() as mode:
        torch.autograd.grad(out, [lin.weight], go)
    assert any("mm" in f for f in mode.seen)


@gpu
@pytest.mark.parametrize("what", ["strides", "address", "expanded", "fewer bits"])
def test_saved_tensors_that_come_back_changed(cuda_dev, what):
    """Hooks on saved tensors that return the operands column by column, off a 16-byte boundary, as an expanded row, or rounded."""

    def unpack(t):
        if t.dim() != 2:
            return t
        if what == "strides":
            return t.t().contiguous().t()
        if what == "expanded":
            return t[:1].expand(t.shape)
        if what == "fewer bits":
            return t.bfloat16().float()
        buf = torch.empty(t.numel() + 1, device="cuda")
        buf[1:] = t.reshape(-1)
        return buf[1:].view(t.shape)

    lin, x, w, go = _operands(200, 136, 144)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), unpack):
        out = _run(lin, x, w)
    got = torch.autograd.grad(out, [x, w, lin.bias], go)
    for a, b in zip(got, (go @ unpack(w.detach()), go.t() @ unpack(x.detach()), go.sum(0))):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max()))


@gpu
def test_saved_scales_that_come_back_rounded(cuda_dev):
    """Hooks that keep saved tensors in bf16.  The activations are bf16 numbers, so the weight's gradient does not change; what the
    function saves besides the operands is its own affair."""
    lin, x, w, go = _operands(300, 264, 200, clips=(127 / 64, -128 / 64))
    assert torch.equal(x, x.bfloat16().float())
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().bfloat16(), lambda t: t.float()):
        out = _run(lin, x, w)
    (got,) = torch.autograd.grad(out, [w], go)
    terms = go.double().abs().t() @ x.detach().double().abs()
    assert bool(((got.double() - go.double().t() @ x.detach().double()).abs() <= 8 * 300**0.5 * 2.0**-24 * terms + 1e-38).all())


@gpu
def test_more_outputs_than_the_flags_cover(cuda_dev):
    """Wider than the gradient's split goes: the library's call, as every other one that the rule leaves out."""
    t, k, n = 128, 128, 1212424
    g = torch.Generator(device="cuda").manual_seed(0)
    lin = QLinear(k, n, num_bits_feature=8, qa_mode="pact+", num_bits_weight=8, qw_mode="sawb+perCh", device="cuda").train()
    x = torch.randn(t, k, generator=g, device="cuda")
    out = lin(x).detach()[:, -100:]
    with torch.no_grad():
        want = lin.quantize_feature(x).double() @ lin.quantize_weight(lin.weight)[-100:].double().t() + lin.bias[-100:]
    assert torch.allclose(out.double(), want, rtol=1e-4, atol=1e-4)


@gpu
@pytest.mark.parametrize("which", ["x", "w", "bias"])
def test_operands_that_are_stored_negated(cuda_dev, which):
    lin, x, w, _ = _operands(1024, 512, 512)
    with torch.no_grad():
        x, w, b = x.detach(), w.detach(), lin.bias.detach()
        if which == "bias":
            lin.bias = torch.nn.Parameter(torch._neg_view(b), requires_grad=False)
        args = (torch._neg_view(x) if which == "x" else x, torch._neg_view(w) if which == "w" else w)
        got = lin._product(*args).double()
    want = (-x if which == "x" else x).double() @ (-w if which == "w" else w).double().t() + (-b if which == "bias" else b)
    assert torch.allclose(got, want, rtol=1e-4, atol=1e-4)


@gpu
def test_memory_of_the_backward_pass(cuda_dev):
    """What the tensor cores' path needs beside the gradients: codes of one operand at a time and the parts of the gradient."""
    m, k, n = 16384, 4096, 128
    lin = QLinear(k, n, num_bits_feature=8, qa_mode="pact+", num_bits_weight=8, qw_mode="sawb+perCh", device="cuda").train()
    x, go = torch.randn(m, k, device="cuda").requires_grad_(True), torch.randn(m, n, device="cuda")
    assert L.host().qat_takes(x, lin.weight, lin.bias, torch.zeros(n, device="cuda"))
    for _ in range(2):
        out = lin(x)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        grads = torch.autograd.grad(out, [x, lin.weight], go)
        peak = torch.cuda.max_memory_allocated() - before
        del out, grads
    assert peak <= 2.5 * (m * k + n * k) * 4 + 6 * m * n


@gpu
def test_rule(cuda_dev):
    host = L.host()
    lin, x, w, _ = _operands(1024, 512, 512)
    cw = lin.quantize_weight.clip_val
    assert host.qat_takes(x, w, lin.bias, cw) and host.qat_takes(x.view(4, 256, 512), w, None, cw)
    assert not host.qat_takes(x[:100], w, lin.bias, cw)  # too small
    assert not host.qat_takes(x[:, :256], w[:, :256], lin.bias, cw)  # not dense
    assert not host.qat_takes(x.half(), w.half(), None, cw)
    assert not host.qat_takes(x.cpu(), w.cpu(), None, cw.cpu())
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not host.qat_takes(x, w, lin.bias, cw)
    before = torch.backends.cuda.matmul.fp32_precision
    torch.backends.cuda.matmul.fp32_precision = "tf32"
    try:
        assert not host.qat_takes(x, w, lin.bias, cw)
    finally:
        torch.backends.cuda.matmul.fp32_precision = before
    assert type(lin._product(x, w).grad_fn).__name__ != type(torch.nn.functional.linear(x, w, lin.bias).grad_fn).__name__


def test_calls_that_something_watches_stay_with_the_library():
    from torch.utils._python_dispatch import TorchDispatchMode

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    x = torch.ones(2, 2)
    assert _ordinary_call(x, torch.nn.Parameter(x.clone()), None)
    assert not _ordinary_call(x, x.as_subclass(Sub))
    with Watch():
        assert not _ordinary_call(x)
    seen = []
    torch.func.vmap(lambda t: (seen.append(_ordinary_call(t)), t)[1])(x)
    with torch.autograd.forward_ad.dual_level():
        seen.append(_ordinary_call(x))
    torch.jit.trace(lambda t: (seen.append(_ordinary_call(t)), t + 1)[1], x, check_trace=False)
    assert seen == [False, False, False]
