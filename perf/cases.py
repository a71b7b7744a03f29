"""The work this package is used for, as cases that can be timed and checked.

Each kind of case is one thing a program calls: a deployed int8 Linear (dynamic or static activation quantisation), the
FP8 Linear (inference, and a training step), the chunk-truncating integer product, a QAT activation quantizer and a QAT
Linear (forward and backward), the quantized batched product of an attention block, and the decoder as a whole.  Sizes
are those of this repository's benchmark (decoder projections of width 4096 / 14336, encoder projections of width 768 /
3072, prompts of up to 16384 tokens, decode batches of 1 to 128) and ragged sizes between them.
"""

import math

import torch
import torch.nn.functional as F

from fms_model_optimizer_b200 import ops
from fms_model_optimizer_b200.decoder import W8A8Decoder
from fms_model_optimizer_b200.modules import LinearFPxAcc, QBmm, QBmmINT8Deploy, QLinear, QLinearINT8Deploy
from fms_model_optimizer_b200.quant.quantizers import get_activation_quantizer

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # one token of one sequence through an MLP projection: the weights are the traffic
        dict(name="w8a8 decode", kind="deploy", tokens=1, k=4096, n=14336, dtype="bf16", act="dynamic", bias=False),
        # a decode batch through the down projection
        dict(name="w8a8 decode batch", kind="deploy", tokens=37, k=14336, n=4096, dtype="bf16", act="dynamic", bias=False),
        # a short prompt of odd length, fp16 model with biases
        dict(name="w8a8 short prompt", kind="deploy", tokens=517, k=4096, n=4096, dtype="fp16", act="dynamic", bias=True),
        # prefill of 8 prompts of 2048 tokens
        dict(name="w8a8 prefill", kind="deploy", tokens=16384, k=4096, n=4096, dtype="bf16", act="dynamic", bias=False),
        # an encoder batch of 32 x 128 tokens in fp32 with a calibrated (static) activation range
        dict(name="w8a8 static encoder", kind="deploy", tokens=4096, k=768, n=3072, dtype="fp32", act="static", bias=True),
        # FP8 inference, per-token scales: prefill through the down projection
        dict(name="fp8 prefill", kind="fp8", tokens=8192, k=14336, n=4096, dtype="bf16", bias=False),
        # FP8 training step of one projection: per-tensor scales, e4m3 forward, e5m2 backward
        dict(name="fp8 training step", kind="fp8_train", tokens=4096, k=4096, n=4096, dtype="bf16"),
        # emulation of a narrow accumulator: chunks of 64, 8 truncated bits
        dict(name="int8 chunk truncate", kind="chunk", m=4096, k=8192, n=4096, chunk=64, bits=8),
        # QAT of a decoder: the PACT+ quantizer of one Linear input, forward and backward
        dict(name="qat activations", kind="pact", rows=8192, cols=4096, dtype="bf16", mode="pact+"),
        # QAT of an encoder: forward and backward of one Linear, PACT+ activations and SAWB+ per-channel weights
        dict(name="qat linear", kind="qat", tokens=4096, k=768, n=3072, dtype="fp32"),
        # attention scores q @ k^T of two sequences of 2048 tokens with 32 heads
        dict(name="int8 attention scores", kind="bmm", heads=64, m=2048, k=128, n=2048, dtype="bf16", what="scores"),
        # a whole call: two full-width decoder layers, two prompts of 1024 tokens, next-token logits
        dict(name="decoder", kind="decoder", layers=2, batch=2, seq=1024, vocab=32000),
    ]


PROJECTIONS = [(4096, 4096), (4096, 1024), (4096, 14336), (14336, 4096), (768, 768), (768, 3072), (3072, 768)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _projection(rng, step):
    """A projection's (k, n): half the time one of a decoder or an encoder, else a width of its own."""
    if rng.random() < 0.5:
        return rng.choice(PROJECTIONS)
    return _log(rng, 256 // step, 8192 // step) * step, _log(rng, 256 // step, 8192 // step) * step


def draw(rng):
    kind = rng.choice(["deploy"] * 5 + ["fp8"] * 2 + ["fp8_train", "chunk", "pact", "qat", "bmm", "bmm", "decoder"])
    if kind == "deploy":
        act, dtype = rng.choice([("dynamic", "bf16"), ("dynamic", "bf16"), ("dynamic", "fp16"), ("dynamic", "fp32"), ("static", "fp32"), ("static", "bf16")])
        k, n = _projection(rng, rng.choice([8, 16, 16, 64]))
        return dict(kind=kind, tokens=min(_log(rng, 1, 16384), 16384 * 4096 * 4096 // (k * n)), k=k, n=n, dtype=dtype, act=act, bias=rng.random() < 0.5)
    if kind == "fp8":
        k, n = _projection(rng, rng.choice([16, 64]))
        return dict(kind=kind, tokens=_log(rng, 1, 8192), k=k, n=n, dtype=rng.choice(["bf16", "bf16", "fp32"]), bias=rng.random() < 0.5)
    if kind == "fp8_train":
        k, n = rng.choice([(4096, 4096), (768, 3072), (3072, 768), (_log(rng, 16, 256) * 16, _log(rng, 16, 256) * 16)])
        return dict(kind=kind, tokens=_log(rng, 8, 256) * 16 + rng.choice([0, 0, 5]), k=k, n=n, dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "chunk":
        return dict(kind=kind, m=_log(rng, 32, 4096), k=_log(rng, 4, 128) * 64, n=_log(rng, 16, 512) * 8, chunk=rng.choice([32, 64, 64, 128]), bits=rng.choice([6, 8, 8, 10]))
    if kind == "pact":
        return dict(kind=kind, rows=_log(rng, 16, 8192), cols=rng.choice([768, 3072, 4096, 1000 + rng.randrange(1000)]), dtype=rng.choice(["bf16", "bf16", "fp32", "fp16"]),
                    mode=rng.choice(["pact+", "pactsym+"]))  # fmt: skip
    if kind == "qat":
        k, n = rng.choice([(768, 768), (768, 3072), (3072, 768)])
        return dict(kind=kind, tokens=_log(rng, 64, 4096), k=k, n=n, dtype="fp32")
    if kind == "bmm":
        seq = _log(rng, 100, 2048)
        what = rng.choice(["scores", "scores", "values"])
        heads = min(rng.choice([12, 24, 32, 64]), max(8, 64 * 2048 * 2048 // (seq * seq) // 8 * 8))
        d = rng.choice([64, 128])
        return dict(kind=kind, heads=heads, m=seq, k=d if what == "scores" else seq, n=seq if what == "scores" else d, dtype=rng.choice(["bf16", "fp16", "fp32"]), what=what)
    return dict(kind=kind, layers=rng.choice([1, 2]), batch=rng.choice([1, 2]), seq=_log(rng, 2, 128) * 8, vocab=rng.choice([32000, 16000]))


# ------------------------------------------------------------------------------------------------ inputs and state
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) & 0x7FFFFFFF)


def _act(g, rows, cols, dtype):
    """Activations as a normalised hidden state has them: N(0, 1) with one channel in a hundred twenty times larger."""
    x = torch.randn(rows, cols, generator=g, device="cuda")
    x[:, torch.randperm(cols, generator=g, device="cuda")[: max(1, cols // 100)]] *= 20
    return x.to(dtype)


def _weight(g, n, k, dtype):
    return (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(dtype)


def _qlinear(case, g, dtype, **kw):
    lin = QLinear(case["k"], case["n"], bias=case.get("bias", True), num_bits_feature=8, num_bits_weight=8, device="cuda", **kw)
    with torch.no_grad():
        lin.weight.copy_(_weight(g, case["n"], case["k"], torch.float32))
        if lin.bias is not None:
            lin.bias.copy_(torch.randn(case["n"], generator=g, device="cuda") * 0.01)
    return lin.to(dtype)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    dtype = DTYPES[case.get("dtype", "bf16")]
    s = {"case": case}
    if kind == "deploy":
        dynamic = case["act"] == "dynamic"
        kw = dict(qa_mode="pertokenmax" if dynamic else "pact+", qw_mode="maxperCh", act_clip_init_val=6.0, act_clip_init_valn=-5.0)
        if dynamic:
            kw["qcfg"] = {"smoothq": True, "smoothq_alpha": 0.5}
        lin = _qlinear(case, g, dtype, **kw)
        s["x"] = _act(g, case["tokens"], case["k"], dtype) if dynamic else (torch.randn(case["tokens"], case["k"], generator=g, device="cuda") * 1.5).to(dtype)
        if dynamic:  # the calibrated activation scale: the absolute maximum of each input channel
            lin.set_act_scale(_act(g, 256, case["k"], torch.float32).abs().amax(0))
        lin.train()
        with torch.no_grad():
            lin(torch.zeros(1, case["k"], device="cuda", dtype=dtype))  # latches the weight quantizer's clip values
        lin.eval()
        s["mod"] = QLinearINT8Deploy.from_fms_mo(lin, use_dynamic_max_act_Qfunc=-1 if dynamic else False, use_PT_native_Qfunc=not dynamic)
        del lin
    elif kind in ("fp8", "fp8_train"):
        lin = torch.nn.Linear(case["k"], case["n"], bias=case.get("bias", True), device="cuda", dtype=dtype)
        with torch.no_grad():
            lin.weight.copy_(_weight(g, case["n"], case["k"], dtype))
            if lin.bias is not None:
                lin.bias.copy_(torch.randn(case["n"], generator=g, device="cuda") * 0.01)
        s["mod"] = LinearFPxAcc.from_nn(lin, dynamic_fp8="per_token" if kind == "fp8" else "per_tensor", chunk_size=64)
        s["x"] = _act(g, case["tokens"], case["k"], dtype)
        if kind == "fp8_train":
            s["x"].requires_grad_(True)
            s["g"] = (torch.randn(case["tokens"], case["n"], generator=g, device="cuda") * 1e-3).to(dtype)
        else:
            with torch.no_grad():
                s["mod"](s["x"][:1])  # the module keeps the weight's codes from its first call on
    elif kind == "chunk":
        s["a"] = torch.randn(case["m"], case["k"], generator=g, device="cuda").mul_(32).round_().clamp_(-127, 127).to(torch.int8)
        s["b"] = torch.randn(case["n"], case["k"], generator=g, device="cuda").mul_(32).round_().clamp_(-127, 127).to(torch.int8).t()
    elif kind == "pact":
        s["q"] = get_activation_quantizer(case["mode"], nbits=8, clip_val=3.0, clip_valn=-2.5, align_zero=True).cuda()
        s["x"] = (torch.randn(case["rows"], case["cols"], generator=g, device="cuda") * 1.5).to(dtype).requires_grad_(True)
        s["g"] = (torch.randn(case["rows"], case["cols"], generator=g, device="cuda") + 0.5 * s["x"].detach().float()).to(dtype)
    elif kind == "qat":
        s["mod"] = _qlinear(case, g, dtype, qa_mode="pact+", qw_mode="sawb+perCh", act_clip_init_val=3.0, act_clip_init_valn=-2.5).train()
        s["x"] = torch.randn(case["tokens"], case["k"], generator=g, device="cuda").to(dtype).requires_grad_(True)
        s["g"] = torch.randn(case["tokens"], case["n"], generator=g, device="cuda").to(dtype)
    elif kind == "bmm":
        scores = case["what"] == "scores"
        # clip values whose zero point is 128 (symmetric codes): the reference's correction term does not broadcast for scores
        q = QBmm(num_bits_m1=8, qm1_mode="pactsym+", num_bits_m2=8, qm2_mode="pactsym+", m1_clip_init_val=7.0 if scores else 0.1875, m2_clip_init_val=7.0,
                 qcfg={})  # fmt: skip
        s["mod"] = QBmmINT8Deploy.from_fms_mo(q, target_device="cuda")
        h, m, k, n = case["heads"], case["m"], case["k"], case["n"]
        lead = (h // 4, 4)
        if scores:
            s["a"] = torch.randn(*lead, m, k, generator=g, device="cuda").to(dtype)
            s["b"] = torch.randn(*lead, n, k, generator=g, device="cuda").to(dtype).transpose(-1, -2)
        else:  # probabilities times values
            s["a"] = torch.softmax(torch.randn(*lead, m, k, generator=g, device="cuda") * 3, -1).to(dtype)
            s["b"] = torch.randn(*lead, k, n, generator=g, device="cuda").to(dtype)
    else:
        cfg = dict(layers=case["layers"], hidden=4096, q_heads=32, kv_heads=8, head_dim=128, ffn=14336, vocab=case["vocab"], rope_theta=500000.0,
                   batch=case["batch"], seq=case["seq"])  # fmt: skip
        s["mod"] = W8A8Decoder(cfg, torch.device("cuda", 0))
        s["ids"] = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=g, device="cuda")
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "deploy":
        return s["mod"](s["x"])
    if kind == "fp8":
        with torch.no_grad():
            return s["mod"](s["x"])
    if kind == "chunk":
        return ops.tl_matmul_chunk_truncate(s["a"], s["b"], chunk_trun_bits=s["case"]["bits"], chunk_size=s["case"]["chunk"])
    if kind == "pact":
        params = list(s["q"].parameters())
        out = s["q"](s["x"])
        return (out, *torch.autograd.grad(out, [s["x"], *params], s["g"]))
    if kind in ("qat", "fp8_train"):
        params = list(s["mod"].parameters())
        out = s["mod"](s["x"])
        return (out, *torch.autograd.grad(out, [s["x"], *params], s["g"]))
    if kind == "bmm":
        return s["mod"](s["a"], s["b"])
    with torch.no_grad():
        tokens = s["mod"].forward(s["ids"])
        return tokens, F.linear(s["mod"].last_hidden, s["mod"].lm_head)


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    kind = case["kind"]
    e = {"bf16": 2, "fp16": 2, "fp32": 4}[case.get("dtype", "bf16")]
    if kind in ("deploy", "fp8"):
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"bytes": t * k * e + n * k + 8 * n + t * n * e, "flops": 2 * t * n * k}
    if kind == "fp8_train":
        t, k, n = case["tokens"], case["k"], case["n"]
        # x, w and the gradient read; output, input gradient, weight gradient written
        return {"bytes": 2 * (t * k + n * k + t * n) * e, "flops": 6 * t * n * k}
    if kind == "chunk":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": m * k + n * k + 4 * m * n, "flops": 2 * m * n * k}
    if kind == "pact":
        v = case["rows"] * case["cols"]
        return {"bytes": 4 * v * e, "flops": 20 * v}  # x and the gradient read, output and input gradient written
    if kind == "qat":
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"bytes": 2 * (t * k + n * k + t * n) * e, "flops": 6 * t * n * k}
    if kind == "bmm":
        h, m, k, n = case["heads"], case["m"], case["k"], case["n"]
        return {"bytes": h * (m * k + n * k + m * n) * e, "flops": 2 * h * m * n * k}
    t, per_layer = case["batch"] * case["seq"], 4096 * (4096 + 1024 + 1024 + 4096 + 3 * 14336)
    return {"bytes": case["layers"] * (per_layer + 4 * t * 4096) + case["vocab"] * 4096 * 2,
            "flops": case["layers"] * (2 * t * per_layer + 2 * t * case["seq"] * 4096) + 2 * case["batch"] * case["vocab"] * 4096}  # fmt: skip


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rnd(v, dtype):
    return v.to(dtype).double()


def exact(case, seed):
    """The operators' definitions with sums, products and scales in 64 bits.  Codes are part of the definition (they depend
    on the model's data type: a scale that is a bf16 number gives other codes than one that is not), so the quantisers'
    own rounding steps to that type are kept; everything from the codes on is unrounded."""
    kind = case["kind"]
    if kind == "decoder":
        return None
    s = prepare(case, seed)
    dtype = DTYPES[case.get("dtype", "bf16")]
    if kind == "deploy":
        m, x = s["mod"], s["x"].double()
        w, ws, b = m.weight.double(), m.w_scale.double(), m.bias.double()
        if case["act"] == "dynamic":
            sq = m.smoothq_scale
            v = _rnd(x / sq.double(), dtype) if bool((sq != 1).all()) else x
            eps = torch.tensor(1e-5, dtype=dtype, device="cuda").double()
            sc = _rnd(v.abs().amax(-1, keepdim=True).clamp(min=eps) / 127, dtype)
            codes = _rnd(v / sc, dtype).round().to(torch.int32).to(torch.int8).double()  # the codes wrap, they are not clamped
        else:
            sc = m.input_scale.double()
            d = torch.promote_types(dtype, m.input_scale.dtype)
            codes = _rnd(_rnd(_rnd(x / sc, d) + m.input_zp.double(), d) - 128, d).round().clamp(-128, 127)
        return (codes @ w.t()) * (sc * ws) + b
    if kind in ("fp8", "fp8_train"):
        m, x = s["mod"], s["x"].detach().double()
        w, b = m.weight.detach().double(), (m.bias.detach().double() if m.bias is not None else 0.0)

        def codes(v, dim, top, eps, f8):
            a = v.abs().amax(dim, keepdim=True) if dim is not None else v.abs().max()
            sc = _rnd(a / top, dtype)
            if eps:
                sc = sc.clamp(min=float(torch.tensor(eps, dtype=dtype)))
            return (v / sc).to(dtype).to(f8).double(), sc

        if kind == "fp8":
            xq, xs = codes(x, -1, 448.0, 1e-5, torch.float8_e4m3fn)
            wq, ws = codes(w, -1, 448.0, 1e-5, torch.float8_e4m3fn)
            return (xq @ wq.t()) * xs * ws.t() + b
        xq, xs = codes(x, None, 448.0, 1e-5, torch.float8_e4m3fn)
        wq, ws = codes(w, None, 448.0, 1e-5, torch.float8_e4m3fn)
        out = (xq @ wq.t()) * xs * ws + b
        xq, xs = codes(x, None, 57344.0, 0.0, torch.float8_e5m2)
        wq, ws = codes(w, None, 57344.0, 0.0, torch.float8_e5m2)
        gq, gs = codes(s["g"].double(), None, 57344.0, 0.0, torch.float8_e5m2)
        return out, (gq @ wq) * gs * ws, (gq.t() @ xq) * gs * xs, gq.sum(0)
    if kind == "chunk":
        a, b, bits = s["a"].float(), s["b"].float(), case["bits"]  # sums of at most 128 products below 2^14: exact in fp32
        acc = torch.zeros(case["m"], case["n"], dtype=torch.int32, device="cuda")
        tf32, torch.backends.cuda.matmul.allow_tf32 = torch.backends.cuda.matmul.allow_tf32, False
        for c in range(0, case["k"], case["chunk"]):
            p = (a[:, c : c + case["chunk"]] @ b[c : c + case["chunk"]]).to(torch.int32)
            acc += ((p + (1 << (bits - 1))) >> bits) << bits
        torch.backends.cuda.matmul.allow_tf32 = tf32
        return acc
    if kind in ("pact", "qat"):
        x, g = s["x"].detach().double(), s["g"].double()
        mod = s["q"] if kind == "pact" else s["mod"].quantize_feature
        cv = float(mod.clip_val.to(dtype))
        sym = not hasattr(mod, "clip_valn")
        if sym:  # codes of (x + cv) / step, 2^8 - 2 levels
            cvn, levels = -cv, 254.0
            step = 2 * cv / levels
            q = ((x.clamp(cvn, cv) - cvn) / step).round() * step + cvn
        else:  # an integral zero point, 2^8 - 1 levels
            cvn, levels = float(mod.clip_valn.to(dtype)), 255.0
            step = (cv - cvn) / levels
            zp = round(cvn / step)
            q = ((x.clamp(cvn, cv) / step - zp).round() + zp) * step
        out, gq, extra = q, g, ()
        if kind == "qat":
            m = s["mod"]
            w, b = m.weight.detach().double(), m.bias.detach().double()
            clip = 31.76 * (w * w).mean(1, keepdim=True).sqrt() - 35.04 * w.abs().mean(1, keepdim=True)
            ws = clip * 2 / 254
            wq = (w / ws).round().clamp(-127, 127) * ws
            out, gq, extra = q @ wq.t() + b, g @ wq, (g.t() @ q, g.sum(0))
        hi, lo = x >= cv, x <= cvn
        z = (x - cvn) / step
        d = (z - z.round()) / levels
        zero = torch.zeros((), dtype=torch.float64, device="cuda")
        gx = torch.where(hi | lo, zero, gq)
        if sym:
            clips = (torch.where(hi, gq, torch.where(lo, -gq, -2 * d * gq)).sum().reshape(1),)
        else:
            clips = (torch.where(hi, gq, torch.where(lo, zero, -gq * d)).sum().reshape(1), torch.where(lo, gq, torch.where(hi, zero, gq * d)).sum().reshape(1))
        return (out, gx, *extra, *clips)
    m = s["mod"]

    def codes8(v, sc, zp):
        d = torch.promote_types(dtype, sc.dtype)
        return _rnd(_rnd(v.double() / sc.double(), d) + zp, d).round().clamp(-128, 127)

    a, b = codes8(s["a"], m.m1_scale, int(m.m1_zp) - 128), codes8(s["b"], m.m2_scale, int(m.m2_zp))
    return (a @ b) * m.m1_scale.double() * m.m2_scale.double()


def tolerance(case):
    """About four times the distance seen between a pass and exact(), which is what the roundings of the output type and of
    the 16-bit accumulator the deployed Linear keeps amount to."""
    kind, dtype = case["kind"], case.get("dtype", "bf16")
    if kind == "chunk":
        return "exact"
    if kind == "deploy":
        return {"rel": 1e-2} if dtype == "bf16" else {"rel": 1.2e-3 if case["act"] == "dynamic" else 3.2e-3}
    if kind in ("fp8", "fp8_train"):
        return {"rel": 1e-2} if dtype == "bf16" else {"rel": 1e-6}
    if kind == "pact":
        return {"rel": {"bf16": 3e-2, "fp16": 1.6e-2, "fp32": 2e-4}[dtype]}
    if kind == "qat":
        return {"rel": 5e-3}
    if kind == "bmm":
        return {"rel": 7e-3} if dtype == "bf16" else {"rel": 1.2e-3}
    # two layers of bf16 activations: a different rounding in the first layer moves some int8 codes of the second
    return {"rel": 4e-2, "differ": 0.5}
