"""The GEMM's dequantising epilogues against the same chain in separately rounded PyTorch operations, bit for bit: every
rounding switch, every output type, right edges that end on and off a 16-byte boundary, and row blocks that end inside a
tile (the int32 accumulators are exact, so nothing but the chain can differ)."""

import itertools

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu

F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32


def _r(t, dt):
    return t if dt is None else t.to(dt).float()


def _chain(acc, rs, cs, bias, epi, prod, scale, mid, accr, out):
    a = acc.float()
    if epi == L.EPI_SCALE_PROD:
        y = a * _r(_r(rs * cs, prod), scale)
    else:
        if epi == L.EPI_SCALE_ACC16:
            a = a.half().float()
        y = _r((a * rs) * cs, mid)
    if bias is not None:
        y = y + bias
    return _r(y, accr).to(out)


@pytest.mark.parametrize("M,N", [(300, 512), (300, 264), (129, 257), (200, 36), (257, 1004), (33, 130)])
@pytest.mark.parametrize("out", [F32, F16, BF16])
def test_dequantise_chains(cuda_dev, M, N, out):
    g = torch.Generator().manual_seed(M * 1000 + N)
    K = 96
    a = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)
    acc = (a.double() @ b.double().t()).int()
    rs = torch.rand(M, generator=g) * 0.02 + 0.001
    cs = torch.rand(N, generator=g) * 0.02 + 0.001
    bias = torch.randn(N, generator=g)
    dev = [t.to(cuda_dev) for t in (a, b, rs, cs, bias)]
    chains = [(L.EPI_SCALE_PROD, p, s, None, r) for p, s, r in itertools.product((None, F16, BF16), (None, F16, BF16), (None, F16, BF16))]
    chains += [(e, None, None, m, r) for e, m, r in itertools.product((L.EPI_SCALE_SEQ, L.EPI_SCALE_ACC16), (None, F16, BF16), (None, F16, BF16))]
    for i, (epi, prod, scale, mid, accr) in enumerate(chains):
        with_bias = i % 2 == 0
        want = _chain(acc, rs[:, None], cs[None, :], bias if with_bias else None, epi, prod, scale, mid, accr, out)
        got = ops.gemm(dev[0], dev[1], epilogue=epi, row_scale=dev[2], col_scale=dev[3], bias=dev[4] if with_bias else None, prod_round=prod,
                       scale_round=scale, mid_round=mid, acc_round=accr, out_dtype=out)  # fmt: skip
        assert torch.equal(got.cpu(), want), (epi, prod, scale, mid, accr, with_bias)
    ops.check_status(cuda_dev)


@pytest.mark.parametrize("B,M,K,N", [(5, 77, 48, 93), (3, 130, 64, 258), (7, 33, 16, 4), (2, 128, 128, 512), (9, 1, 32, 1)])
def test_batched_products_of_any_alignment(cuda_dev, B, M, K, N):
    """One launch over all problems whatever the size of a problem's output: raw sums and the fused fp16 scale chain."""
    g = torch.Generator().manual_seed(B * M + N)
    a = torch.randint(-127, 128, (B, M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-127, 128, (B, N, K), generator=g, dtype=torch.int8)
    acc = torch.matmul(a.double(), b.double().transpose(1, 2))
    ad, bd = a.to(cuda_dev), b.to(cuda_dev)
    assert torch.equal(ops.bmm_i8(ad, bd).cpu(), acc.int())
    s1, s2 = torch.tensor([0.0137]), torch.tensor([0.071])
    for dt in (F32, F16, BF16):
        want = (acc.int().to(F16) * s1 * s2).to(dt)
        got = ops.bmm_i8(ad, bd, (s1.to(cuda_dev), s2.to(cuda_dev)), dt)
        assert torch.equal(got.cpu(), want), dt
    ops.check_status(cuda_dev)
