"""The quantiser and its GEMM as one dependent pair of launches against the two separate calls, bit for bit: every GEMM kernel
behind it (few-row with one and several K splits and ragged tiles, single-CTA, CTA-pair, chunked), every kind of quantiser
launch, reduction lengths that need padding, repeated calls that reuse buffers, and replay from a CUDA graph."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


def _both(x, w, quant, mul):
    codes, scale, _ = ops.act_quant(x, **quant)
    rs = mul.pop("row_scale", None)
    want = ops.gemm(codes, w, row_scale=scale if rs is None else rs, **mul)
    got = ops.quant_gemm(x, w, row_scale=rs, **quant, **mul)
    return got, want


@pytest.mark.parametrize("M", [1, 2, 31, 33, 128, 129, 200, 256, 517])
@pytest.mark.parametrize("K,N", [(4096, 1000), (512, 136), (2048, 4112), (1000, 72), (14336, 512), (128, 30016)])
def test_pair_of_launches(cuda_dev, M, K, N):
    g = torch.Generator().manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g).bfloat16().to(cuda_dev)
    w8 = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8).to(cuda_dev)
    cs, bias = (torch.rand(N, generator=g) * 0.01).to(cuda_dev), torch.randn(N, generator=g).to(cuda_dev)
    prod = dict(epilogue=L.EPI_SCALE_PROD, scale_round=torch.float16, acc_round=torch.float16, col_scale=cs, bias=bias, out_dtype=torch.bfloat16)
    got, want = _both(x, w8, dict(mode=L.Q_I8_DYN, native_chain=7), dict(prod))
    assert torch.equal(got, want)
    static = dict(mode=L.Q_I8_STATIC, scale0=torch.tensor([0.05], device=cuda_dev), zp0=torch.tensor([117], device=cuda_dev, dtype=torch.int32), shift=128.0)
    got, want = _both(x.float(), w8, static, dict(prod, row_scale=static["scale0"], out_dtype=torch.float32))
    assert torch.equal(got, want)
    wf = torch.randn(N, K, generator=g).to(torch.float8_e4m3fn).to(cuda_dev)
    seq = dict(epilogue=L.EPI_SCALE_SEQ, col_scale=cs, mid_round=torch.bfloat16, acc_round=torch.bfloat16, out_dtype=torch.bfloat16)
    got, want = _both(x, wf, dict(mode=L.Q_F8_DYN, native_chain=3), seq)
    assert torch.equal(got, want)
    if K % 128 == 0 and N < 5000:
        got, want = _both(x, w8, dict(mode=L.Q_I8_DYN, native_chain=7), dict(prod, chunk_k=64, trun_bits=8))
        assert torch.equal(got, want)
    ops.check_status(cuda_dev)


@pytest.mark.parametrize("M,K,N", [(1, 4096, 14336), (37, 14336, 4096), (300, 4096, 1024)])
def test_back_to_back_and_in_a_graph(cuda_dev, M, K, N):
    g = torch.Generator().manual_seed(3)
    ws = [torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8).to(cuda_dev) for _ in range(2)]
    xs = [torch.randn(M, K, generator=g).bfloat16().to(cuda_dev) for _ in range(4)]
    cs = (torch.rand(N, generator=g) * 0.01).to(cuda_dev)
    kw = dict(mode=L.Q_I8_DYN, native_chain=7, epilogue=L.EPI_SCALE_PROD, scale_round=torch.float16, acc_round=torch.float16, col_scale=cs, out_dtype=torch.bfloat16)

    def call(i):
        return ops.quant_gemm(xs[i % 4], ws[i % 2], **kw)

    want = []
    for i in range(4):
        codes, scale, _ = ops.act_quant(xs[i], mode=L.Q_I8_DYN, native_chain=7)
        want.append(ops.gemm(codes, ws[i % 2], epilogue=L.EPI_SCALE_PROD, scale_round=torch.float16, acc_round=torch.float16, row_scale=scale, col_scale=cs,
                             out_dtype=torch.bfloat16))  # fmt: skip
    outs = [call(i) for i in range(64)]
    for i, o in enumerate(outs):
        assert torch.equal(o, want[i % 4]), i
    del outs
    s = torch.cuda.Stream(cuda_dev)
    s.wait_stream(torch.cuda.current_stream(cuda_dev))
    with torch.cuda.stream(s):
        call(0)
    torch.cuda.current_stream(cuda_dev).wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = [call(i) for i in range(8)]
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for i, o in enumerate(held):
        assert torch.equal(o, want[i % 4]), i
    ops.check_status(cuda_dev)
