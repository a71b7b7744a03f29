"""Per-tensor FP8 quantisation with transposed codes and column sums against the row quantiser's per-tensor mode (the general
kernel) and PyTorch: same codes and scale for every data type, format and ragged size, the transposed codes are the codes
turned (padding included), the column sums agree with 64-bit sums to fp32 accuracy."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


def _general(x, e5m2, eps, flush):
    amax = ops.tensor_absmax(x)
    native = 0 if x.dtype == torch.float32 else 3
    codes, scale, _ = ops.act_quant(x, mode=L.Q_F8_TENSOR, native_chain=native, scale_in=amax, scale0=(57344.0 if e5m2 else 448.0), dyn_eps=eps,
                                    f8_e5m2=e5m2, dl8_flush=flush)  # fmt: skip
    return codes, scale[:1]


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 17), (128, 64), (129, 80), (517, 1000), (1000, 4096)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("kind", ["normal", "tiny", "zero", "inf", "nan"])
def test_per_tensor_codes(cuda_dev, rows, cols, dtype, kind):
    g = torch.Generator().manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=g)
    if kind == "tiny":
        x *= 1e-6 if dtype == torch.float16 else 1e-22
    if kind == "zero":
        x *= 0
    x = x.to(dtype)
    if kind in ("inf", "nan"):
        x.view(-1)[rows * cols // 2] = float(kind)
    x = x.to(cuda_dev)
    parts = ops.absmax_parts(x)
    for e5m2, eps in ((False, 1e-5), (True, 0.0)):
        for flush in (False, True):
            want, ws = _general(x, e5m2, eps, flush)
            codes, codes_t, scale, colsum = ops.fp8_quant_tensor(x, parts, e5m2=e5m2, eps=eps, dl8_flush=flush, want_t=True, want_colsum=e5m2)
            assert torch.equal(scale, ws) or (torch.isnan(scale).all() and torch.isnan(ws).all())
            u, w = codes.view(torch.uint8), want.view(torch.uint8)
            # a flushed negative value and a NaN may carry either sign
            same = (u == w) | (((u | w) & 0x7F) == 0) & torch.tensor(flush, device=cuda_dev)
            assert bool(same.all()), (e5m2, flush, int((~same).sum()))
            assert torch.equal(codes_t.view(torch.uint8), u.t())
            one, _, _, _ = ops.fp8_quant_tensor(x, parts, e5m2=e5m2, eps=eps, dl8_flush=flush)
            assert torch.equal(one.view(torch.uint8), u)
            if e5m2:
                ref = codes.double().sum(0)
                bound = 2e-6 * codes.double().abs().sum(0) + 1e-30  # 128-row tiles, then tiles in order: far below rows * 2^-24
                ok = (colsum.double() - ref).abs() <= bound
                assert bool((ok | ~torch.isfinite(ref)).all())
    ops.check_status(cuda_dev)


@pytest.mark.parametrize("rows,cols,pitch", [(2085, 3000, 3000), (2560, 2048, 2048), (130, 64 * 620 + 16, 64 * 620 + 19)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
def test_blocks_that_walk_over_tiles(cuda_dev, rows, cols, pitch, dtype):
    """More tiles than resident blocks: the next tile is loaded while this one is written; ragged edges, rows off 16 bytes."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, pitch, generator=g, device="cuda").to(dtype)[:, :cols]
    parts = ops.absmax_parts(x.contiguous())
    for e5m2, eps in ((False, 1e-5), (True, 0.0)):
        want, ws = _general(x.contiguous(), e5m2, eps, False)
        codes, codes_t, scale, _ = ops.fp8_quant_tensor(x, parts, e5m2=e5m2, eps=eps, want_t=True, want_colsum=e5m2)
        assert torch.equal(scale, ws) and torch.equal(codes.view(torch.uint8), want.view(torch.uint8))
        assert torch.equal(codes_t.view(torch.uint8), codes.view(torch.uint8).t())
