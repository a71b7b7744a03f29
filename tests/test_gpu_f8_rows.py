"""Per-token e4m3 quantisation of bf16 rows (packed single-multiply kernel) against the definition in PyTorch on the CPU: codes
and scales bit for bit, over row lengths from one slice to several per thread, with zeros, infinities, NaN, subnormal rows
and the DL8 flush."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


def _want(x, flush):
    bf = torch.bfloat16
    # the row maximum ignores NaN, as the kernel's does
    amax = torch.nan_to_num(x.abs().float(), nan=0.0, posinf=float("inf")).amax(-1, keepdim=True).to(bf)
    s = torch.maximum(amax / 448, torch.tensor(1e-5, dtype=bf))
    q = (x / s).to(torch.float8_e4m3fn)
    if flush:
        q = torch.where(q.float().abs() < 0.0087890625, torch.zeros_like(q.float()), q.float()).to(torch.float8_e4m3fn)
    return q, s.float().reshape(-1)


@pytest.mark.parametrize("rows,cols", [(1, 16), (5, 272), (300, 4096), (3, 4112), (37, 14336), (2, 16400), (2, 24576)])
def test_f8_rows_bf16(cuda_dev, rows, cols):
    g = torch.Generator().manual_seed(cols)
    x = (torch.randn(rows, cols, generator=g) * torch.logspace(-6, 3, rows).view(-1, 1)).bfloat16()
    x[0, :4] = torch.tensor([0.0, -0.0, 1e-38, -1e-38]).bfloat16()
    if rows > 2:
        x[1, 3] = float("nan")
        x[2, 5] = float("inf")
    for flush in (False, True):
        codes, scale, _ = ops.act_quant(x.to(cuda_dev), mode=L.Q_F8_DYN, native_chain=3, dl8_flush=flush)
        want, s = _want(x, flush)
        assert torch.equal(scale.cpu(), s)
        got, want = codes.cpu().view(torch.uint8), want.view(torch.uint8)
        both_nan = ((got & 0x7F) == 0x7F) & ((want & 0x7F) == 0x7F)
        zero = ((got & 0x7F) == 0) & ((want & 0x7F) == 0) & torch.tensor(flush)
        assert bool(((got == want) | both_nan | zero).all()), (flush, (got != want).sum())
