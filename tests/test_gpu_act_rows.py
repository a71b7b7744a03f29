"""Dynamic quantisation of many short bf16 rows (four rows at a time) against the definition in PyTorch on the CPU: codes and
scales bit for bit, at row counts on both sides of where that kernel takes over and with a ragged last group."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [-1, 0, 1, 331])
@pytest.mark.parametrize("cols", [16, 272, 1040, 4096])
@pytest.mark.parametrize("mode", ["i8", "i8_smooth", "i8_clamp", "f8"])
def test_many_short_rows(cuda_dev, over, cols, mode):
    rows = 12 * torch.cuda.get_device_properties(cuda_dev).multi_processor_count + over
    g = torch.Generator().manual_seed(cols)
    bf = torch.bfloat16
    x = (torch.randn(rows, cols, generator=g) * torch.logspace(-4, 3, rows)[torch.randperm(rows, generator=g)].view(-1, 1)).to(bf)
    x[3] = 0
    kw, v = {}, x
    if mode == "i8_smooth":
        sm = (torch.rand(cols, generator=g) + 0.5).to(bf)
        v = x / sm
        smd = sm.float().to(cuda_dev)
        kw = dict(smooth=smd, smooth_rcp=ops.smooth_reciprocal(smd))
    if mode == "i8_clamp":
        kw = dict(clamp_codes=True, levels=7)
    amax = v.abs().amax(-1, keepdim=True)
    if mode == "f8":
        s = torch.maximum(amax / 448, torch.tensor(1e-5, dtype=bf))
        want = (v / s).to(torch.float8_e4m3fn).view(torch.uint8)
    else:
        s = torch.maximum(amax, torch.tensor(1e-5, dtype=bf)) / kw.get("levels", 127)
        want = torch.round(v / s)
        if mode == "i8_clamp":
            want = want.clamp(-7, 7)
        want = want.to(torch.int32).to(torch.int8).view(torch.uint8)
    # a view with a pitch, so that a row is not simply the next one's neighbour
    xd = torch.empty(rows, cols + 8, dtype=bf, device=cuda_dev)[:, :cols]
    xd.copy_(x)
    codes, scale, _ = ops.act_quant(xd, mode=L.Q_F8_DYN if mode == "f8" else L.Q_I8_DYN, native_chain=3 if mode == "f8" else 7, **kw)
    assert torch.equal(scale.cpu(), s.float().reshape(-1))
    assert torch.equal(codes.cpu().view(torch.uint8), want)
