"""The flat kernel of the static quantisers against the row-wise kernels (which a tensor with a row pitch still takes), over
every static mode, data type, rounding chain and ragged size, with infinities, NaN, zeros and ties among the values; and
scalars read from device memory against the same scalars as launch arguments."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu

MODES = {
    L.Q_I8_STATIC: dict(zp0=117.0, shift=128.0, add2=1.0),
    L.Q_I8_STATIC_CLAMP_FIRST: dict(zp0=-113.0, lo=-5.5, hi=6.25, shift=128.0),
    L.Q_I8_STATIC_ROUND_FIRST: dict(zp0=115.0, lo=0.0, hi=255.0, shift=128.0),
    L.Q_I8_AFFINE_RCP: dict(zp0=3.0),
}


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 17), (64, 128), (5, 1000), (700, 768), (2, 4099)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_flat_kernel_equals_row_kernels(cuda_dev, rows, cols, dtype):
    g = torch.Generator().manual_seed(rows * cols)
    x = torch.randn(rows, cols, generator=g) * 4
    flat = x.view(-1)
    special = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), 3e38, -3e38, 1e-30, 0.0235, 0.0705])
    n = min(flat.numel(), len(special))
    flat[:n] = special[:n]
    x = x.to(dtype).to(cuda_dev)
    pitched = torch.zeros(rows, cols + 24, dtype=dtype, device=cuda_dev)[:, 8 : 8 + cols]
    pitched.copy_(x)
    if rows == 1:  # a single row has no pitch: an odd start takes the row kernels
        pitched = torch.zeros(cols + 1, dtype=dtype, device=cuda_dev)[1:].view(1, cols)
        pitched.copy_(x)
    for mode, kw in MODES.items():
        if mode == L.Q_I8_AFFINE_RCP and dtype != torch.float32:
            continue
        for scale in (0.047, 0.046875, 1.9999999, 3e-20):  # the last two take the ordinary division
            for native in (0, 3) if dtype != torch.float32 else (0,):
                got, sc, _ = ops.act_quant(x, mode=mode, native_chain=native, scale0=scale, **kw)
                want, sc2, _ = ops.act_quant(pitched, mode=mode, native_chain=native, scale0=scale, **kw)
                assert torch.equal(got, want), (mode, scale, native)
                assert torch.equal(sc, sc2) and sc.shape == (rows,)
                dev = {k: torch.tensor([v], device=cuda_dev) for k, v in kw.items() if k in ("zp0", "lo", "hi")}
                if "zp0" in dev:
                    dev["zp0"] = dev["zp0"].to(torch.int32)
                s_t = torch.tensor([scale], device=cuda_dev)
                for src in (x, pitched):
                    got, sc, _ = ops.act_quant(src, mode=mode, native_chain=native, scale0=s_t, **{**kw, **dev})
                    assert torch.equal(got, want) and torch.equal(sc, sc2), (mode, scale, native)
    ops.check_status(cuda_dev)
