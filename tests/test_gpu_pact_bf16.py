"""The packed bf16 PACT+ kernels against the element-by-element functions (which a tensor that starts off a 16-byte boundary
still takes): outputs and input gradients bit for bit over every bf16 number, NaN, infinities and subnormal numbers included,
for all three quantisers, several widths and clip values (one of them with a step that takes the ordinary division).

Clip gradients: both sides add the same terms, each at most |g|, in fp32 in another order; either sum of n terms is within
n * 2^-24 * sum |g| of the exact one, so they differ by at most twice that, which is asserted."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


def _shifted(t):
    """The same values starting 2 bytes off a 16-byte boundary."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    out = buf[1 : 1 + t.numel()]
    out.copy_(t)
    assert out.data_ptr() % 16 != 0
    return out


@pytest.mark.parametrize("variant", [L.PACT_TWO_SIDED, L.PACT_ONE_SIDED, L.PACT_SYMMETRIC])
@pytest.mark.parametrize("bits", [2, 4, 7, 8, 10])
@pytest.mark.parametrize("clips", [(3.0, -2.5), (6.0, -6.0), (0.7, 0.1), (1e-17, -1e-17), (2.0, 2.0)])
def test_every_bf16_number(cuda_dev, variant, bits, clips):
    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    g = torch.randn(65536, generator=torch.Generator().manual_seed(bits)).bfloat16()
    x, g = x.to(cuda_dev), g.to(cuda_dev)
    cv, cvn = (torch.tensor([c], device=cuda_dev) for c in clips)
    for align in (True, False):
        want = ops.pact2_fwd(_shifted(x), cv, cvn, bits, align, variant)
        got = ops.pact2_fwd(x, cv, cvn, bits, align, variant)
        same = (got.view(torch.int16) == want.view(torch.int16)) | (torch.isnan(got) & torch.isnan(want))
        assert bool(same.all()), x[~same][:8]
        finite = ~torch.isnan(x)
        xf, gf = x[finite], g[finite]
        wx, wc = ops.pact2_bwd(_shifted(xf), _shifted(gf), cv, cvn, bits, align, variant)
        gx, gc = ops.pact2_bwd(xf, gf, cv, cvn, bits, align, variant)
        same = gx.view(torch.int16) == wx.view(torch.int16)
        assert bool(same.all()), xf[~same][:8]
        n = 2 if variant == L.PACT_TWO_SIDED else 1
        bound = 2 * 65536 * 2.0**-24 * gf.float().abs().sum()
        ok = ((gc[:n] - wc[:n]).abs() <= bound) | (torch.isnan(gc[:n]) & torch.isnan(wc[:n]))
        assert bool(ok.all()), (gc, wc)
        wx, _ = ops.pact2_bwd(_shifted(x), _shifted(g), cv, cvn, bits, align, variant)
        gx, _ = ops.pact2_bwd(x, g, cv, cvn, bits, align, variant)
        assert torch.equal(gx.view(torch.int16), wx.view(torch.int16))
