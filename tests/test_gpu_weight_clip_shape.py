"""The clip values that the per-channel weight quantizer returns: one per row, in one dimension, whatever shape they were given in."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(24,), (24, 1), (4, 6), (1, 24, 1)])
def test_given_clip_values(cuda_dev, dtype, shape):
    w = torch.randn(24, 48, generator=torch.Generator().manual_seed(0)).to(cuda_dev)
    clip = (torch.rand(24, generator=torch.Generator().manual_seed(1)) + 0.5).to(dtype).to(cuda_dev)
    want = ops.weight_fq_perch(w, num_bits=8, mode=L.W_GIVEN, clip=clip)
    given = clip.view(shape)
    got = ops.weight_fq_perch(w, num_bits=8, mode=L.W_GIVEN, clip=given)
    assert got[2].shape == (24,) and torch.equal(got[2], clip.float()) and torch.equal(got[0], want[0])
    assert got[2].data_ptr() != given.data_ptr()
