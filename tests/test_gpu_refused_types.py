"""Activations of a type that the row quantizers do not take are refused by the deployed Linear with a RuntimeError."""

import pytest
import torch

from fms_model_optimizer_b200.modules import QLinear, QLinearINT8Deploy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.int32])
@pytest.mark.parametrize("dynamic", [True, False])
def test_types_that_are_refused(cuda_dev, dtype, dynamic):
    lin = QLinear(64, 48, num_bits_feature=8, qa_mode="pertokenmax" if dynamic else "pact+", num_bits_weight=8, qw_mode="maxperCh", device=cuda_dev)
    lin(torch.zeros(1, 64, device=cuda_dev))
    mod = QLinearINT8Deploy.from_fms_mo(lin.eval(), use_dynamic_max_act_Qfunc=-1 if dynamic else False, use_PT_native_Qfunc=not dynamic)
    with pytest.raises(RuntimeError, match="dtype"):
        mod(torch.ones(3, 64, device=cuda_dev).to(dtype))
    assert mod(torch.ones(3, 64, device=cuda_dev)).shape == (3, 48)
