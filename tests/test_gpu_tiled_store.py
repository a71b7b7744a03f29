"""GEMM outputs stored by TMA: several tiles a CTA, so that a warp's two pieces of staging memory are used over and over, with
right edges and last rows that leave pieces partly or wholly outside the output.  int8 sums are exact, so every bit is compared."""

import pytest
import torch

from fms_model_optimizer_b200 import _lib as L
from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


def _i8(g, *shape):
    return torch.randint(-127, 128, shape, generator=g, dtype=torch.int8, device="cuda")


@pytest.mark.parametrize("M,N", [(5000, 2088), (20001, 1048), (200, 40000), (4096, 1028)])
def test_many_tiles_with_ragged_edges(cuda_dev, M, N):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = _i8(g, M, 96), _i8(g, N, 96)
    acc = (a.double() @ b.double().t()).int()
    rs = torch.rand(M, generator=g, device="cuda") * 0.01 + 0.001
    cs = torch.rand(N, generator=g, device="cuda") * 0.01 + 0.001
    assert torch.equal(ops.gemm(a, b), acc)
    want = acc.float() * (rs[:, None] * cs).bfloat16().half().float()
    for acc_round, out, w in ((torch.float16, torch.bfloat16, want.half().bfloat16()), (None, torch.float32, want)):
        got = ops.gemm(a, b, epilogue=L.EPI_SCALE_PROD, row_scale=rs, col_scale=cs, prod_round=torch.bfloat16, scale_round=torch.float16,
                       acc_round=acc_round, out_dtype=out)  # fmt: skip
        assert torch.equal(got, w), out
    ops.check_status(cuda_dev)


@pytest.mark.parametrize("B,M,N", [(40, 300, 264), (150, 33, 520), (7, 700, 1032)])
def test_many_batched_tiles_with_ragged_edges(cuda_dev, B, M, N):
    g = torch.Generator(device="cuda").manual_seed(B + M)
    a, b = _i8(g, B, M, 64), _i8(g, B, N, 64)
    acc = torch.matmul(a.double(), b.double().transpose(1, 2)).int()
    assert torch.equal(ops.bmm_i8(a, b), acc)
    s1, s2 = torch.tensor([0.0137], device="cuda"), torch.tensor([0.071], device="cuda")
    for dt in (torch.float32, torch.float16, torch.bfloat16):
        assert torch.equal(ops.bmm_i8(a, b, (s1, s2), dt), (acc.half() * s1 * s2).to(dt)), dt
    ops.check_status(cuda_dev)


@pytest.mark.parametrize("B,M,K,N", [(5, 260, 384, 264), (5, 260, 400, 264), (148, 200, 512, 72), (149, 200, 512, 72), (9, 130, 512, 136), (3, 300, 2064, 64)])
def test_batched_products_on_both_sides_of_the_short_rule(cuda_dev, B, M, K, N):
    g = torch.Generator(device="cuda").manual_seed(B + M + K)
    a, b = _i8(g, B, M, K), _i8(g, B, N, K)
    acc = torch.matmul(a.double(), b.double().transpose(1, 2)).int()
    assert torch.equal(ops.bmm_i8(a, b), acc)
    s1, s2 = torch.tensor([0.0137], device="cuda"), torch.tensor([0.071], device="cuda")
    small = a // 16  # sums that fp16 holds
    want = torch.matmul(small.double(), b.double().transpose(1, 2)).half().float() * s1 * s2
    assert torch.equal(ops.bmm_i8(small, b, (s1, s2), torch.bfloat16), want.bfloat16())
    ops.check_status(cuda_dev)
