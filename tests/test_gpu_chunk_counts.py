"""Chunk-truncating int8 GEMM with the low byte rounded away, even and odd chunks and the total issued by three warps.
Against the definition on the CPU, for chunk counts from one to 520, odd counts, several tiles per block and ragged edges;
results are whole numbers and must be equal."""

import pytest
import torch

from fms_model_optimizer_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N", [(1, 128, 16), (130, 256, 136), (200, 384, 264), (129, 640, 144), (64, 16384, 48), (64, 16640, 48), (2600, 384, 2080)])
@pytest.mark.parametrize("chunk", [32, 64, 128])
def test_low_byte_chunks(cuda_dev, M, K, N, chunk):
    g = torch.Generator().manual_seed(K + chunk)
    a = torch.randint(-128, 128, (M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-128, 128, (N, K), generator=g, dtype=torch.int8)
    want = torch.zeros(M, N, dtype=torch.int64)
    for k in range(0, K, chunk):  # |sum| <= 128 * 2^14: exact in fp32
        part = (a[:, k : k + chunk].float() @ b[:, k : k + chunk].float().t()).to(torch.int64)
        want += ((part + 128) >> 8) << 8
    got = ops.gemm(a.to(cuda_dev), b.to(cuda_dev), chunk_k=chunk, trun_bits=8)
    assert torch.equal(got.cpu().to(torch.int64), want)
