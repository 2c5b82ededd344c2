"""Weight-gradient products (A^T B over T*B rows) whose row count is no multiple of 8: the tensor-core
kernels zero-fill the tail; against fp32 matmuls, one bf16 rounding of an fp32 sum."""
import pytest
import torch

from elman_b200 import _lib
from elman_b200 import hasty_pytorch_lib as H
from oracle.elman_oracle import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 128, 1), (256, 512, 63), (304, 136, 65), (512, 512, 4332),
                                   (1280, 1280, 1089)])
def test_transposed_product_with_a_ragged_row_count(M, N, K):
    g = torch.Generator().manual_seed(M + K)
    A = torch.randn(K, M, generator=g).bfloat16().cuda()
    B = (torch.randn(K, N, generator=g) / K ** 0.5).bfloat16().cuda()
    before = _lib.tc_launch_count()
    out = H.gemm(H.GEMM_TN, A, B)
    torch.cuda.synchronize()
    assert _lib.tc_launch_count() > before and _lib.device_status()[0] == 0
    assert rel_err(out, A.float().cpu().T @ B.float().cpu()) < 4e-3
