"""Sizes at the edges of the GEMM dispatch: few rows, short K."""
import pytest
import torch

from prime_b200.ops import kernels as ops

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


# 256 rows or columns, K that the slices do not divide, N that is no multiple of the tile
@pytest.mark.parametrize("M,N,K,res", [(256, 256, 8192, True), (256, 704, 4099, False), (1024, 260, 2304, True), (300, 1024, 2048, False)])
def test_split_k_of_narrow_products(M, N, K, res):
    torch.manual_seed(0)
    a = torch.randn(K, (M + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :M]      # row pitch of whole 16-byte units
    b = torch.randn(K, (N + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :N]
    assert ops._splitk_slices(M, N, K, a.device) > 1
    ref = a.float().t() @ b.float()
    for dt in (torch.bfloat16, torch.float32):
        ld = (N + 7) // 8 * 8
        r = torch.randn(M, ld, device="cuda", dtype=dt)[:, :N] if res else None
        out = torch.empty(M, ld, device="cuda", dtype=dt)[:, :N]
        ops.gemm(a, b, out=out, residual=r, a_mn=True, b_mn=True)
        ops.check_status()
        assert _rel(out, ref + (r.float() if res else 0)) < (1e-2 if dt == torch.bfloat16 else 1e-3)
