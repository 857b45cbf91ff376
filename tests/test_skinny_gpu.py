"""The skinny (M = batch) linear at the edges of its tiling: every batch variant and a second pass over
the samples, row groups that are not full, both row counts per warp, K chunks with a remainder.

Tolerance: a lane adds K / 32 products in sequence and a five-step tree follows, so the error of a
sum is at most (K / 32 + 6) * 2^-24 times the sum of the products' absolute values."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,K", [(1, 7, 8), (3, 8, 392), (4, 9, 776), (5, 33, 1536), (9, 1537, 2048), (17, 40, 384),
                                   (1, 9472, 1536), (2, 9503, 768), (4, 12001, 1544), (7, 9473, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_skinny_linear_edges(sd3, B, N, K, dtype):
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(B, K, device="cuda", generator=gen)
    w = torch.randn(N, K, device="cuda", generator=gen).to(dtype)
    b = torch.randn(N, device="cuda", generator=gen)
    o = sd3.skinny_linear(x, w, b)
    torch.cuda.synchronize()
    assert sd3.device_status() == 0
    x64, w64 = x.double(), w.double()
    bound = (x64.abs() @ w64.abs().t() + b.abs()) * (K / 32 + 6) * 2.0 ** -24
    assert ((o.double() - (x64 @ w64.t() + b)).abs() <= bound).all()
