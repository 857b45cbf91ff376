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


@pytest.mark.parametrize("B,N,K", [(1, 40, 8), (2, 33, 256), (4, 1536, 1536), (9, 65, 2048), (3, 9473, 776)])
def test_skinny_linear_sum_order(sd3, B, N, K):
    """The order of a sum is part of the result (its roundings reach every block through the conditioning
    vector): lane l adds the products of k = 256 i + 8 l + j in the order of i and j, then the 32 lanes are
    added in pairs 16, 8, 4, 2, 1 apart.  Bit for bit; float64 holds product plus sum exactly but for
    pairs more than 2^20 apart."""
    gen = torch.Generator(device="cuda").manual_seed(B + N + K)
    x = torch.randn(B, K, device="cuda", generator=gen)
    w = torch.randn(N, K, device="cuda", generator=gen).bfloat16()
    b = torch.randn(N, device="cuda", generator=gen)
    o = sd3.skinny_linear(x, w, b)
    steps = (K + 255) // 256
    xp = torch.nn.functional.pad(x, (0, 256 * steps - K)).double().view(B, 1, steps, 32, 8)
    wp = torch.nn.functional.pad(w, (0, 256 * steps - K)).double().view(1, N, steps, 32, 8)
    acc = torch.zeros(B, N, 32, device="cuda")
    for i in range(steps):
        for j in range(8):
            acc = (xp[:, :, i, :, j] * wp[:, :, i, :, j] + acc.double()).float()
    lanes = torch.arange(32, device="cuda")
    for d in (16, 8, 4, 2, 1):
        acc = acc + acc[..., lanes ^ d]
    assert torch.equal(o, acc[..., 0] + b)
