"""The fp32 mode's blocks against the oracle in float64, at the sizes where the tensor-core kernels
behind it (fp32 operands as three bf16 planes) can go wrong: partial row and column tiles, every tile
width, ragged and single key tiles, remainders of the 64-wide K blocks, unfused head sizes.

What is compared is what a block adds to its streams (out - in), relative to its norm: the residual would hide
a part of the error.  Tolerance 1e-6.  Below it: a result passes through some ten stages (LayerNorms, four
chained GEMMs, softmax), each of which rounds like a chain of a few fp32 operations, 2^-23; in quadrature 4e-7
(five times less than what the FFMA kernels had).  Above it: a plane product that is missing costs 2^-17 to 2^-18 of every
term.  Emulated with float64 sums of the plane products for these cases, one lost product in every GEMM
gives 3.2e-6 or more here; in a single GEMM or in the attention, 1.2e-6 or more in
test_attention_sublayer_fp32_against_float64, whose scores are larger and whose MLP adds nothing."""
import pytest
import torch

from oracle import mmdit_oracle as O

pytestmark = pytest.mark.gpu

TOLERANCE = 1e-6


def branch_errors(sd3, p, E, NH, x, c, y, dual, last):
    """Relative error of what the block adds to the image and, unless it is discarded, the context stream."""
    p64 = {k: v.double().cuda() for k, v in p.items()}
    c_ref, x_ref = O.dit_block(x.double().cuda(), c.double().cuda(), y.double().cuda(), p64, NH, dual, True, last)
    m = sd3.Model(1, [0] if dual else [], 0, 0, 0, E, NH, 4, 0, 0, 0, True, sd3.PRECISION_F32,
                  last_discards_context=last, block_only=True)
    m.load({k: v.cuda() for k, v in p.items()}, prefix="transformer.0.")
    xx, cc = x.cuda(), c.cuda()
    m.block_forward(0, y.cuda(), cc, xx)
    torch.cuda.synchronize()
    assert sd3.device_status() == 0
    m.close()
    pairs = ((xx, x_ref, x),) + (() if last else ((cc, c_ref, c),))
    return [((got.double() - ref).norm() / (ref - start.double().cuda()).norm()).item() for got, ref, start in pairs]


@pytest.mark.parametrize("E,NH,B,Tx,Tc,dual,last", [
    (64, 1, 1, 1, 1, True, False),         # one token per stream
    (64, 1, 2, 63, 65, True, False),       # samples straddle a row tile
    (128, 2, 3, 128, 1, False, False),     # exact key tile + 1
    (192, 3, 1, 255, 130, True, False),    # ragged last key tile, N not a multiple of 256
    (192, 3, 2, 129, 77, False, True),     # last block: no context output
    (72, 3, 2, 40, 24, True, False),       # head_dim 24: unfused norm, K with a remainder of 8
    (128, 4, 1, 130, 33, True, False),     # head_dim 32
    (1536, 24, 1, 256, 77, True, False),   # 64-wide tiles, K split
    (1536, 24, 1, 1024, 333, True, False),  # 128-wide tiles
    (1536, 24, 4, 1000, 154, False, False),  # several waves of them
    (64, 1, 8, 2040, 20, True, False),     # more tokens than are merged: separate LayerNorms, QKV and attentions
])
def test_block_fp32_against_float64(sd3, E, NH, B, Tx, Tc, dual, last):
    gen = torch.Generator().manual_seed(E + 7 * Tx + Tc)
    p = O.random_params(O.block_param_shapes(E, 4, E // NH, dual, last, True), seed=Tx, std=0.02 * (1536 / E) ** 0.5,
                        bias_std=0.02, norm_std=0.3)
    x, c = torch.randn(B, Tx, E, generator=gen), torch.randn(B, Tc, E, generator=gen)
    y = torch.nn.functional.silu(torch.randn(B, E, generator=gen))
    assert max(branch_errors(sd3, p, E, NH, x, c, y, dual, last)) < TOLERANCE


@pytest.mark.parametrize("E,NH,B,Tx,Tc", [
    (64, 1, 1, 1, 1), (64, 1, 2, 63, 65), (128, 2, 3, 128, 1), (192, 3, 1, 255, 130), (256, 4, 1, 600, 77),
    (1536, 24, 1, 256, 77)])
def test_attention_sublayer_fp32_against_float64(sd3, E, NH, B, Tx, Tc):
    """QKV, both attentions and the out-projections of a dual block alone: the MLPs' second weights are zero, the
    scores have a standard deviation of about 4."""
    gen = torch.Generator().manual_seed(E + 7 * Tx + Tc)
    p = O.random_params(O.block_param_shapes(E, 4, E // NH, True, False, True), seed=Tx, std=E ** -0.5, bias_std=0.02,
                        norm_std=0.3)
    p = {k: v * (2.0 if "rmsnorm" in k else 0.0 if "lin2" in k else 1.0) for k, v in p.items()}
    x, c = torch.randn(B, Tx, E, generator=gen), torch.randn(B, Tc, E, generator=gen)
    y = torch.nn.functional.silu(torch.randn(B, E, generator=gen))
    assert max(branch_errors(sd3, p, E, NH, x, c, y, True, False)) < TOLERANCE


@pytest.mark.parametrize("what", ["activation", "weight", "infinite activation"])
def test_values_above_bf16_range(sd3, what):
    """The end of float32's range lies above bf16's (3.4028e38, 3.3895e38): such an operand of the second MLP linear
    counts with its value, and an infinite one makes its row infinite with the signs of its weights."""
    E, big = 64, 3.4e38
    gen = torch.Generator().manual_seed(5)
    p = O.random_params(O.block_param_shapes(E, 4, E, False, False, True), seed=5, std=0.1, bias_std=0.02, norm_std=0.3)
    x, c = torch.randn(2, 65, E, generator=gen), torch.randn(2, 20, E, generator=gen)
    y = torch.nn.functional.silu(torch.randn(2, E, generator=gen))
    w1, b1, w2 = (p["latent_mlp." + k] for k in ("lin1.weight", "lin1.bias", "lin2.weight"))
    w1[:, 0] = 0.0  # hidden channel 0 is gelu(b1[0])
    b1[0] = {"activation": big, "weight": 1e-30, "infinite activation": float("inf")}[what]
    if what == "activation":
        w2[0] = 1e-30 * torch.randn(E, generator=gen)
    if what == "weight":
        w2[0] = big
    if what != "infinite activation":
        assert max(branch_errors(sd3, p, E, 1, x, c, y, False, False)) < TOLERANCE
        return
    m = sd3.Model(1, [], 0, 0, 0, E, 1, 4, 0, 0, 0, True, sd3.PRECISION_F32, last_discards_context=False,
                  block_only=True)
    m.load({k: v.cuda() for k, v in p.items()}, prefix="transformer.0.")
    xx, cc = x.cuda(), c.cuda()
    m.block_forward(0, y.cuda(), cc, xx)
    torch.cuda.synchronize()
    m.close()
    ref = O.dit_block(x.double(), c.double(), y.double(), {k: v.double() for k, v in p.items()}, 1, False, True, False)
    assert ref[1].isinf().all() and torch.equal(xx.cpu().double(), ref[1])
    assert cc.isfinite().all()


def test_captions_at_any_address(sd3):
    """Captions that start in the middle of a vector load give the bits of aligned ones (fp32 and bf16 tensors)."""
    L, E, NH, P, C = 2, 64, 1, 64, 128
    p = O.random_params(O.model_param_shapes(L, (0,), 16, E, P, C, 2, NH, 4), seed=1, std=0.1)
    m = sd3.Model(L, (0,), P, C, 16, E, NH, 4, 2, 32, 16, True, sd3.PRECISION_F32)
    m.load({k: v.cuda() for k, v in p.items()})
    gen = torch.Generator().manual_seed(2)
    for dtype in (torch.float32, torch.bfloat16):
        pooled, caps = torch.randn(1, P, generator=gen).to(dtype).cuda(), torch.randn(1, 9, C, generator=gen).to(dtype).cuda()
        lat, t = torch.randn(1, 16, 8, 8, generator=gen).to(dtype).cuda(), torch.tensor([500.0]).cuda()
        odd = torch.empty(caps.numel() + 1, device="cuda", dtype=dtype)[1:].view_as(caps)
        odd.copy_(caps)
        assert odd.data_ptr() % 8 and odd.is_contiguous()
        assert torch.equal(m.forward(pooled, caps, lat, t), m.forward(pooled, odd, lat, t))
    torch.cuda.synchronize()
    assert sd3.device_status() == 0
    m.close()
