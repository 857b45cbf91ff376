"""A dual block launches its LayerNorms, QKV projections and attentions together up to 16384 tokens and one by
one above; a sample's result is the same bits on either side."""
import pytest
import torch

from oracle import mmdit_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["BF16", "FP8", "F32"])
def test_same_bits_on_both_sides_of_the_line(sd3, precision):
    # eight heads: 1024 CTAs per attention, 3.5 waves each, 6.9 together, so the attentions are merged as well
    E, NH, Tx, Tc = 512, 8, 2028, 20
    gen = torch.Generator().manual_seed(11)
    dtype = torch.float32 if precision == "F32" else torch.bfloat16
    p = O.random_params(O.block_param_shapes(E, 4, 64, True, False, True), seed=11, std=E ** -0.5, dtype=dtype, norm_std=0.1)
    m = sd3.Model(1, [0], 0, 0, 0, E, NH, 4, 0, 0, 0, True, getattr(sd3, "PRECISION_" + precision),
                  last_discards_context=False, block_only=True)
    m.load({k: v.cuda() for k, v in p.items()}, prefix="transformer.0.")
    x, c = torch.randn(9, Tx, E, generator=gen), torch.randn(9, Tc, E, generator=gen)
    y = torch.nn.functional.silu(torch.randn(9, E, generator=gen)).cuda()
    out = {}
    for B in (8, 9):  # 16384 and 18432 tokens
        cc, xx = c[:B].cuda(), x[:B].cuda()
        m.block_forward(0, y[:B].contiguous(), cc, xx)
        out[B] = (cc, xx)
    torch.cuda.synchronize()
    assert sd3.device_status() == 0
    m.close()
    for a, b, start in zip(out[8], out[9], (c, x)):
        assert torch.equal(a, b[:8]) and a.isfinite().all() and not torch.equal(a.cpu(), start[:8])
