"""The CTA pair that runs a tile of a dual block's joint out-projection runs the image-only one's tile of the same rows
next.  Several such tiles per pair, and launches without the context rows' problem: the bits of separate launches
(a batch above 16384 tokens)."""
import pytest
import torch

from oracle import mmdit_oracle as O

pytestmark = pytest.mark.gpu


# 64, 128 and 256 tiles of 128 or 256 columns for 74 pairs; fewer than 256 context rows run in the one-CTA kernel
@pytest.mark.parametrize("Tx,Tc,precision", [(4000, 333, "BF16"), (4000, 20, "BF16"), (4000, 333, "FP8")])
def test_samples_below_the_line_agree_with_a_batch_above_it(sd3, Tx, Tc, precision):
    E, NH, B = 512, 8, 5
    gen = torch.Generator().manual_seed(21)
    p = O.random_params(O.block_param_shapes(E, 4, 64, True, False, True), seed=21, std=E ** -0.5, dtype=torch.bfloat16,
                        norm_std=0.1)
    m = sd3.Model(1, [0], 0, 0, 0, E, NH, 4, 0, 0, 0, True, getattr(sd3, "PRECISION_" + precision),
                  last_discards_context=False, block_only=True)
    m.load({k: v.cuda() for k, v in p.items()}, prefix="transformer.0.")
    x, c = torch.randn(B, Tx, E, generator=gen).cuda(), torch.randn(B, Tc, E, generator=gen).cuda()
    y = torch.nn.functional.silu(torch.randn(B, E, generator=gen)).cuda()
    assert B * (Tx + Tc) > 16384 >= 3 * (Tx + Tc)
    cc, xx = c.clone(), x.clone()
    m.block_forward(0, y, cc, xx)
    for n in (1, 2, 3, 3):
        c1, x1 = c[:n].clone(), x[:n].clone()
        m.block_forward(0, y[:n].contiguous(), c1, x1)
        assert torch.equal(x1, xx[:n])
        assert torch.equal(c1, cc[:n]) or n * Tc < 256  # the one-CTA kernel adds the residual in one rounding less
    assert sd3.device_status() == 0 and not torch.equal(xx, x)
    m.close()
