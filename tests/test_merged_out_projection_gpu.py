"""A dual block's two out-projections into the image stream share a launch up to 16384 tokens; the joint attention's
part is added first, so a sample's result is the same bits as from separate launches (a batch above the line)."""
import pytest
import torch

from oracle import mmdit_oracle as O

pytestmark = pytest.mark.gpu


# one tile of image rows beside a context that the one-CTA kernel takes; ragged tiles of both
@pytest.mark.parametrize("Tx,Tc,precision", [(256, 20, "BF16"), (700, 300, "BF16"), (700, 300, "FP8")])
def test_one_sample_and_a_batch_above_the_line_agree(sd3, Tx, Tc, precision):
    E, NH = 512, 8
    B = 16384 // (Tx + Tc) + 1
    gen = torch.Generator().manual_seed(12)
    p = O.random_params(O.block_param_shapes(E, 4, 64, True, False, True), seed=12, std=E ** -0.5, dtype=torch.bfloat16,
                        norm_std=0.1)
    m = sd3.Model(1, [0], 0, 0, 0, E, NH, 4, 0, 0, 0, True, getattr(sd3, "PRECISION_" + precision),
                  last_discards_context=False, block_only=True)
    m.load({k: v.cuda() for k, v in p.items()}, prefix="transformer.0.")
    x, c = torch.randn(B, Tx, E, generator=gen).cuda(), torch.randn(B, Tc, E, generator=gen).cuda()
    y = torch.nn.functional.silu(torch.randn(B, E, generator=gen)).cuda()
    cc, xx = c.clone(), x.clone()
    m.block_forward(0, y, cc, xx)
    for n in (1, 1, 3):  # again on the same words, then with others
        c1, x1 = c[:n].clone(), x[:n].clone()
        m.block_forward(0, y[:n].contiguous(), c1, x1)
        assert torch.equal(x1, xx[:n])
        assert torch.equal(c1, cc[:n]) or n * Tc < 256  # the one-CTA kernel adds the residual in one rounding less
    assert sd3.device_status() == 0 and not torch.equal(xx, x)
    m.close()
