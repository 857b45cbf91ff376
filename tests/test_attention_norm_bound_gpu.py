"""Blocks whose norm weights give no usable bound on the scores: the attention compares |q| |k| of every 32 query rows
with its limit and runs those rows with or without a running maximum."""
import pytest
import torch

from oracle import mmdit_oracle as O

pytestmark = pytest.mark.gpu


# The weights alone give gain^2 11.7 = 187 and 494, the limit is 80; by the norms all rows are below it at gain 4, some
# at 6.5.  Ragged tokens, context rows in the one-CTA kernel, a key split (few heads, long), merged and separate attentions.
@pytest.mark.parametrize("B,Tx,Tc,NH,gain,dual", [(1, 300, 20, 8, 4.0, True), (2, 1000, 333, 8, 6.5, True),
                                                  (8, 2028, 60, 4, 6.5, True), (1, 2500, 20, 4, 6.5, False)])
def test_block_matches_oracle(sd3, B, Tx, Tc, NH, gain, dual):
    E = 64 * NH
    gen = torch.Generator().manual_seed(3)
    p = O.random_params(O.block_param_shapes(E, 4, 64, dual, False, True), seed=3, std=E ** -0.5, dtype=torch.bfloat16,
                        norm_std=0.1)
    for k in p:
        if "rmsnorm" in k:  # one dimension carries most of a norm: rows differ by how much of it they have
            w = torch.full((64,), 0.5)
            w[7] = gain
            p[k] = (w * torch.exp(0.1 * torch.randn(64, generator=gen))).to(torch.bfloat16)
    m = sd3.Model(1, [0] if dual else [], 0, 0, 0, E, NH, 4, 0, 0, 0, True, sd3.PRECISION_BF16,
                  last_discards_context=False, block_only=True)
    m.load({k: v.cuda() for k, v in p.items()}, prefix="transformer.0.")
    x, c = torch.randn(B, Tx, E, generator=gen), torch.randn(B, Tc, E, generator=gen)
    y = torch.nn.functional.silu(torch.randn(B, E, generator=gen))
    cc, xx = c.cuda(), x.cuda()
    m.block_forward(0, y.cuda(), cc, xx)
    torch.cuda.synchronize()
    assert sd3.device_status() == 0
    m.close()
    p32 = {k: v.float().cuda() for k, v in p.items()}
    rc, rx = O.dit_block(x.cuda(), c.cuda(), y.cuda(), p32, NH, dual, True, False)[:2]
    # What the block adds.  q and k are bf16: a score of S (in powers of two, about 10 for the rows' largest at gain 6.5)
    # is off by about 2^-9 S, its weight by 0.69 times that, 1.4 %; the other operands give 5e-3.
    assert ((xx - rx).norm() / (rx - x.cuda()).norm()).item() < 2e-2
    assert ((cc - rc).norm() / (rc - c.cuda()).norm()).item() < 2e-2
