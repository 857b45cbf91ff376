"""The norm weights of a block decide how its attentions run: queries pre-scaled and no running maximum where the
weights bound the scores, unscaled queries and a running maximum for every row where they do not."""
import pytest
import torch

from oracle import mmdit_oracle as O

pytestmark = pytest.mark.gpu


# The weights give gain^2 11.7 = 187 and 494, the limit is 80; the scores themselves stay below it for all rows at gain
# 4, for some at 6.5.  Ragged tokens, context rows in the one-CTA kernel, a key split (few heads, long), merged and separate attentions.
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


# gain 1: 11.7, below the limit.  The block is the same launches as its operations called one by one, so the bits tell
# which of the two ways its attentions ran.
@pytest.mark.parametrize("gain", [1.0, 4.0, 6.5])
@pytest.mark.parametrize("B,Tx,Tc,NH", [(1, 300, 20, 8), (2, 1000, 333, 8), (1, 2500, 20, 4)])
def test_block_gives_the_bits_of_its_operations(sd3, B, Tx, Tc, NH, gain):
    E, T = 64 * NH, Tx + Tc
    gen = torch.Generator().manual_seed(3)
    p = O.random_params(O.block_param_shapes(E, 4, 64, True, False, True), seed=3, std=E ** -0.5, dtype=torch.bfloat16,
                        norm_std=0.1)
    for k in p:
        if "rmsnorm" in k:
            w = torch.full((64,), 0.5)
            w[7] = gain
            p[k] = (w * torch.exp(0.1 * torch.randn(64, generator=gen))).to(torch.bfloat16)
    p = {k: v.cuda() for k, v in p.items()}
    m = sd3.Model(1, [0], 0, 0, 0, E, NH, 4, 0, 0, 0, True, sd3.PRECISION_BF16, last_discards_context=False, block_only=True)
    m.load(p, prefix="transformer.0.")
    x, c = torch.randn(B, Tx, E, generator=gen).cuda(), torch.randn(B, Tc, E, generator=gen).cuda()
    cc, xx = c.clone(), x.clone()
    m.block_forward(0, torch.zeros(B, E, device="cuda"), cc, xx)  # the modulation is the AdaLN bias

    def mod(name):
        return [v.expand(B, E).contiguous() for v in p[name + ".bias"].float().view(-1, E)]

    def lin(name):
        return sd3.pack_weight(p[name + ".weight"]), p[name + ".bias"].float()

    def norm(name):
        return p[name + ".weight"].float()

    def attend(qkv, T, Tc, streams):
        wq, wk = [norm(s + "_rmsnorm_query") for s in streams], [norm(s + "_rmsnorm_key") for s in streams]
        to_log2 = 1.4426950408889634 / 8
        bound = sd3.qk_norm_score_bound(wq, wk) * to_log2
        assert (bound <= 80) == (gain == 1.0)
        for s, (h, tokens, off) in streams.items():
            q = norm(s + "_rmsnorm_query") * (to_log2 if bound <= 80 else 1.0)
            sd3.qkv_project(h, *lin(s + "_to_qkv"), q, norm(s + "_rmsnorm_key"), 1e-6, qkv, B, tokens, T, off, E)
        scratch = sd3.attention_scratch(B, T, NH)
        return (sd3.attention(qkv, B, T, NH, Tc, 0.0, scratch=scratch, score_bound=bound) if bound <= 80 else
                sd3.attention(qkv, B, T, NH, Tc, 0.125, scratch=scratch))

    def mlp(s, r, tokens, shift, scale, gate):
        h = sd3.layernorm_modulate(r, B, tokens, E, 1e-6, shift, scale)[0]
        h = sd3.linear(h, *lin(s + "_mlp.lin1"), act=sd3.ACT_GELU_TANH)
        sd3.linear_gate_residual(h, *lin(s + "_mlp.lin2"), gate, tokens, r)

    cm, xm = mod("context_ada_lnorm.linear"), mod("latent_ada_lnorm.linear")
    h_c = sd3.layernorm_modulate(c, B, Tc, E, 1e-6, cm[0], cm[1])[0]
    h_x, h_x2 = sd3.layernorm_modulate(x, B, Tx, E, 1e-6, xm[0], xm[1], xm[6], xm[7])
    qkv = torch.empty(B, T, 3 * E, device="cuda", dtype=torch.bfloat16)
    qkv2 = torch.empty(B, Tx, 3 * E, device="cuda", dtype=torch.bfloat16)
    o_c, o_x = attend(qkv, T, Tc, {"context": (h_c, Tc, 0), "latent": (h_x, Tx, Tc)})
    o_x2 = attend(qkv2, Tx, 0, {"latent_dual": (h_x2, Tx, 0)})[1]
    rc, rx = c.view(B * Tc, E), x.view(B * Tx, E)
    sd3.linear_gate_residual(o_x.view(B * Tx, E), *lin("latent_attn_Wout"), xm[2], Tx, rx)
    sd3.linear_gate_residual(o_c.view(B * Tc, E), *lin("context_attn_Wout"), cm[2], Tc, rc)
    sd3.linear_gate_residual(o_x2.view(B * Tx, E), *lin("latent_dual_attn_Wout"), xm[8], Tx, rx)
    mlp("latent", rx, Tx, xm[3], xm[4], xm[5])
    mlp("context", rc, Tc, cm[3], cm[4], cm[5])
    assert sd3.device_status() == 0
    assert torch.equal(xx, x) and torch.equal(cc, c)
    m.close()
