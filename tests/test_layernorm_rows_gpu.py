"""LayerNorm + modulate runs a CTA per row, a warp per row or several rows per CTA, by their number: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# a quad per lane and one quad more; a ragged last quad group; the widest row of the CTA-per-row kernel
@pytest.mark.parametrize("E", [128, 132, 1000, 1536])
@pytest.mark.parametrize("dual", [False, True])
def test_few_rows_match_many(sd3, E, dual):
    T, B = 33, 1000  # 33000 rows: several per CTA, which take rows of neighbouring samples
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.empty(B, T, E, device="cuda").normal_(1.0, 3.0, generator=gen)
    mod = torch.empty(B, 4 * E, device="cuda").normal_(generator=gen)

    def run(n):
        args = [mod[:n, i * E:(i + 1) * E] for i in range(4 if dual else 2)]
        return sd3.layernorm_modulate(x[:n].contiguous(), n, T, E, 1e-6, *args)

    many = run(B)
    for n in (1, 3, 100, 150):  # up to 3300 rows a CTA per row, 4950 with one modulation a warp per row
        few = run(n)
        for a, b in zip(few, many):
            assert (a is None and b is None) or torch.equal(a.view(n, T, E), b.view(B, T, E)[:n])
    ref = torch.nn.functional.layer_norm(x[:3], (E,), eps=1e-6) * (1 + mod[:3, None, E:2 * E]) + mod[:3, None, :E]
    # one bf16 rounding, half an ulp
    assert ((many[0].view(B, T, E)[:3].float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()
