"""Both outputs of LayerNorm + modulate against float64, on all samples: CTAs that take one row, a warp per row, several
rows that cross from one sample into the next, and rows wider than the CTA-per-row kernels take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 66, 4851 and 33000 rows; 1540 is one quad past the widest row of the CTA-per-row kernels
@pytest.mark.parametrize("E", [128, 1000, 1536, 1540])
@pytest.mark.parametrize("B,T", [(2, 33), (147, 33), (1000, 33)])
@pytest.mark.parametrize("dual", [False, True])
def test_all_samples_match_float64(sd3, E, B, T, dual):
    gen = torch.Generator(device="cuda").manual_seed(E + B)
    x = torch.empty(B, T, E, device="cuda").normal_(1.0, 3.0, generator=gen)
    mod = torch.empty(B, 4 * E, device="cuda").normal_(generator=gen)
    args = [mod[:, i * E:(i + 1) * E] for i in range(4 if dual else 2)]
    outs = sd3.layernorm_modulate(x, B, T, E, 1e-6, *args)
    for i in range(2 if dual else 1):
        shift, scale = args[2 * i].double()[:, None], args[2 * i + 1].double()[:, None]
        ref = torch.nn.functional.layer_norm(x.double(), (E,), eps=1e-6) * (1 + scale) + shift
        # bf16: half an ulp, 2^-8; fp32 arithmetic before it: a few roundings of 6e-8 on terms of up to 5 * 6
        assert ((outs[i].view(B, T, E).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 4e-5).all()
    assert sd3.device_status() == 0
