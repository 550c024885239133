"""Conv backward with chunks long enough for loads a group ahead (wide bfloat16 problems), against torch in float32."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Bsz,L,ED", [(8, 2048, 1536), (16, 1031, 1544)])
def test_wide_bfloat16_backward(Bsz, L, ED):
    import mamba_b200
    g = torch.Generator(device="cuda").manual_seed(L)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, dy, w, b = new(Bsz, L, ED).bfloat16().requires_grad_(), new(Bsz, L, ED).bfloat16(), new(ED, 1, 4).requires_grad_(), new(ED).requires_grad_()
    got = torch.autograd.grad(mamba_b200.mamba.causal_conv1d_silu(x, w, b), (x, w, b), dy)
    x32 = x.detach().float().requires_grad_()
    y = F.silu(F.conv1d(x32.transpose(1, 2), w, b, groups=ED, padding=3)[..., :L].transpose(1, 2))
    for a, r in zip(got, torch.autograd.grad(y, (x32, w, b), dy.float())):
        assert ((a.float() - r).norm() / r.norm()).item() < 5e-3
