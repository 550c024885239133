"""Fused depthwise causal conv1d + SiLU against the reference's own op sequence run on the CPU."""
import pytest
import torch
import torch.nn.functional as F

from tests.helpers import assert_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _reference(x, w, b):
    """mambapy/mamba.py:217-221 in float64: transpose, Conv1d(padding=3, groups=ED), slice, transpose, silu."""
    L = x.shape[1]
    y = F.conv1d(x.transpose(1, 2), w, b, padding=w.shape[-1] - 1, groups=w.shape[0])[:, :, :L].transpose(1, 2)
    return F.silu(y)


@pytest.mark.parametrize("Bsz,L,ED", [(2, 64, 32), (1, 1, 8), (3, 130, 40), (2, 257, 33), (1, 3, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_conv1d_silu_forward_backward(Bsz, L, ED, dtype):
    import mamba_b200
    g = torch.Generator().manual_seed(L + ED)
    x = torch.randn(Bsz, L, ED, generator=g).to(dtype).float()
    w = torch.randn(ED, 1, 4, generator=g) * 0.5
    b = torch.randn(ED, generator=g) * 0.1
    gy = torch.randn(Bsz, L, ED, generator=g).to(dtype).float()
    xr, wr, br = (t.double().requires_grad_() for t in (x, w, b))
    yr = _reference(xr, wr, br)
    yr.backward(gy.double())
    xc, wc, bc = x.to(DEV).to(dtype).requires_grad_(), w.to(DEV).requires_grad_(), b.to(DEV).requires_grad_()
    y = mamba_b200.causal_conv1d_silu(xc, wc, bc)
    y.backward(gy.to(DEV).to(dtype))
    tol = (1e-4, 1e-5) if dtype == torch.float32 else (2e-2, 2e-2)
    assert y.dtype == dtype and y.shape == (Bsz, L, ED)
    assert_close(y, yr.float(), *tol, "y")
    assert_close(xc.grad, xr.grad.float(), *tol, "dx")
    scale = max(1.0, wr.grad.abs().max().item())
    assert_close(wc.grad, wr.grad.float(), tol[0] * 10, tol[1] * scale * 4, "dw")
    assert_close(bc.grad, br.grad.float(), tol[0] * 10, tol[1] * scale * 4, "dbias")


def test_conv1d_silu_on_a_chunk_view():
    """x as the first half of the in_proj output (a strided view), as MambaBlock.forward has it."""
    import mamba_b200
    g = torch.Generator().manual_seed(5)
    xz = torch.randn(2, 100, 64, generator=g).to(DEV)
    x, _ = xz.chunk(2, dim=-1)
    w = torch.randn(32, 1, 4, generator=g).to(DEV)
    y = mamba_b200.causal_conv1d_silu(x, w, None)
    yr = _reference(x.cpu().double(), w.cpu().double(), None)
    assert_close(y, yr.float(), 1e-4, 1e-5)


@pytest.mark.parametrize("Bsz,L,ED", [(8, 2048, 1536), (16, 1031, 1544)])
def test_wide_bfloat16_backward(Bsz, L, ED):
    """Chunks long enough for loads a group ahead, against torch in float32."""
    import mamba_b200
    g = torch.Generator(device="cuda").manual_seed(L)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, dy, w, b = new(Bsz, L, ED).bfloat16().requires_grad_(), new(Bsz, L, ED).bfloat16(), new(ED, 1, 4).requires_grad_(), new(ED).requires_grad_()
    got = torch.autograd.grad(mamba_b200.mamba.causal_conv1d_silu(x, w, b), (x, w, b), dy)
    x32 = x.detach().float().requires_grad_()
    y = F.silu(F.conv1d(x32.transpose(1, 2), w, b, groups=ED, padding=3)[..., :L].transpose(1, 2))
    for a, r in zip(got, torch.autograd.grad(y, (x32, w, b), dy.float())):
        assert ((a.float() - r).norm() / r.norm()).item() < 5e-3


@pytest.mark.parametrize("Bsz,L,ED", [(64, 301, 772), (64, 301, 195), (64, 197, 772), (64, 31, 132), (64, 31, 131), (3, 1003, 516)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_backward_chunks(Bsz, L, ED, dtype):
    """Long chunks (64 steps in the first two) and short ones, four channels a thread and one, against float64.  float32: two factors of every term come from a
    sigmoid good to 1e-5; bfloat16: dx is rounded to 2^-9."""
    import mamba_b200
    g = torch.Generator(device="cuda").manual_seed(L + ED)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, dy, w, b = new(Bsz, L, ED).to(dtype).requires_grad_(), new(Bsz, L, ED).to(dtype), new(ED, 1, 4).requires_grad_(), new(ED).requires_grad_()
    got = torch.autograd.grad(mamba_b200.mamba.causal_conv1d_silu(x, w, b), (x, w, b), dy)
    x64, w64, b64 = (t.detach().double().requires_grad_() for t in (x, w, b))
    xp = F.pad(x64, (0, 0, 3, 0))
    y = F.silu(sum(xp[:, k:k + L] * w64[:, 0, k] for k in range(4)) + b64)
    for a, r in zip(got, torch.autograd.grad(y, (x64, w64, b64), dy.double())):
        assert ((a.double() - r).norm() / r.norm()).item() < (3e-3 if dtype == torch.bfloat16 else 2e-5)


@pytest.mark.parametrize("Bsz,L,ED", [(8, 2048, 1536), (8, 2041, 1536), (8, 1985, 1540), (4, 31, 2052)]
                         + [(8, 1984 + left, 1536) for left in (8, 9, 16, 17, 32, 33, 63)]
                         + [(2, L, ED) for L in (1, 8, 9, 16, 17, 31, 32, 33, 41, 49, 63) for ED in (132, 33)] + [(150, 300, 132), (150, 300, 33)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_forward_chunks(Bsz, L, ED, dtype):
    """Chunks of 64 (one wave of CTAs), whole, a step short, and with last ones at both ends of every number of groups; chunks of 32
    the same, four channels a thread and one.  (150 rows of 300 steps: 64-step chunks for five of a CTA's eight warps.)"""
    import mamba_b200
    g = torch.Generator(device="cuda").manual_seed(L)
    new = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, b = new(Bsz, L, ED).to(dtype), new(ED, 1, 4), new(ED)
    y = mamba_b200.mamba.causal_conv1d_silu(x, w, b)
    xp = F.pad(x.float(), (0, 0, 3, 0))
    r = F.silu(sum(xp[:, k:k + L] * w[:, 0, k] for k in range(4)) + b)
    assert ((y.float() - r).norm() / r.norm()).item() < (3e-3 if dtype == torch.bfloat16 else 1e-5)
