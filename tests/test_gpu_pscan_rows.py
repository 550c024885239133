"""PScan rows spread over one CTA: lengths around the steps of a thread, of a CTA and of several rounds of it; channel counts off the
tile and off the vector; incoming and outgoing state; bfloat16; against the sequential oracle."""
import pytest
import torch

from oracle import scan_oracle as O
from tests.helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 7, 8, 9, 127, 255, 257, 512, 513, 1025, 2048])
@pytest.mark.parametrize("D,N,dtype", [(1, 1, torch.float32), (3, 16, torch.float32), (5, 7, torch.float32), (3, 8, torch.bfloat16), (1, 5, torch.bfloat16)])
def test_rows_in_one_cta(L, D, N, dtype):
    from mamba_b200.pscan import pscan_fwd_raw, pscan_bwd_raw
    g = torch.Generator().manual_seed(L * 31 + D)
    shape = (2, L, D, N)
    A = (0.3 + 0.7 * torch.rand(shape, generator=g)).to(dtype)
    X, G = (torch.randn(shape, generator=g).to(dtype) for _ in range(2))
    h0 = torch.randn(2, D * N, generator=g)
    Ad, Xd = A.double().requires_grad_(), X.double().requires_grad_()
    Xs = torch.cat([Xd[:, :1] + Ad[:, :1] * h0.double().view(2, 1, D, N), Xd[:, 1:]], 1)
    want = O.scan_sequential(Ad, Xs)
    a, x, gy = (t.cuda() for t in (A, X, G))
    H, hT = pscan_fwd_raw(a, x, h0=h0.cuda(), want_last=True)
    rt, at = (1e-4, 1e-5) if dtype == torch.float32 else (2e-2, 2e-2)
    assert_close(H, want.float(), rt, at, "H")
    assert_close(hT, want[:, -1].reshape(2, -1).float(), 1e-4, 1e-5 if dtype == torch.float32 else 1e-4, "state")
    Hs = want.to(dtype).detach()
    gA, gX = torch.autograd.grad(want, (Ad, Xd), G.double())
    ga, gx = pscan_bwd_raw(a, Hs.cuda(), gy, h0=h0.cuda())
    assert_close(ga, gA.float(), rt, 20 * at, "gradA")
    assert_close(gx, gX.float(), rt, 5 * at, "gradX")
