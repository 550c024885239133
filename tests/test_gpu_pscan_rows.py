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


def test_products_that_overflow_before_any_state():
    """A above 1 over the steps before the first input that is not zero (64 steps of a warp forwards, 32 backwards): the product of A
    overflows, and the states stay zero there and numbers after it."""
    from mamba_b200.pscan import pscan_fwd_raw, pscan_bwd_raw
    g = torch.Generator().manual_seed(2)
    A, X = torch.full((2, 64, 3, 16), 8.0), torch.randn(2, 64, 3, 16, generator=g)
    X[:, :40] = 0
    assert_close(pscan_fwd_raw(A.cuda(), X.cuda())[0], O.scan_sequential(A.double(), X.double()).float(), 1e-4, 1e-5)
    A, H, G = torch.full((2, 32, 3, 16), 64.0), torch.randn(2, 32, 3, 16, generator=g), torch.randn(2, 32, 3, 16, generator=g)
    G[:, 12:] = 0
    want = O.scan_sequential(A.double(), G.flip(1).double()).flip(1)
    ga, gx = pscan_bwd_raw(A.cuda(), H.cuda(), G.cuda())
    assert_close(gx, want.float(), 1e-4, 1e-5)
    assert_close(ga[:, 1:], (H[:, :-1].double() * want[:, 1:]).float(), 1e-4, 1e-5)


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("t", [0, 1, 4, 7, 8, 16, 63, 64, 511])
def test_values_that_are_no_numbers(t, value):
    """One such value in A leaves numbers where it leaves them step by step, and only there.  (An infinite state may come out as NaN
    further on: spans are combined with states that start from zero, whose sign may be the other one.)"""
    import mamba_b200
    g = torch.Generator().manual_seed(t)
    A, X = 0.3 + 0.7 * torch.rand(1, 512, 2, 16, generator=g), torch.randn(1, 512, 2, 16, generator=g)
    A[0, t, 1] = value
    want = O.scan_sequential(A, X)
    if t == 0:                                                 # the kernels walk from zero, and zero times these is NaN
        want[0, :, 1] = float("nan")
    got = mamba_b200.pscan(A.cuda(), X.cuda()).cpu()
    assert torch.equal(got.isfinite(), want.isfinite())
    assert_close(got[want.isfinite()], want[want.isfinite()], 1e-4, 1e-5)
