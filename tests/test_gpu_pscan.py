"""PScan kernels against the golden vectors of the reference and the CPU oracle (needs a GPU)."""
import numpy as np
import pytest
import torch

from oracle import scan_oracle as O
from tests.helpers import golden, assert_close

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-4, 1e-5          # float32 tolerance of the parity contract


def _dev():
    return torch.device("cuda:0")


def test_golden_forward_backward():
    import mamba_b200
    g = golden("pscan_cases.npz")
    for L in g["Ls"]:
        A = torch.from_numpy(g[f"L{L}_A"]).to(_dev()).requires_grad_()
        X = torch.from_numpy(g[f"L{L}_X"]).to(_dev()).requires_grad_()
        A0, X0 = A.detach().clone(), X.detach().clone()
        H = mamba_b200.pscan(A, X)
        H.backward(torch.from_numpy(g[f"L{L}_G"]).to(_dev()))
        assert_close(H, g[f"L{L}_H"], RTOL, ATOL, f"H L={L}")
        assert_close(A.grad, g[f"L{L}_gA"], RTOL, ATOL, f"gradA L={L}")
        assert_close(X.grad, g[f"L{L}_gX"], RTOL, ATOL, f"gradX L={L}")
        assert torch.equal(A.detach(), A0) and torch.equal(X.detach(), X0), "inputs were modified"
        assert H.shape == X.shape and H.dtype == X.dtype


def test_known_answer_vector():
    import mamba_b200
    g = golden("pscan_kat.npz")
    X = torch.from_numpy(g["X"]).view(1, 16, 1, 1).to(_dev())
    H = mamba_b200.pscan(torch.ones_like(X), X)
    assert np.array_equal(H.reshape(-1).cpu().numpy(), g["H"])      # integers: exact


@pytest.mark.parametrize("shape", [(1, 4096, 3, 16), (2, 1000, 5, 8), (3, 129, 7, 4), (1, 65, 1, 1),
                                   (2, 300, 33, 16)])
def test_against_sequential_oracle(shape):
    """Shapes that take the segmented (low-parallelism) and the scalar (unaligned) paths."""
    import mamba_b200
    g = torch.Generator().manual_seed(sum(shape))
    A = torch.exp(-torch.nn.functional.softplus(torch.randn(shape, generator=g)))
    X = torch.randn(shape, generator=g)
    G = torch.randn(shape, generator=g)
    Ad, Xd = A.double().requires_grad_(), X.double().requires_grad_()
    Hs = O.scan_sequential(Ad, Xd)
    Hs.backward(G.double())
    Ac, Xc = A.to(_dev()).requires_grad_(), X.to(_dev()).requires_grad_()
    H = mamba_b200.pscan(Ac, Xc)
    H.backward(G.to(_dev()))
    assert_close(H, Hs.float(), RTOL, ATOL)
    assert_close(Ac.grad, Ad.grad.float(), RTOL, 5 * ATOL)
    assert_close(Xc.grad, Xd.grad.float(), RTOL, 5 * ATOL)


def test_strided_inputs_and_empty():
    import mamba_b200
    g = torch.Generator().manual_seed(7)
    big = torch.rand(2, 50, 6, 32, generator=g).to(_dev())
    A, X = big[..., :16], big[..., 16:]                       # last-dim slices: (D, N) block not dense
    H = mamba_b200.pscan(A, X)
    Hs = O.scan_sequential(A.cpu().double(), X.cpu().double())
    assert_close(H, Hs.float(), RTOL, ATOL)
    At, Xt = big.transpose(0, 1)[:, :, :, :16], big.transpose(0, 1)[:, :, :, 16:]   # (50, 2, 6, 16)
    H2 = mamba_b200.pscan(At, Xt)
    Hs2 = O.scan_sequential(At.cpu().double(), Xt.cpu().double())
    assert_close(H2, Hs2.float(), RTOL, ATOL)
    E = torch.empty(2, 0, 3, 16, device=_dev())
    assert mamba_b200.pscan(E, E).shape == (2, 0, 3, 16)


def test_bf16_io_fp32_state():
    import mamba_b200
    g = torch.Generator().manual_seed(11)
    shape = (2, 257, 8, 16)
    A = torch.exp(-torch.nn.functional.softplus(torch.randn(shape, generator=g))).bfloat16()
    X = torch.randn(shape, generator=g).bfloat16()
    H = mamba_b200.pscan(A.to(_dev()), X.to(_dev()))
    assert H.dtype == torch.bfloat16
    Hs = O.scan_sequential(A.double(), X.double())
    assert_close(H, Hs.float(), 2e-2, 2e-2)                   # bf16 output rounding


def test_full_size_split_consistency():
    """At the benchmark's per-row size: scanning a sequence equals scanning its two halves with
    the state carried over (a size-independent property, no oracle needed)."""
    from mamba_b200.pscan import pscan_fwd_raw
    g = torch.Generator(device="cuda").manual_seed(5)
    shape = (2, 2048, 1536, 16)
    A = torch.exp(-torch.nn.functional.softplus(torch.randn(shape, generator=g, device=_dev())))
    X = torch.randn(shape, generator=g, device=_dev())
    H, hT = pscan_fwd_raw(A, X, want_last=True)
    m = 1000
    H0, h0 = pscan_fwd_raw(A[:, :m], X[:, :m], want_last=True)
    H1, h1 = pscan_fwd_raw(A[:, m:], X[:, m:], h0=h0, want_last=True)
    assert torch.allclose(torch.cat([H0, H1], 1), H, rtol=1e-5, atol=1e-6)
    assert torch.allclose(h1, hT, rtol=1e-5, atol=1e-6)
    assert torch.allclose(hT.view(2, 1536, 16), H[:, -1], rtol=0, atol=0)


@pytest.mark.parametrize("L", [1, 7, 8, 9, 127, 255, 257, 512, 513, 1025, 2048])
@pytest.mark.parametrize("D,N,dtype", [(1, 1, torch.float32), (3, 16, torch.float32), (5, 7, torch.float32), (3, 8, torch.bfloat16), (1, 5, torch.bfloat16)])
def test_rows_in_one_cta(L, D, N, dtype):
    """Rows spread over one CTA: lengths around the steps of a thread, of a CTA and of several rounds of it; channel counts off the
    tile and off the vector; incoming and outgoing state; bfloat16; against the sequential oracle."""
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
