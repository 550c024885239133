"""Saved states in their two orders: (ED, N) per entry and two by two (MB200_PAIRED_STATES)."""
import pytest
import torch

from tests.helpers import assert_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _strides(*ts):
    return [s for t in ts for s in (t.stride(0), t.stride(1))]


def _forward(lib, d, flags, paired):
    B, L, E = d["x"].shape
    N, c = d["A"].shape[1], (L + 7) // 8
    y = torch.empty_strided(d["x"].shape, d["x"].stride(), device=DEV)
    carries = torch.full((B, c, N // 2, E, 2) if paired else (B, c, E, N), float("nan"), device=DEV)
    rc = lib.mb200_sscan_fwd(d["x"].data_ptr(), d["delta"].data_ptr(), d["z"].data_ptr(), d["A"].data_ptr(), d["B"].data_ptr(), d["C"].data_ptr(),
                             d["D"].data_ptr(), None, None, y.data_ptr(), None, carries.data_ptr(), B, L, E, N,
                             *_strides(d["x"], d["delta"], d["z"], d["B"], d["C"], y), 0, flags | (8 if paired else 0), None)
    assert rc == 0
    return carries


def _backward(lib, d, carries, flags, paired):
    B, L, E = d["x"].shape
    N = d["A"].shape[1]
    dx, dd, dz = (torch.empty_strided(d["x"].shape, d["x"].stride(), device=DEV) for _ in range(3))
    dB, dC, dA, dD = (torch.zeros(s, device=DEV) for s in ((B, L, N), (B, L, N), (E, N), (E,)))
    rc = lib.mb200_sscan_bwd(d["x"].data_ptr(), d["delta"].data_ptr(), d["z"].data_ptr(), d["A"].data_ptr(), d["B"].data_ptr(), d["C"].data_ptr(),
                             d["D"].data_ptr(), None, d["dy"].data_ptr(), carries.data_ptr(), None, dx.data_ptr(), dd.data_ptr(), dz.data_ptr(),
                             dB.data_ptr(), dC.data_ptr(), dA.data_ptr(), dD.data_ptr(), None, None, B, L, E, N,
                             *_strides(d["x"], d["delta"], d["z"], d["B"], d["C"], d["dy"], dx, dd, dz), 0, flags | (8 if paired else 0), None)
    assert rc == 0
    return dx, dd, dz, dB, dC, dA, dD


# Widths: whole tiles, ragged, odd (the second channel of the last pair missing), one channel.  Rows off the 16-byte grid
# (stride = 35) and N = 32 (backward) take the general kernels.
@pytest.mark.parametrize("E, stride, N, reverse", [(64, 64, 16, False), (40, 40, 16, True), (33, 36, 16, False), (33, 36, 16, True),
                                                   (1, 4, 16, False), (35, 35, 16, False), (40, 40, 32, False)])
@pytest.mark.parametrize("L", [1, 8, 45])
def test_both_orders_agree(E, stride, N, reverse, L):
    from mamba_b200 import _lib
    lib = _lib.load()
    g = torch.Generator().manual_seed(E + L)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)
    d = {k: r(2, L, stride)[..., :E] for k in ("x", "z", "dy")}
    d["delta"] = torch.nn.functional.softplus(r(2, L, stride) - 3)[..., :E]
    d.update(A=-torch.exp(r(E, N)), B=r(2, L, N), C=r(2, L, N), D=r(E))
    flags = 2 if reverse else 0
    plain, paired = _forward(lib, d, flags, False), _forward(lib, d, flags, True)
    assert torch.equal(paired.permute(0, 1, 3, 2, 4).reshape(plain.shape), plain)
    for name, a, b in zip("dx ddelta dz dB dC dA dD".split(), _backward(lib, d, plain, flags, False), _backward(lib, d, paired, flags, True)):
        if name in ("dx", "ddelta", "dz"):
            assert torch.equal(a, b), name
        else:                       # float atomics: at most 90 terms in another order, each sum good to 90 * 2^-24 of its largest
            assert_close(a, b, 1e-5, 1e-5 * max(1.0, b.abs().max().item()))


@pytest.mark.parametrize("reverse", [False, True])
def test_raw_backward_takes_both_orders(reverse):
    """States of either order, told apart by their shape, give the same gradients through the raw launchers."""
    from mamba_b200.kernels import sscan_bwd_raw, sscan_fwd_raw
    g = torch.Generator().manual_seed(2)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)
    B, L, E, N = 2, 37, 40, 16
    x, z, dy, Bm, Cm, D = r(B, L, E), r(B, L, E), r(B, L, E), r(B, L, N), r(B, L, N), r(E)
    delta, A = torch.nn.functional.softplus(r(B, L, E) - 3), -torch.exp(r(E, N))
    paired = sscan_fwd_raw(x, delta, A, Bm, Cm, D, z, want_carries=True, reverse=reverse)[2]
    plain = paired.permute(0, 1, 3, 2, 4).reshape(B, -1, E, N).contiguous()
    want, got = (sscan_bwd_raw(x, delta, A, Bm, Cm, D, z, None, dy, c, reverse=reverse) for c in (paired, plain))
    for i, (a, b) in enumerate(zip(got, want)):
        if a is None:
            continue
        if i < 3:
            assert torch.equal(a, b)
        else:                       # float atomics, as above: at most 2 * 37 terms in another order
            assert_close(a, b, 1e-5, 1e-5 * max(1.0, b.abs().max().item()))
