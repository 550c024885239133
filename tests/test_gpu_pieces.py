"""Sequences cut into uneven pieces inside the kernels (tensor-map path): last pieces of one timestep, one tile, ragged tiles;
ragged channel tiles; pieces that are not whole saved-state chunks of the row; against the float64 oracle."""
import pytest
import torch

from tests.helpers import scan_inputs, assert_close
from tests.test_gpu_sscan import RTOL, ATOL, BF_RTOL, BF_ATOL, _oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("Bsz,L,ED,pieces", [(1, 33, 32, 3), (1, 129, 40, 3), (2, 200, 96, 5), (1, 257, 64, 2), (3, 100, 8, 4), (1, 500, 36, 7)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_uneven_pieces_vs_oracle(Bsz, L, ED, pieces, dtype, monkeypatch):
    """The entry points with pieces, called as the host code calls them."""
    import ctypes
    from mamba_b200 import _lib
    if dtype == torch.bfloat16 and ED % 8:
        pytest.skip("no tensor map for this width")
    lib = _lib.load()
    inp = scan_inputs(L + ED, Bsz, L, ED, 16, dtype=dtype, structured_A=False, big_delta=True)
    yo, ho, go = _oracle(inp)
    t = {k: v.to(DEV).to(dtype if k in ("x", "delta", "B", "C", "z", "gy") else torch.float32).contiguous() for k, v in inp.items()}
    n = -(-L // (16 * pieces)) * 16
    assert (pieces - 1) * n < L
    new = lambda *s, dt=torch.float32: torch.zeros(*s, dtype=dt, device=DEV)
    code, st = _lib.dtype_code(dtype), torch.cuda.current_stream().cuda_stream
    p = lambda v: None if v is None else v.data_ptr()
    ss = lambda *vs: [k for v in vs for k in (v.stride(0), v.stride(1))]
    P, S, h_in, G, g_in = (new(Bsz, pieces, ED, 16) for _ in range(5))
    y, hT, car = new(Bsz, L, ED, dt=dtype), new(Bsz, ED, 16), new(Bsz, -(-L // 8), ED, 16)
    i64, i32, vp = ctypes.c_int64, ctypes.c_int, ctypes.c_void_p

    def call(name, ptrs, strides, N=16):
        fn = getattr(lib, name)
        fn.argtypes = [vp] * len(ptrs) + [i64] * 3 + [i32] + [i64] * len(strides) + [i32, i32, i64, i64, vp]
        rc = fn(*map(p, ptrs), Bsz, L, ED, N, *strides, code, 0, pieces, n, st)
        assert rc == 0, (name, lib.mb200_strerror(rc))

    x, d, z, Bm, Cm, gy, A, D = (t[k] for k in ("x", "delta", "z", "B", "C", "gy", "A", "D"))
    call("mb200_sscan_fwd_carry_pieces", [x, d, A, Bm, None, S, P], ss(x, d, Bm))
    fold = lambda a, b, o, rev: lib.mb200_carry_fold_range(p(a), p(b), None, p(o), Bsz, pieces, ED * 16, 0, pieces, rev, st)
    assert fold(P, S, h_in, 0) == 0
    call("mb200_sscan_fwd_pieces", [x, d, z, A, Bm, Cm, D, None, h_in, y, hT, car], ss(x, d, z, Bm, Cm, y))
    for saved in (None, torch.zeros_like(car)):                         # without y too: one state a row, and nothing behind them
        last = torch.full((Bsz * pieces, ED, 16), 7.0, device=DEV)
        call("mb200_sscan_fwd_pieces", [x, d, z, A, Bm, Cm, D, None, h_in, None, last, saved], ss(x, d, z, Bm, Cm, y))
        assert torch.equal(last[:Bsz], hT) and (last[Bsz:] == 7.0).all() and (saved is None or torch.equal(saved, car))
    call("mb200_sscan_bwd_carry_pieces", [d, z, gy, Cm, A, None, G], ss(d, z, gy, Cm))
    assert fold(P, G, g_in, 1) == 0
    dx, dd, dz = (new(Bsz, L, ED, dt=dtype) for _ in range(3))
    dB, dC, dA, dD, g_out = new(Bsz, L, 16), new(Bsz, L, 16), new(ED, 16), new(ED), new(Bsz, ED, 16)
    call("mb200_sscan_bwd_pieces", [x, d, z, A, Bm, Cm, D, None, gy, car, g_in, dx, dd, dz, dB, dC, dA, dD, None, g_out],
         ss(x, d, z, Bm, Cm, gy, dx, dd, dz))
    rt, at = (RTOL, ATOL) if dtype == torch.float32 else (BF_RTOL, BF_ATOL)
    assert_close(y, yo.float(), rt, at * max(1.0, yo.abs().max().item()), "y")
    assert_close(hT, ho.float(), RTOL, ATOL * max(1.0, ho.abs().max().item()), "state")
    for k, g in {"x": dx, "delta": dd, "z": dz, "B": dB, "C": dC, "A": dA, "D": dD}.items():
        assert_close(g, go[k].float(), rt, at * 4 * max(1.0, go[k].abs().max().item()), "grad " + k)


def test_library_chooses_pieces_and_handles_awkward_gradients():
    """A short problem the library cuts by itself, with a gradient that is a narrow view, an incoming state and the outgoing one."""
    import mamba_b200
    inp = scan_inputs(5, 1, 777, 160, 16, structured_A=False, big_delta=True)
    h0 = torch.randn(1, 160, 16, generator=torch.Generator().manual_seed(1))
    yo, ho, go = _oracle(inp, h0=h0)
    lv = {k: inp[k].to(DEV).requires_grad_() for k in ("x", "delta", "A", "B", "C", "D", "z")}
    hl = h0.to(DEV).requires_grad_()
    y, hT = mamba_b200.selective_scan_fn(lv["x"], lv["delta"], lv["A"], lv["B"], lv["C"], lv["D"], z=lv["z"], h0=hl, return_last_state=True)
    wide = torch.zeros(1, 777, 165, device=DEV)
    wide[..., 3:163] = inp["gy"].to(DEV)
    y.backward(wide[..., 3:163])
    assert_close(y, yo.float(), RTOL, ATOL * yo.abs().max().item(), "y")
    assert_close(hT, ho.float(), RTOL, ATOL * max(1.0, ho.abs().max().item()), "state")
    for k in ("x", "delta", "A", "B", "C", "D", "z"):
        assert_close(lv[k].grad, go[k].float(), RTOL, ATOL * 4 * max(1.0, go[k].abs().max().item()), "grad " + k)
    assert_close(hl.grad, go["h0"].float(), RTOL, ATOL * 4 * max(1.0, go["h0"].abs().max().item()), "grad h0")


def test_carries_that_were_not_written_do_not_enter():
    """The last piece of a row has no carry pass: whatever lies in its decay product must not reach the gradient carries."""
    from mamba_b200.kernels import carry_fold_range
    P, G = torch.rand(2, 3, 40, 16, device=DEV), torch.randn(2, 3, 40, 16, device=DEV)
    P[:, -1] = float("nan")
    got = carry_fold_range(P, G, None, 0, 3, True)
    assert torch.equal(got[:, 2], torch.zeros_like(got[:, 2])) and torch.equal(got[:, 1], G[:, 2])
    assert torch.allclose(got[:, 0], P[:, 1] * G[:, 2] + G[:, 1], atol=1e-5)
    x = torch.full((1 << 24,), float("nan"), device=DEV)                    # garbage for the next allocations
    del x
    a = [torch.randn(1, 2048, 1536, device=DEV, dtype=torch.bfloat16, requires_grad=True) for _ in range(2)]
    A = -torch.rand(1536, 16, device=DEV) - 0.5
    BC = [torch.randn(1, 2048, 16, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    import mamba_b200
    y = mamba_b200.selective_scan_fn(a[0], a[1], A, *BC, delta_bias=torch.zeros(1536, device=DEV))
    for g in torch.autograd.grad(y, a, torch.ones_like(y)):
        assert torch.isfinite(g).all()


@pytest.mark.parametrize("reverse", [False, True])
def test_first_call_of_a_thread(reverse):
    """A scan's backward as the first CUDA call that autograd's thread makes, and a forward as the first of a new thread: tensor maps are
    encoded there as everywhere (rows of any length are cut, and scanned in reverse, on the tensor-map path only)."""
    import os
    import subprocess
    import sys
    from tests.helpers import ROOT
    code = ("import threading, torch, mamba_b200\n"
            "torch.manual_seed(0); r = lambda *s: torch.randn(*s, device='cuda')\n"
            "leaves = [t.requires_grad_() for t in (r(1, 1003, 256), 0.1 * r(1, 1003, 256).abs(), -r(256, 16).exp(), r(1, 1003, 16), r(1, 1003, 16))]\n"
            f"run = lambda: mamba_b200.selective_scan_fn(*leaves, reverse={reverse})\n"
            "dy, first = r(1, 1003, 256), []\n"
            "t = threading.Thread(target=lambda: first.append(run().detach())); t.start(); t.join()\n"
            "y = run(); a = torch.autograd.grad(y, leaves, dy); b = torch.autograd.grad(run(), leaves, dy)\n"
            "assert torch.equal(first[0], y)\n"
            "for p, q in zip(a, b): assert (p - q).norm() <= 1e-5 * q.norm()\n"
            "print('done')\n")
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "done" in p.stdout, p.stdout + p.stderr
