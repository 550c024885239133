"""Several small matrix products in one launch: sizes around the tile and the slab, transposed and padded operands, beta, both types."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

i64, f32, vp = ctypes.c_int64, ctypes.c_float, ctypes.c_void_p


class Product(ctypes.Structure):
    _fields_ = [("a", vp), ("b", vp), ("out", vp)] + [(k, i64) for k in ("M", "N", "K", "a_rm", "a_ck", "b_rk", "b_cn", "out_rm")] + [
        ("alpha", f32), ("beta", f32), ("out_dtype", ctypes.c_int)]


@pytest.mark.parametrize("dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("sizes", [[(1, 1, 1)], [(31, 33, 32), (32, 32, 64)], [(65, 7, 33), (2, 96, 200), (40, 40, 31), (122, 64, 256)], [(5, 6, 0)]])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True)])
def test_products(dtype, out_dtype, sizes, ta, tb):
    from mamba_b200 import _lib
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    jobs, want, outs = (Product * len(sizes))(), [], []
    keep = []
    for j, (M, N, K) in enumerate(sizes):
        new = lambda r, c, t: (torch.randn(c, r + 3, generator=g, device="cuda").to(dtype)[:, :r].t() if t
                               else torch.randn(r, c + 3, generator=g, device="cuda").to(dtype)[:, :c])
        a, b, beta = new(M, K, ta), new(K, N, tb), 0.5 * (j % 2)
        pad = torch.full((M, N + 5), 7.0, dtype=out_dtype, device="cuda")
        o = pad[:, :N]
        want.append((0.25 * (a.double() @ b.double()) + beta * o.double()))
        jobs[j] = Product(a.data_ptr(), b.data_ptr(), o.data_ptr(), M, N, K, a.stride(0), a.stride(1), b.stride(0), b.stride(1), o.stride(0), 0.25, beta,
                          _lib.dtype_code(out_dtype))
        outs.append((pad, o))
        keep += [a, b]
    lib.mb200_small_gemm.argtypes = [vp, ctypes.c_int, ctypes.c_int, vp]
    rc = lib.mb200_small_gemm(ctypes.byref(jobs), len(sizes), _lib.dtype_code(dtype), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.mb200_strerror(rc)
    tol = 1e-5 if out_dtype == torch.float32 else 1e-2
    for (pad, o), w in zip(outs, want):
        assert torch.allclose(o.double(), w, rtol=tol, atol=tol * 10)
        assert (pad[:, o.shape[1]:] == 7).all()
