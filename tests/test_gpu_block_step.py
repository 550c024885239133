"""The whole-block decode step in one launch, against the CPU oracle: token counts on both sides of its limit, widths that leave
part of the grid without rows, ragged loads, every parameter type, repeated launches on one set of barrier counters."""
import pytest
import torch

from oracle import scan_oracle as O
from tests.helpers import RefShapedBlock, assert_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("Bsz,d_model,N", [(1, 16, 16), (1, 768, 16), (2, 20, 8), (3, 136, 16), (5, 64, 32), (8, 200, 64), (8, 1024, 16), (9, 64, 16),
                                           (8, 752, 16), (5, 768, 16), (3, 1536, 8), (2, 3072, 8),        # activations of just under and of 48 KB
                                           (4, 1024, 16), (4, 1032, 16), (8, 512, 8), (2, 2056, 8), (8, 2560, 16)])  # and around bfloat16's limit
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_block_step_vs_oracle(Bsz, d_model, N, dtype):
    from mamba_b200 import step
    torch.manual_seed(Bsz * 1000 + d_model)
    blk = RefShapedBlock(d_model, d_state=N)
    with torch.no_grad():
        blk.A_log.add_(0.1 * torch.randn_like(blk.A_log))
        blk.dt_proj.bias.uniform_(-4.0, -2.0)
    blk = blk.to(dtype)
    W = {k: v.detach().float() for k, v in blk.weights().items()}
    blk = blk.to(DEV)
    h, win = torch.randn(Bsz, 2 * d_model, N), torch.randn(Bsz, 2 * d_model, 3).to(dtype)
    co, ck = (h.clone(), win.float()), (h.to(DEV), win.to(DEV))
    rt, at = (1e-4, 1e-5) if dtype == torch.float32 else (3e-2, 3e-2)
    with torch.no_grad():
        for _ in range(3):
            x = torch.randn(Bsz, d_model).to(dtype)
            want, co = O.block_step(x.float(), co, W)
            got, ck = step(blk, x.to(DEV), ck)
            assert got.dtype == dtype and ck[0].dtype == torch.float32 and ck[1].dtype == dtype
            assert_close(got, want, rt, at * max(1.0, want.abs().max().item()), "output")
            assert_close(ck[0], co[0], rt, at * max(1.0, co[0].abs().max().item()), "state")
            assert_close(ck[1], co[1], rt, at * max(1.0, co[1].abs().max().item()), "window")


def test_block_step_first_token_and_graph():
    """h = None starts from zeros; a captured step replays like an eager one (a graph has barrier counters of its own)."""
    from mamba_b200 import step
    torch.manual_seed(3)
    blk = RefShapedBlock(64).to(DEV)
    x, win = torch.randn(2, 64, device=DEV), torch.zeros(2, 128, 3, device=DEV)
    with torch.no_grad():
        o0, c0 = step(blk, x, (None, win))
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            step(blk, x, (None, win))
        torch.cuda.current_stream().wait_stream(s)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            o1, c1 = step(blk, x, (None, win))
        for _ in range(3):
            g.replay()
    torch.cuda.synchronize()
    assert torch.equal(o0, o1) and torch.equal(c0[0], c1[0]) and torch.equal(c0[1], c1[1])


@pytest.mark.parametrize("Bsz", [2, 9])
def test_longest_filter(Bsz):
    """A filter of 8 steps runs, one of 9 is refused, on each path of a step."""
    from mamba_b200 import step
    for K in (8, 9):
        blk, x, win = RefShapedBlock(32, d_conv=K).to(DEV), torch.randn(Bsz, 32, device=DEV), torch.randn(Bsz, 64, K - 1, device=DEV)
        with torch.no_grad():
            if K == 9:
                with pytest.raises(RuntimeError):
                    step(blk, x, (None, win))
                continue
            got, (_, new) = step(blk, x, (None, win))
            want, (_, w2) = O.block_step(x.cpu(), (None, win.cpu()), {k: v.detach().cpu() for k, v in blk.weights().items()})
        assert_close(got, want, 1e-4, 1e-5)
        assert_close(new, w2, 1e-4, 1e-5)


def test_replicas_and_pruned_modules():
    """Blocks whose parameters are plain attributes run through their modules and give what the block itself gives."""
    import torch.nn.utils.prune as prune
    from mamba_b200 import mamba, step
    torch.manual_seed(5)
    blk = RefShapedBlock(32).to(DEV)
    x, token, cache = torch.randn(2, 20, 32, device=DEV), torch.randn(2, 32, device=DEV), (None, torch.zeros(2, 64, 3, device=DEV))
    replica = blk._replicate_for_data_parallel()
    for part, source in [(replica, blk)] + [(c._replicate_for_data_parallel(), c) for c in blk.children()]:
        for name, p in source._parameters.items():
            setattr(part, name, p)
        if part is not replica:
            replica._modules[next(k for k, v in blk._modules.items() if v is source)] = part
    with torch.no_grad():
        want = mamba.forward(blk, x), step(blk, token, cache)[0]
        got = [(mamba.forward(replica, x), step(replica, token, cache)[0])]
        for name, p in (("conv1d", "bias"), ("in_proj", "weight"), ("out_proj", "weight")):
            prune.identity(getattr(blk, name), p)
        got.append((mamba.forward(blk, x), step(blk, token, cache)[0]))
    for pair in got:
        for a, b in zip(pair, want):
            assert_close(a, b, 1e-4, 1e-5)


@pytest.mark.parametrize("Bsz", [2, 9, 31, 40])
@pytest.mark.parametrize("d_model", [32, 33])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_parameters_off_the_16_byte_grid(Bsz, d_model, dtype):
    """Every parameter one element into a flat buffer gives what parameters of their own give, on each path of a step."""
    from mamba_b200 import step
    torch.manual_seed(Bsz)
    blk = RefShapedBlock(d_model).to(dtype).to(DEV)
    x, h, win = (torch.randn(*s, device=DEV) for s in ((Bsz, d_model), (Bsz, 2 * d_model, 16), (Bsz, 2 * d_model, 3)))
    x, win = x.to(dtype), win.to(dtype)
    with torch.no_grad():
        want, (want_h, _) = step(blk, x, (h, win))
        for p in blk.parameters():
            flat = torch.zeros(p.numel() + 8, dtype=dtype, device=DEV)
            flat[1:1 + p.numel()] = p.flatten()
            p.data = flat[1:1 + p.numel()].view(p.shape)
            assert p.data_ptr() % 16
        got, (got_h, _) = step(blk, x, (h, win))
    rt, at = (1e-4, 1e-5) if dtype == torch.float32 else (3e-2, 3e-2)
    assert_close(got, want, rt, at)
    assert_close(got_h, want_h, rt, at)


@pytest.mark.expects_wait_timeout
def test_a_step_that_gave_up_is_reported_and_not_for_good():
    """Counters marked as a launch that gave up leaves them: later steps on them report it, and once that has been read the stream works
    again.  With MB200_CHECK_STATUS=1 the step itself raises."""
    import os
    import subprocess
    import sys
    from mamba_b200 import _lib, step
    from tests.helpers import ROOT
    torch.manual_seed(1)
    blk, x, cache = RefShapedBlock(64).to(DEV), torch.randn(2, 64, device=DEV), (None, torch.zeros(2, 128, 3, device=DEV))
    side = torch.cuda.Stream()
    with torch.no_grad():
        for stream in (torch.cuda.current_stream(), side):
            with torch.cuda.stream(stream):
                want = step(blk, x, cache)[0]
                _lib.host().selftest_block_step_give_up(x)
                step(blk, x, cache)
                stream.synchronize()
                assert _lib.device_status(0) == 1 and _lib.device_status(0) == 0
                for _ in range(2):
                    assert torch.equal(step(blk, x, cache)[0], want)
                stream.synchronize()
                assert _lib.device_status(0) == 0
    code = ("import torch; from mamba_b200 import _lib, step; from tests.helpers import RefShapedBlock\n"
            "b, x = RefShapedBlock(64).cuda(), torch.zeros(2, 64, device='cuda'); c = (None, torch.zeros(2, 128, 3, device='cuda'))\n"
            "with torch.no_grad():\n"
            "    step(b, x, c); _lib.host().selftest_block_step_give_up(x)\n"
            "    try: step(b, x, c); print('silent')\n"
            "    except RuntimeError as e: print('raised', 'gave up' in str(e))\n"
            "    step(b, x, c); g = torch.cuda.CUDAGraph()\n"
            "    with torch.cuda.graph(g): step(b, x, c)\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, MB200_CHECK_STATUS="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "raised True" in r.stdout, r.stdout + r.stderr


def test_streams_of_others_keep_nothing():
    """A stream that torch did not make may be destroyed and its handle used again: it has counters for each call."""
    import ctypes
    from mamba_b200 import _lib, step
    torch.manual_seed(2)
    blk, x, cache = RefShapedBlock(64).to(DEV), torch.randn(2, 64, device=DEV), (None, torch.zeros(2, 128, 3, device=DEV))
    rt = ctypes.CDLL("libcudart.so.12")
    handle = ctypes.c_void_p()
    with torch.no_grad():
        want = step(blk, x, cache)[0]
        torch.cuda.synchronize()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(handle), 1) == 0
        with torch.cuda.stream(torch.cuda.ExternalStream(handle.value)):
            for _ in range(3):
                assert torch.equal(step(blk, x, cache)[0], want)
                _lib.host().selftest_block_step_give_up(x)
        torch.cuda.synchronize()
        assert rt.cudaStreamDestroy(handle) == 0
