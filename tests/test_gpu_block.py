"""The native Mamba block (projections, one or both directions, one autograd node) against a float64 restatement of it: ranks off
the 16-byte grid, a projection the native call leaves to its module, frozen inputs, both directions with the halving."""
import math

import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from tests.helpers import RefShapedBlock

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _build(d_model, d_state, both):
    torch.manual_seed(d_model + d_state)
    m = RefShapedBlock(d_model, d_state)
    m.config.bidirectional, m.config.divide_output = both, True
    with torch.no_grad():
        m.dt_proj.bias.fill_(-3.0)
        m.A_log.add_(0.2 * torch.randn_like(m.A_log))
    if both:
        other = RefShapedBlock(d_model, d_state)
        for k in ("conv1d", "x_proj", "dt_proj", "A_log", "D"):
            setattr(m, k + "_b", getattr(other, k))
    return m.to(DEV)


def _direction(p, xz, R, N):
    w, b, wx, wdt, bdt, A_log, D = p
    L, W = xz.shape[1], xz.shape[2] // 2
    x = F.silu(F.conv1d(xz[..., :W].transpose(1, 2), w, b, groups=W, padding=3)[..., :L]).transpose(1, 2)
    dt, B, C = torch.split(x @ wx.t(), [R, N, N], -1)
    delta, A = F.softplus(dt @ wdt.t() + bdt), -torch.exp(A_log)
    h, ys = 0.0, []
    for t in range(L):
        h = torch.exp(delta[:, t, :, None] * A) * h + (delta[:, t] * x[:, t])[..., None] * B[:, t, None]
        ys.append((h * C[:, t, None]).sum(-1) + D * x[:, t])
    return torch.stack(ys, 1) * F.silu(xz[..., W:])


def _params(m, s):
    conv, x_proj, dt_proj = (getattr(m, k + s) for k in ("conv1d", "x_proj", "dt_proj"))
    return [conv.weight, conv.bias, x_proj.weight, dt_proj.weight, dt_proj.bias, getattr(m, "A_log" + s), getattr(m, "D" + s)]


def _plain(m, x, both, leaves):
    it = iter(leaves)
    d = {id(p): next(it) for p in m.parameters()}
    g = lambda s: [d[id(p)] for p in _params(m, s)]
    R, N = m.config.dt_rank, m.config.d_state
    xz = x @ d[id(m.in_proj.weight)].t()
    y = _direction(g(""), xz, R, N)
    if both:
        y = (y + _direction(g("_b"), xz.flip(1), R, N).flip(1)) / 2
    y = y @ d[id(m.out_proj.weight)].t()
    return y if m.out_proj.bias is None else y + d[id(m.out_proj.bias)]


@pytest.mark.parametrize("d_model,d_state,both,variant", [(32, 16, False, ""), (40, 16, False, "many"), (32, 16, True, "ragged"), (40, 16, False, "bias"), (24, 8, False, "hook"),
                                                          (48, 16, True, ""), (64, 16, True, "bias"), (20, 16, False, "frozen")])
@pytest.mark.parametrize("amp", [False, True])
def test_block_against_float64(d_model, d_state, both, variant, amp):
    from mamba_b200 import mamba, vim
    m = _build(d_model, d_state, both)
    if variant == "bias":
        m.out_proj = nn.Linear(2 * d_model, d_model, bias=True, device=DEV)
    if variant == "hook":
        m.in_proj.register_forward_hook(lambda mod, i, o: o)
    rows = {"many": 40, "ragged": 83}.get(variant, 3)               # tokens enough to cut the weight gradients, evenly or not
    x = torch.randn(rows, 37, d_model, device=DEV, requires_grad=variant != "frozen")
    if variant == "frozen":
        m.in_proj.weight.requires_grad_(False)
    dy = torch.randn(rows, 37, d_model, device=DEV)
    run = vim.forward if both else mamba.forward
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=amp):
        y = run(m, x)
    wanted = [t for t in [x, *m.parameters()] if t.requires_grad]
    got = torch.autograd.grad(y, wanted, dy.to(y.dtype))
    leaves = [p.detach().double().requires_grad_(p.requires_grad) for p in m.parameters()]
    x64 = x.detach().double().requires_grad_(x.requires_grad)
    want_y = _plain(m, x64, both, leaves)
    want = torch.autograd.grad(want_y, [t for t in [x64, *leaves] if t.requires_grad], dy.double())
    tol = 3e-2 if amp else 2e-5
    for a, b, t in zip([y, *got], [want_y, *want], [y, *wanted]):
        assert a.dtype == t.dtype and a.shape == b.shape
        err = ((a.double() - b).norm() / b.norm().clamp_min(1e-12)).item()
        assert err < tol and math.isfinite(err), (tuple(b.shape), err)


@pytest.mark.parametrize("both", [False, True])
@pytest.mark.parametrize("keep", ["clones", "host", "checkpoint"])
def test_saved_tensors_may_come_back_as_copies(both, keep):
    """Saved-tensor hooks and checkpointing hand the backward other tensors than the forward saved, each with storage of its own."""
    from torch.utils.checkpoint import checkpoint
    from mamba_b200 import mamba, vim
    m = _build(40, 16, both)
    run = vim.forward if both else mamba.forward
    x, dy = torch.randn(3, 37, 40, device=DEV, requires_grad=True), torch.randn(3, 37, 40, device=DEV)
    wanted = [x, *m.parameters()]
    want = torch.autograd.grad(run(m, x), wanted, dy)
    if keep == "checkpoint":
        y = checkpoint(run, m, x, use_reentrant=False)
    else:
        hooks = torch.autograd.graph.save_on_cpu() if keep == "host" else torch.autograd.graph.saved_tensors_hooks(torch.clone, lambda t: t)
        with hooks:
            y = run(m, x)
    for a, b in zip(torch.autograd.grad(y, wanted, dy), want):
        assert ((a - b).norm() / b.norm().clamp_min(1e-12)).item() < 1e-5      # sums over atomics, in any order


def _count(m, seen, kind):
    """Has `m` report its calls into `seen`, one way or another."""
    call = m.forward

    def forward(*a):
        seen.append(kind)
        return call(*a)
    if kind == "forward":
        m.forward = forward
    else:
        getattr(m, f"register_{kind}")(lambda *a: seen.append(kind))


@pytest.mark.parametrize("kind", ["forward_hook", "forward_pre_hook", "full_backward_hook", "full_backward_pre_hook", "forward"])
@pytest.mark.parametrize("name,both", [("in_proj", False), ("out_proj", False), ("in_proj", True), ("x_proj", True), ("x_proj_b", True), ("out_proj", True)])
def test_intercepted_projections_are_called(name, both, kind):
    """A projection that somebody listens to or has replaced is called as the module it is, with the same results."""
    from mamba_b200 import mamba, step, vim
    m, seen = _build(32, 16, both), []
    run = vim.forward if both else mamba.forward
    x, dy = torch.randn(2, 20, 32, device=DEV, requires_grad=True), torch.randn(2, 20, 32, device=DEV)
    token, cache = torch.randn(2, 32, device=DEV), (None, torch.zeros(2, 64, 3, device=DEV))
    want = [y := run(m, x), *torch.autograd.grad(y, [x, *m.parameters()], dy)]
    with torch.no_grad():
        want_step = step(m, token, cache)[0]
    _count(getattr(m, name), seen, kind)
    got = [y := run(m, x), *torch.autograd.grad(y, [x, *m.parameters()], dy)]
    assert seen == [kind]
    for a, b in zip(got, want):
        assert ((a - b).norm() / b.norm().clamp_min(1e-12)).item() < 1e-5
    with torch.no_grad():
        got_step = step(m, token, cache)[0]
    assert len(seen) == 1 + (name != "x_proj_b" and "backward" not in kind)
    assert ((got_step - want_step).norm() / want_step.norm()).item() < 1e-5


def test_bidirectional_block_with_biases_where_none_are_usual():
    """x_proj with a bias, dt_proj without one: accepted, and the biases count."""
    from mamba_b200 import vim
    m = _build(32, 16, True)
    x = torch.randn(2, 20, 32, device=DEV)
    with torch.no_grad():
        want = vim.forward(m, x)
        for s in ("", "_b"):
            old = getattr(m, "x_proj" + s)
            new = nn.Linear(64, 34, device=DEV)
            new.weight.copy_(old.weight)
            new.bias.zero_()
            setattr(m, "x_proj" + s, new)
        assert (vim.forward(m, x) - want).norm() / want.norm() < 1e-5
        m.x_proj_b.bias.fill_(0.5)
        assert (vim.forward(m, x) - want).norm() / want.norm() > 1e-3
        m.dt_proj.bias = None
        m.dt_proj.weight.abs_()
        assert torch.isfinite(vim.forward(m, 0.01 * x)).all()


@pytest.mark.parametrize("name,shape", [("in_proj", (96, 32)), ("in_proj", (128, 40)), ("conv1d", (48, 1, 4)), ("x_proj", (33, 64)), ("x_proj", (34, 48)),
                                        ("dt_proj", (64, 3)), ("dt_proj", (48, 2)), ("out_proj", (32, 48)), ("A_log", (48, 16)), ("A_log", (64, 8)),
                                        ("D", (48,))])
@pytest.mark.parametrize("both", [False, True])
def test_parameters_of_other_sizes_are_refused(name, shape, both):
    """What no longer is compared by calling the modules one by one is compared by the native block and step."""
    from mamba_b200 import mamba, step, vim
    m = _build(32, 16, both)
    p = nn.Parameter(torch.zeros(shape, device=DEV))
    if name in ("A_log", "D"):
        setattr(m, name, p)
    else:
        getattr(m, name).weight = p
    with torch.no_grad(), pytest.raises(RuntimeError):
        (vim.forward if both else mamba.forward)(m, torch.zeros(2, 20, 32, device=DEV))
    for rows in (2, 9):
        with torch.no_grad(), pytest.raises(RuntimeError):
            step(m, torch.zeros(rows, 32, device=DEV), (None, torch.zeros(rows, 64, 3, device=DEV)))


def test_activations_and_caches_of_other_sizes_are_refused():
    from mamba_b200 import mamba, step
    m = _build(32, 16, False)
    z = lambda *s: torch.zeros(*s, device=DEV)
    with torch.no_grad():
        for bad in (lambda: mamba.forward(m, z(2, 20, 40)), lambda: step(m, z(2, 40), (None, z(2, 64, 3))), lambda: step(m, z(2, 32), (None, z(1, 64, 3))),
                    lambda: step(m, z(2, 32), (z(1, 64, 16), z(2, 64, 3))), lambda: mamba.causal_conv1d_silu(z(2, 20, 32), z(16, 1, 4)),
                    lambda: mamba.conv_step_fn(z(2, 32), z(2, 32, 3), z(16, 1, 4), None)):
            with pytest.raises(RuntimeError):
                bad()


@pytest.mark.parametrize("what", ["block", "both", "rms_norm", "add_rms_norm", "conv", "scan", "pscan"])
@pytest.mark.parametrize("grad", [False, True])
def test_tangents_are_refused(what, grad):
    """None of these has a forward-mode derivative: a tangent is an error and not lost."""
    import torch.autograd.forward_ad as fw
    import mamba_b200
    from mamba_b200 import mamba, vim
    r = lambda *s: torch.randn(*s, device=DEV)
    block, both, B = _build(32, 16, False), _build(32, 16, True), r(2, 20, 16)
    call = {"block": lambda x: mamba.forward(block, x), "both": lambda x: vim.forward(both, x), "rms_norm": lambda x: mamba.rms_norm(x, r(32)),
            "add_rms_norm": lambda x: mamba.add_rms_norm(r(2, 20, 32), x, r(32)), "conv": lambda x: mamba.causal_conv1d_silu(x, r(32, 1, 4)),
            "scan": lambda x: mamba_b200.selective_scan_fn(r(2, 20, 32), x, -torch.ones(32, 16, device=DEV), B, B),
            "pscan": lambda x: mamba_b200.pscan(x[..., None], x[..., None])}[what]
    call(r(2, 20, 32))
    with fw.dual_level(), torch.set_grad_enabled(grad), pytest.raises(NotImplementedError):
        call(fw.make_dual(r(2, 20, 32), r(2, 20, 32)))


def test_last_residual_add_keeps_a_tangent():
    import torch.autograd.forward_ad as fw
    from mamba_b200 import _lib
    x, s, t = (torch.randn(2, 20, 32, device=DEV) for _ in range(3))
    with fw.dual_level():
        assert torch.equal(fw.unpack_dual(_lib.host().add_residual(x.bfloat16(), fw.make_dual(s, t))).tangent, t)
