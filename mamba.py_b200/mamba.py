"""Drop-ins for the scan methods of the reference's MambaBlock (mambapy/mamba.py).

The functions below take `self` first so they can be bound onto the reference's MambaBlock
(see `mamba_b200.install`) or onto any object with the same attribute names:

    selective_scan(self, x, delta, A, B, C, D)      mambapy/mamba.py:274-295
    selective_scan_seq(self, x, delta, A, B, C, D)  mambapy/mamba.py:297-327 (same kernel)
    ssm_step(self, x, h)                            mambapy/mamba.py:384-414
    step(self, x, cache)                            mambapy/mamba.py:351-382
    ssm(self, x, z) / forward(self, x)              mambapy/mamba.py:236-272 / :205-234 with the
                                                    softplus, the scan and the gate in one kernel

`selective_scan_fn` is the functional form with the optional gate `z`, the fused
`softplus(delta + delta_bias)`, an incoming state `h0` and the outgoing state.
Everything runs in libmamba_b200.so on CUDA tensors; there is no CPU path.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F
from torch import nn
from torch.nn.modules.module import _has_any_global_hook

from ._lib import host as _host
from .kernels import sscan_fwd_raw, sscan_bwd_raw  # noqa: F401  (re-exported)


def selective_scan_fn(x, delta, A, B, C, D=None, z=None, delta_bias=None, h0=None,
                      return_last_state=False, reverse=False, subshards=None):
    """Fused selective scan.

    x, delta, z : (B, L, ED)   B, C : (B, L, N)   A : (ED, N)   D : (ED)
    With `delta_bias` the kernel applies delta = softplus(delta + delta_bias) itself (the
    contract of the fused seam at mambapy/mamba.py:260); with `z` it also applies the
    y * silu(z) gate (mambapy/mamba.py:229-231).  Returns y (B, L, ED), plus the final state
    (B, ED, N) float32 when `return_last_state`.

    `reverse=True` scans from the last timestep to the first (h0 enters at t = L-1, the returned state
    leaves t = 0): the second direction of the reference's bidirectional model, which flips the
    sequence, scans and flips back (mambapy/vim.py:228-261).  The kernels do it in place when the
    tensors meet the tensor-map alignment rules (and d_state is 16 if gradients are needed);
    otherwise this function flips, as the reference does.

    With few batch rows the sequence is cut into `subshards` consecutive pieces that are scanned side by
    side (two extra carry passes, see split.py): None picks the number from the shape, 1 never cuts, any
    other value is used if L is a multiple of 16 * subshards.
    """
    return _host().selective_scan(x, delta, A, B, C, D, z, delta_bias, h0, return_last_state, reverse, subshards)


# ----------------------------------------------------------------- MambaBlock method drop-ins

def selective_scan(self, x, delta, A, B, C, D):
    """mambapy/mamba.py:274-295.  x, delta: (B, L, ED); A: (ED, N); B, C: (B, L, N); D: (ED)."""
    return selective_scan_fn(x, delta, A, B, C, D)


def selective_scan_seq(self, x, delta, A, B, C, D):
    """mambapy/mamba.py:297-327.  The sequential variant computes the same y; same kernel."""
    return selective_scan_fn(x, delta, A, B, C, D)


def ssm_step_fn(x, h, delta, A, B, C, D=None, z=None, delta_bias=None, inplace=False):
    """One decode step on projected inputs.  x, delta, z: (B, ED); B, C: (B, N); h: (B, ED, N) or None.

    Returns (y, h_new); h_new is a fresh float32 tensor (the reference also returns a new one,
    mambapy/mamba.py:408).  `inplace=True` (opt-in, for decode loops that own their cache)
    overwrites a float32 contiguous `h` instead and returns it."""
    return _host().ssm_step(x, h, delta, A, B, C, D, z, delta_bias, inplace)


def conv_step_fn(x, inputs, weight, bias, inplace=False):
    """Conv-window part of a decode step (mambapy/mamba.py:366-369, :379).

    x: (B, ED) new pre-conv input; inputs: (B, ED, d_conv-1) cached window;
    weight: (ED, 1, d_conv) depthwise filter; bias: (ED) or None.
    Returns (silu(conv(x)), new window).  The window is a fresh tensor unless `inplace=True`
    (opt-in), which shifts a contiguous window of the activation dtype in place."""
    return _host().conv_step(x, inputs, weight, bias, inplace)


def causal_conv1d_silu(x, weight, bias=None):
    """silu(conv1d(x)) of MambaBlock.forward (mambapy/mamba.py:217-221) without the transposes.

    x: (B, L, ED); weight: (ED, 1, 4) as nn.Conv1d(groups=ED) holds it; bias: (ED) or None."""
    return _host().conv1d_silu(x, weight, bias)


def rms_norm(x, weight=None, eps=1e-5):
    """RMSNorm over the last dimension; weight None is the reference's muP variant (no gain)."""
    return _host().rms_norm(x, weight, eps)


def add_rms_norm(x, residual=None, weight=None, eps=1e-5):
    """s = x + residual (residual None: s = x); y = RMSNorm(s).  Returns (y, s) from ONE pass over the data:
    the residual add of one layer fused with the normalisation in front of the next
    (mambapy/mamba.py:106-112).  Under autocast y comes out in the autocast dtype, which is what the
    projection that consumes it would cast it to anyway."""
    return _host().add_rms_norm(x, residual, weight, eps)


def stack_forward(self, x):
    """Drop-in for Mamba.forward (mambapy/mamba.py:77-85): the loop over ResidualBlocks
    (`x = mixer(norm(x)) + x`, mambapy/mamba.py:106-112) with each layer's residual add fused into the
    next layer's RMSNorm; the last add is an ordinary add."""
    h, res = x, None
    for layer in self.layers:
        norm = layer.norm
        normed, res = add_rms_norm(h, res, None if getattr(norm, "use_mup", False) else norm.weight, norm.eps)
        h = layer.mixer(normed)
    return _host().add_residual(h, res) if res is not None else h


def rmsnorm_forward(self, x):
    """Drop-in for RMSNorm.forward (mambapy/mamba.py:427-433)."""
    return rms_norm(x, None if getattr(self, "use_mup", False) else self.weight, self.eps)


def _project(self, x):
    """delta (pre-softplus, without bias), B, C from x as in mambapy/mamba.py:393-396."""
    cfg = self.config
    deltaBC = self.x_proj(x)
    delta, B, C = torch.split(deltaBC, [cfg.dt_rank, cfg.d_state, cfg.d_state], dim=-1)
    delta, B, C = self._apply_layernorms(delta, B, C)
    return delta, B, C


def ssm_step(self, x, h):
    """mambapy/mamba.py:384-414.  x: (B, ED); h: (B, ED, N) or None.  Returns (y, h)."""
    A = -torch.exp(self.A_log.float())
    delta, B, C = _project(self, x)
    delta = F.linear(delta, self.dt_proj.weight)          # bias and softplus happen in the kernel
    return ssm_step_fn(x, h, delta, A, B, C, self.D, delta_bias=self.dt_proj.bias)


def step(self, x, cache):
    """mambapy/mamba.py:351-382.  x: (B, D); cache = (h (B, ED, N) or None, inputs (B, ED, d_conv-1)).

    Returns (output (B, D), (h, inputs)) with fresh cache tensors."""
    h, inputs = cache
    p = _plain_block(self)
    if p is not None:
        cfg = self.config
        out, h, inputs = _host().block_step(x, h, inputs, *p, cfg.dt_rank, cfg.d_state)
        return out, (h, inputs)
    xz = self.in_proj(x)
    xs, z = xz.chunk(2, dim=1)
    xc, inputs = conv_step_fn(xs, inputs, self.conv1d.weight, self.conv1d.bias)
    A = -torch.exp(self.A_log.float())
    delta, B, C = _project(self, xc)
    delta = F.linear(delta, self.dt_proj.weight)
    y, h = ssm_step_fn(xc, h, delta, A, B, C, self.D, z=z, delta_bias=self.dt_proj.bias)
    return self.out_proj(y), (h, inputs)


_Linear, _linear_forward = nn.Linear, nn.Linear.forward


def _plain_linear(m):
    """(weight, bias) of a projection that is an ordinary nn.Linear and nothing else, so that calling it is the matrix product: no
    subclass, no hook of any kind, no `forward` of its own (offload and dispatch wrappers put theirs on the instance), not compiled
    by itself, and an ordinary tensor as its weight (quantised and distributed ones dispatch for themselves) among its parameters
    (replicas and pruning keep theirs as plain attributes)."""
    if type(m) is not _Linear or _Linear.forward is not _linear_forward:
        return None
    d = m.__dict__
    if (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or "forward" in d
            or d.get("_compiled_call_impl") is not None):
        return None
    p = d["_parameters"]
    w = p.get("weight")
    if not (type(w) is nn.Parameter or type(w) is torch.Tensor) or "bias" not in p:
        return None
    return w, p["bias"]


def _plain_block(self):
    """The block's tensors in the order the native step takes them, or None if any part of it has been replaced, hooked or
    extended (layer norms on dt, B, C) and has to be called as the module it is."""
    d = self.__dict__
    mods, pars = d.get("_modules"), d.get("_parameters")
    if not mods or _has_any_global_hook() or not (mods.get("dt_layernorm") is mods.get("B_layernorm") is mods.get("C_layernorm") is None):
        return None
    lin = [_plain_linear(mods.get(k)) for k in ("in_proj", "x_proj", "dt_proj", "out_proj")]
    conv, A_log, D = mods.get("conv1d"), pars.get("A_log"), pars.get("D")
    if any(p is None for p in lin) or conv is None or A_log is None or D is None or lin[1][1] is not None or lin[2][1] is None:
        return None
    if self.config.d_state not in (8, 16, 32, 64):
        return None
    conv = conv._parameters
    if conv.get("weight") is None or "bias" not in conv:
        return None
    return *lin[0], conv["weight"], conv["bias"], lin[1][0], *lin[2], A_log, D, *lin[3]


def _fusable(self, x, dtype):
    """Whether the native block takes this module on activations of `dtype` made from x."""
    cfg = self.config
    return (x.is_cuda and dtype in (torch.float32, torch.bfloat16) and self.conv1d.weight.shape[-1] == 4
            and getattr(self, "dt_layernorm", None) is None and getattr(self, "B_layernorm", None) is None
            and getattr(self, "C_layernorm", None) is None and cfg.d_state in (8, 16, 32, 64))


def _native_linear(m, dtype, amp):
    """The weight of a projection the native block can run itself on activations of `dtype`: an ordinary nn.Linear without
    a bias, of the activations' type or cast to it by autocast.  None for any other, which is called as the module it is."""
    p = _plain_linear(m)
    if p is None or p[1] is not None:
        return None
    w = p[0]
    return w if w.is_cuda and (w.dtype == dtype or (amp and w.dtype in (torch.float32, torch.bfloat16))) else None


def run_block(self, x, directions, halve=False, called=()):
    """in_proj, the scans of `directions` (lists of seven parameters) and out_proj as one native call, with those projections
    called as modules that are not ordinary ones.  None if the block does not take the native path, as it does not when one of
    `called`, projections whose weights are among the parameters, has to be called; the second value is in_proj(x) if that has been
    computed on the way."""
    amp = torch.is_autocast_enabled("cuda")
    dtype = torch.get_autocast_dtype("cuda") if amp else x.dtype
    own = not _has_any_global_hook()
    in_w = _native_linear(self.in_proj, dtype, amp) if own and x.dim() == 3 and x.dtype in (torch.float32, torch.bfloat16) else None
    if in_w is None or not _fusable(self, x, dtype):
        x, in_w = self.in_proj(x), None
        dtype = x.dtype
        if not _fusable(self, x, dtype):
            return None, x
    for m in called:
        if not own or _native_linear(m, dtype, amp) is None:
            return None, x if in_w is None else self.in_proj(x)
    cfg = self.config
    params = [p for d in directions for p in d]
    out_w = _native_linear(self.out_proj, dtype, amp) if own else None
    if out_w is not None:
        return _host().block(x, in_w, out_w, params, cfg.dt_rank, cfg.d_state, halve), None
    y = _host().block(x, in_w, None, params, cfg.dt_rank, cfg.d_state, False)
    return self.out_proj(y / 2 if halve else y), None


def ssm(self, x, z):
    """mambapy/mamba.py:236-272 with softplus(delta + dt_bias), the scan and the gate fused.

    Like the reference's own fused branch (mambapy/mamba.py:252-261) this returns the GATED y,
    so the matching `forward` below skips the z branch."""
    A = -torch.exp(self.A_log.float())
    delta, B, C = _project(self, x)
    delta = F.linear(delta, self.dt_proj.weight)          # (B, L, ED), no transposes needed
    return selective_scan_fn(x, delta, A, B, C, self.D, z=z, delta_bias=self.dt_proj.bias)


def forward(self, x):
    """mambapy/mamba.py:205-234 with the scan path fused; x: (B, L, D) -> (B, L, D)."""
    _, L, _ = x.shape
    out, xz = run_block(self, x, [[self.conv1d.weight, self.conv1d.bias, self.x_proj.weight, self.dt_proj.weight,
                                   self.dt_proj.bias, self.A_log, self.D]])
    if out is not None:
        return out
    xs, z = xz.chunk(2, dim=-1)
    if self.conv1d.weight.shape[-1] == 4:
        xs = causal_conv1d_silu(xs, self.conv1d.weight, self.conv1d.bias)
    else:
        xs = F.silu(self.conv1d(xs.transpose(1, 2))[:, :, :L].transpose(1, 2))
    y = ssm(self, xs, z)
    return self.out_proj(y)
