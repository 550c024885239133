"""Drop-in for the bidirectional block of the reference's Vision Mamba (mambapy/vim.py:205-261).

The reference runs its second direction as flip(xz) -> conv -> projections -> scan -> flip(y).  Here
the second scan walks the ORIGINAL sequence from its last timestep to its first inside the kernels
(`selective_scan_fn(..., reverse=True)`), gated by the un-flipped z, and the convolution kernel takes the rows
backwards through a negative stride; nothing is flipped or copied.  Blocks the fused interior cannot take (other
d_state, activations off the 16-byte grid) flip the convolution input as the reference does.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from ._lib import host as _host
from .mamba import causal_conv1d_silu, run_block, selective_scan_fn


def _conv_silu(conv, xs, L):
    if conv.weight.shape[-1] == 4:
        return causal_conv1d_silu(xs, conv.weight, conv.bias)
    return F.silu(conv(xs.transpose(1, 2))[:, :, :L].transpose(1, 2))


def _ssm(self, x, z, A_log, D, x_proj, dt_proj, reverse):
    """mambapy/vim.py:263-299 with softplus(delta + bias), the scan and the gate in one kernel."""
    cfg = self.config
    A = -torch.exp(A_log.float())
    delta, B, C = torch.split(x_proj(x), [cfg.dt_rank, cfg.d_state, cfg.d_state], dim=-1)
    delta, B, C = self._apply_layernorms(delta, B, C)
    delta = F.linear(delta, dt_proj.weight)
    return selective_scan_fn(x, delta, A, B, C, D, z=z, delta_bias=dt_proj.bias, reverse=reverse)


def forward(self, x):
    """mambapy/vim.py:205-261; x: (B, L, D) -> (B, L, D)."""
    _, L, _ = x.shape
    cfg = self.config
    conv, x_proj, dt_proj = self.conv1d, self.x_proj, self.dt_proj
    directions = [[conv.weight, conv.bias, x_proj.weight, dt_proj.weight, dt_proj.bias, self.A_log, self.D]]
    called = [x_proj]                                     # as modules, unless calling them is no more than the product
    native = True
    if cfg.bidirectional:
        dtype = torch.get_autocast_dtype("cuda") if torch.is_autocast_enabled("cuda") else x.dtype
        conv, x_proj, dt_proj = self.conv1d_b, self.x_proj_b, self.dt_proj_b
        directions.append([conv.weight, conv.bias, x_proj.weight, dt_proj.weight, dt_proj.bias, self.A_log_b, self.D_b])
        called.append(x_proj)
        native = _host().reversible(directions[1][6].shape[0], cfg.d_state, dtype) and conv.weight.shape[-1] == 4
    # without a bias of dt_proj the scan takes delta as it is
    if native and all(d[4] is not None for d in directions):
        out, xz = run_block(self, x, directions, cfg.bidirectional and cfg.divide_output, called)
        if out is not None:
            return out
    else:
        xz = self.in_proj(x)
    xs, z = xz.chunk(2, dim=-1)
    y = _ssm(self, _conv_silu(self.conv1d, xs, L), z, self.A_log, self.D, self.x_proj, self.dt_proj, False)
    if not cfg.bidirectional:
        return self.out_proj(y)
    # second direction: the reference convolves the flipped sequence; in original time order that is
    # flip(conv(flip(x))).  Everything after it is per-timestep, and the scan runs right to left.
    xb = _conv_silu(self.conv1d_b, xs.flip(1), L).flip(1)
    yb = _ssm(self, xb, z, self.A_log_b, self.D_b, self.x_proj_b, self.dt_proj_b, True)
    s = y + yb
    return self.out_proj(s / 2 if cfg.divide_output else s)
