"""The work a user of this package has it do, as a list of cases that can be timed.

Every case goes through the public entry points (`selective_scan_fn`, `pscan`, `mamba.step`,
`mamba.stack_forward`, `vim.forward`, `rms_norm`), the way the reference's own classes reach them once
`install()` has run.  Four kinds of case:

  scan     the fused selective scan on a layer's tensors: training (forward and every gradient) or prefill
           (forward under no_grad with the state handed to the decoder)
  pscan    the PScan operator on (B, L, D, N) tensors, forward and both gradients
  decode   one token for a batch through a stack of layers: norm, `step` with its caches, residual add
  stack    whole layers over a sequence: training under autocast or in float32, prefill, and the
           bidirectional block

d_state is 16 and d_conv 4 everywhere, as in every configuration this repository names.
"""
import contextlib
import math
import types

import torch
import torch.nn.functional as F
from torch import nn

import mamba_b200
from mamba_b200 import mamba as layers
from mamba_b200 import vim

N, K = 16, 4
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def listed():
    return [
        # The layer scan of a 130m model in training: batch 8 of 2048 tokens, bfloat16 activations, freshly
        # initialised A (the package's headline benchmark).
        {"name": "scan_train_130m", "kind": "scan", "batch": 8, "length": 2048, "d_inner": 1536, "dtype": "bf16",
         "train": True, "softplus": True, "trained_A": False},
        # One very long sequence of a wide layer, delta already through its softplus (the long-sequence config).
        {"name": "scan_train_long", "kind": "scan", "batch": 1, "length": 131072, "d_inner": 5120, "dtype": "bf16",
         "train": True, "softplus": False, "trained_A": False},
        # Fine-tuning a trained model in float32 on a batch of ragged length and an uneven width.
        {"name": "scan_train_ragged_f32", "kind": "scan", "batch": 3, "length": 1003, "d_inner": 1000, "dtype": "f32",
         "train": True, "softplus": True, "trained_A": True},
        # The small float32 layer of the CPU config: a call whose kernels take no time.
        {"name": "scan_train_tiny_f32", "kind": "scan", "batch": 2, "length": 64, "d_inner": 32, "dtype": "f32",
         "train": True, "softplus": False, "trained_A": False},
        # Reading one prompt into the state of a trained 2.8b-shaped layer before decoding.
        {"name": "scan_prefill", "kind": "scan", "batch": 1, "length": 1777, "d_inner": 5120, "dtype": "bf16",
         "train": False, "softplus": True, "trained_A": True},
        # The PScan operator at its benchmark size, and at a size that an unpatched block of a small model uses.
        {"name": "pscan_large", "kind": "pscan", "batch": 16, "length": 2048, "d_inner": 1536, "dtype": "f32"},
        {"name": "pscan_small", "kind": "pscan", "batch": 1, "length": 1000, "d_inner": 128, "dtype": "f32"},
        # Decoding one stream with a 130m-shaped model, float32 as the reference loads it: one layer.
        {"name": "decode_one_stream", "kind": "decode", "batch": 1, "d_model": 768, "layers": 1, "dtype": "f32"},
        # Batched decoding with the 2.8b shape: four of its layers, so that their states do not fit the L2.
        {"name": "decode_2p8b_batch", "kind": "decode", "batch": 256, "d_model": 2560, "layers": 4, "dtype": "bf16"},
        # Training two whole layers of the 130m shape under bfloat16 autocast: norms, projections, conv and scan.
        {"name": "stack_train_130m", "kind": "stack", "batch": 8, "length": 2048, "d_model": 768, "layers": 2,
         "dtype": "bf16", "train": True, "bidirectional": False},
        # Training a toy model in float32 (the reference's examples): launches and host work only.
        {"name": "stack_train_small_f32", "kind": "stack", "batch": 2, "length": 61, "d_model": 64, "layers": 2,
         "dtype": "f32", "train": True, "bidirectional": False},
        # A bidirectional block over image patches: many short rows, both directions.
        {"name": "bidirectional_train", "kind": "stack", "batch": 64, "length": 197, "d_model": 192, "layers": 1,
         "dtype": "bf16", "train": True, "bidirectional": True},
    ]


def _log(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("scan", "scan", "scan", "pscan", "decode", "stack", "stack"))
    if kind == "scan":
        dtype = rng.choice(("bf16", "bf16", "f32"))
        while True:
            width = 32 * _log(rng, 1, 160)                    # twice a d_model that is a multiple of 16
            batch, length = _log(rng, 1, 64), _log(rng, 33, 131072)
            if batch * length * max(width, 2048) <= 131072 * 5120 // (1 if dtype == "bf16" else 2):
                break
        return {"kind": kind, "batch": batch, "length": length, "d_inner": width, "dtype": dtype,
                "train": rng.random() < 0.7, "softplus": rng.random() < 0.8, "trained_A": rng.random() < 0.5}
    if kind == "pscan":
        while True:
            batch, length, width = _log(rng, 1, 32), _log(rng, 33, 8192), 2 * _log(rng, 8, 1280)
            if batch * length * width <= 16 * 2048 * 1536:
                break
        return {"kind": kind, "batch": batch, "length": length, "d_inner": width, "dtype": "f32"}
    if kind == "decode":
        return {"kind": kind, "batch": _log(rng, 1, 256), "d_model": 64 * _log(rng, 1, 40), "layers": rng.choice((1, 2, 4)),
                "dtype": rng.choice(("bf16", "f32"))}
    bidirectional = rng.random() < 0.3
    while True:
        d_model = 64 * _log(rng, 1, 24)
        batch, length = _log(rng, 1, 64), _log(rng, 33, 8192)
        if batch * length * d_model <= 8 * 2048 * 768:
            break
    return {"kind": kind, "batch": batch, "length": length, "d_model": d_model, "layers": 1 if bidirectional else rng.choice((1, 2)),
            "dtype": rng.choice(("bf16", "f32")), "train": rng.random() < 0.7, "bidirectional": bidirectional}


# ------------------------------------------------------------------------------------ inputs

def _dt_bias(width, gen):
    """Inverse softplus of dt ~ log-uniform [1e-3, 1e-1], the reference's initialisation."""
    dt = torch.exp(torch.rand(width, generator=gen, device="cuda") * math.log(100.0) + math.log(1e-3))
    return dt + torch.log(-torch.expm1(-dt))


def _A_log(width, gen, trained):
    """log(1..N) per channel (the initialisation); a trained model's has moved away from it."""
    A_log = torch.log(torch.arange(1, N + 1, dtype=torch.float32, device="cuda")).repeat(width, 1)
    return A_log + 0.2 * torch.randn(width, N, generator=gen, device="cuda") if trained else A_log


def _prepare_scan(case, gen):
    B, L, W, dtype = case["batch"], case["length"], case["d_inner"], DTYPES[case["dtype"]]
    R = math.ceil(W / 32)
    normal = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    xz = normal(B, L, 2 * W).to(dtype)                 # in_proj's output; its second half is the gate
    x = F.silu(xz[..., :W])                            # stands for the convolution's output
    if case["softplus"]:
        delta, bias = (normal(B, L, W) * 0.5).to(dtype), _dt_bias(W, gen)
    else:
        delta, bias = F.softplus(normal(B, L, W) * 0.5 - 4.6).to(dtype), None
    dbc = normal(B, L, R + 2 * N).to(dtype)            # x_proj's output: dt, B, C side by side
    s = {"x": x, "delta": delta, "A": -torch.exp(_A_log(W, gen, case["trained_A"])), "B": dbc[..., R:R + N],
         "C": dbc[..., R + N:], "D": 1.0 + 0.1 * normal(W), "z": xz[..., W:], "delta_bias": bias}
    if case["train"]:
        s["dy"] = normal(B, L, W).to(dtype)
        for k, t in s.items():
            if t is not None and k != "dy":
                s[k] = t.detach().requires_grad_()
    return s


def _run_scan(s):
    args = (s["x"], s["delta"], s["A"], s["B"], s["C"], s["D"])
    if "dy" not in s:
        with torch.no_grad():
            return mamba_b200.selective_scan_fn(*args, z=s["z"], delta_bias=s["delta_bias"], return_last_state=True)
    y = mamba_b200.selective_scan_fn(*args, z=s["z"], delta_bias=s["delta_bias"])
    wanted = [t for k, t in s.items() if k != "dy" and t is not None]
    return y.detach(), torch.autograd.grad(y, wanted, s["dy"])


def _prepare_pscan(case, gen):
    shape = (case["batch"], case["length"], case["d_inner"], N)
    A = torch.exp(-F.softplus(torch.randn(shape, generator=gen, device="cuda")))
    X = torch.randn(shape, generator=gen, device="cuda")
    return {"A": A.requires_grad_(), "X": X.requires_grad_(), "G": torch.randn(shape, generator=gen, device="cuda")}


def _run_pscan(s):
    H = mamba_b200.pscan(s["A"], s["X"])
    return H.detach(), torch.autograd.grad(H, (s["A"], s["X"]), s["G"])


class _Norm(nn.Module):
    """Holds what the reference's RMSNorm holds."""

    def __init__(self, d_model, gen):
        super().__init__()
        self.eps, self.use_mup = 1e-5, False
        self.weight = nn.Parameter(1.0 + 0.1 * torch.randn(d_model, generator=gen, device="cuda"))

    forward = layers.rmsnorm_forward


class _Block(nn.Module):
    """The parameters of one block under the reference's names (those of the second direction end in _b)."""

    def __init__(self, d_model, gen, bidirectional=False):
        super().__init__()
        W, R = 2 * d_model, math.ceil(d_model / 16)
        self.config = types.SimpleNamespace(d_model=d_model, d_inner=W, dt_rank=R, d_state=N, d_conv=K,
                                            bidirectional=bidirectional, divide_output=True)
        self.in_proj = nn.Linear(d_model, 2 * W, bias=False, device="cuda")
        self.out_proj = nn.Linear(W, d_model, bias=False, device="cuda")
        for suffix in ("", "_b") if bidirectional else ("",):
            setattr(self, "conv1d" + suffix, nn.Conv1d(W, W, K, groups=W, padding=K - 1, device="cuda"))
            setattr(self, "x_proj" + suffix, nn.Linear(W, R + 2 * N, bias=False, device="cuda"))
            setattr(self, "dt_proj" + suffix, nn.Linear(R, W, device="cuda"))
            setattr(self, "A_log" + suffix, nn.Parameter(_A_log(W, gen, True)))
            setattr(self, "D" + suffix, nn.Parameter(1.0 + 0.1 * torch.randn(W, generator=gen, device="cuda")))
        with torch.no_grad():
            for m in self.modules():
                if isinstance(m, (nn.Linear, nn.Conv1d)):
                    bound = 1 / math.sqrt(m.weight[0].numel())
                    m.weight.uniform_(-bound, bound, generator=gen)
                if isinstance(m, nn.Conv1d):
                    m.bias.uniform_(-0.5, 0.5, generator=gen)
                elif isinstance(m, nn.Linear) and m.bias is not None:
                    m.bias.copy_(_dt_bias(W, gen))

    def _apply_layernorms(self, dt, B, C):
        return dt, B, C

    step = layers.step

    def forward(self, x):
        return vim.forward(self, x) if self.config.bidirectional else layers.forward(self, x)


class _Layer(nn.Module):
    def __init__(self, d_model, gen, bidirectional=False):
        super().__init__()
        self.norm, self.mixer = _Norm(d_model, gen), _Block(d_model, gen, bidirectional)


class _Stack(nn.Module):
    """The layer loop of the reference's Mamba, `forward` and `step`."""

    def __init__(self, n, d_model, gen, bidirectional=False):
        super().__init__()
        self.layers = nn.ModuleList(_Layer(d_model, gen, bidirectional) for _ in range(n))

    forward = layers.stack_forward

    def step(self, x, caches):
        out = []
        for layer, cache in zip(self.layers, caches):
            y, cache = layer.mixer.step(layer.norm(x), cache)
            x = y + x
            out.append(cache)
        return x, out


def _prepare_decode(case, gen):
    B, D, dtype = case["batch"], case["d_model"], DTYPES[case["dtype"]]
    model = _Stack(case["layers"], D, gen).to(dtype)
    normal = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    caches = [(normal(B, 2 * D, N), normal(B, 2 * D, K - 1).to(dtype)) for _ in range(case["layers"])]
    return {"model": model, "x": normal(B, D).to(dtype), "caches": caches}


def _run_decode(s):
    with torch.no_grad():
        return s["model"].step(s["x"], s["caches"])


def _prepare_stack(case, gen):
    shape = (case["batch"], case["length"], case["d_model"])
    model = _Stack(case["layers"], case["d_model"], gen, case["bidirectional"])
    s = {"model": model, "x": torch.randn(shape, generator=gen, device="cuda"), "autocast": case["dtype"] == "bf16"}
    if case["train"]:
        s["x"].requires_grad_()
        s["dy"] = torch.randn(shape, generator=gen, device="cuda")
        s["wanted"] = [s["x"]] + list(model.parameters())
    return s


def _run_stack(s):
    cast = torch.autocast("cuda", dtype=torch.bfloat16) if s["autocast"] else contextlib.nullcontext()
    if "dy" not in s:
        with torch.no_grad(), cast:
            return s["model"](s["x"])
    with cast:
        y = s["model"](s["x"])
    return y.detach(), torch.autograd.grad(y, s["wanted"], s["dy"].to(y.dtype))


_KINDS = {"scan": (_prepare_scan, _run_scan), "pscan": (_prepare_pscan, _run_pscan),
          "decode": (_prepare_decode, _run_decode), "stack": (_prepare_stack, _run_stack)}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return {"kind": case["kind"], **_KINDS[case["kind"]][0](case, gen)}


def run(state):
    s = {k: v for k, v in state.items() if k != "kind"}
    return _KINDS[state["kind"]][1](s)


# ------------------------------------------------------------------------------------ work and tolerance

def work(case):
    """Each input read once, each output written once.  Operations: 8 per state element of a scan forward
    (exponential, its argument, input, recurrence, contraction), 22 backward; 2 per multiply-add of a projection."""
    e = 2 if case.get("dtype") == "bf16" else 4
    if case["kind"] == "scan":
        rows, W = case["batch"] * case["length"], case["d_inner"]
        params = 4 * W * (N + 2)
        if case["train"]:
            return {"bytes": rows * (8 * W + 4 * N) * e + 2 * params, "flops": 30 * rows * W * N}
        return {"bytes": rows * (4 * W + 2 * N) * e + params + 4 * case["batch"] * W * N, "flops": 8 * rows * W * N}
    if case["kind"] == "pscan":
        n = case["batch"] * case["length"] * case["d_inner"] * N
        return {"bytes": 6 * n * 4, "flops": 5 * n}       # A, X, G in; H, gradA, gradX out
    D, R = case["d_model"], math.ceil(case["d_model"] / 16)
    W = 2 * D
    directions = 2 if case.get("bidirectional") else 1
    linear = 2 * W * D + W * D + directions * (W * (R + 2 * N) + R * W)
    other = D + directions * W * (K + N + 3)
    if case["kind"] == "decode":
        B = case["batch"]
        per = (linear + other) * e + 2 * B * W * (N * 4 + (K - 1) * e)
        return {"bytes": case["layers"] * per + 2 * B * D * e, "flops": case["layers"] * B * (2 * linear + W * (8 * N + 2 * K))}
    rows = case["batch"] * case["length"]
    scan = directions * W * N
    if case["train"]:                                     # x, dy in; y, dx out; parameters in, their gradients out
        return {"bytes": 4 * rows * D * 4 + case["layers"] * 2 * (linear + other) * 4,
                "flops": case["layers"] * rows * (6 * linear + 30 * scan)}
    return {"bytes": 2 * rows * D * 4 + case["layers"] * (linear + other) * 4, "flops": case["layers"] * rows * (2 * linear + 8 * scan)}


def tolerance(case):
    """bfloat16 activations: their own rounding.  float32: sums over up to 10^5 terms in another order, and
    exponentials of up to 2^-20 relative error fed back through the recurrence."""
    if case["kind"] == "pscan":
        return {"rel": 1e-5}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 5e-5}
