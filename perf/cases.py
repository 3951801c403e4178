"""The work users of this package have it do, as cases that can be timed: single quantised projections, decode and
prefill through Llama MLP blocks, plain W2A8 GEMMs on ready-made int8 activations, and loading a float weight.

Every case goes through the public entry points (``W2A8Linear``, ``W2A8LlamaMLP``, ``W2A8Plan.gemm``, the functional
``w2a8_gemm``).  Kinds:

  linear  `layers` projections of one shape, each on its own float activations (quantised inside the call)
  mlp     `layers` Llama MLP blocks, each on its own float activations
  gemm    `layers` GEMMs on int8 activations and per-token scales; `api` says whether through a kept plan or the
          functional op
  load    one float weight quantised and packed on the GPU, the plan made, and a first projection through it

`layers` > 1 stands for the layers a decode step passes through: each weight matrix is read once per step, so together
they exceed the L2 cache and come from HBM, as they do in a model.
"""
from __future__ import annotations

import math

import torch

from slimkernels_b200.torch import W2A8Linear, W2A8LlamaMLP, W2A8Plan, w2a8_gemm

_DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}


def _case(kind, **kw):
    base = {"kind": kind, "layers": 1, "group": 128, "zero_point": 1, "dtype": "f16", "api": "plan"}
    base.update(kw)
    return base


def listed():
    return [
        # one token through one attention output projection of Llama-2-7B: the smallest call a model makes
        _case("linear", name="linear_m1_4096x4096", M=1, N=4096, K=4096),
        # a batch of 16 sequences decoding with bf16 activations: the fused QKV projections of 12 layers
        _case("linear", name="linear_m16_qkv_bf16", M=16, N=12288, K=4096, layers=12, dtype="bf16"),
        # a small batch decoding through the widest projection of Llama-3-70B, called as the functional op
        _case("gemm", name="gemm_m8_gate_up_70b", M=8, N=57344, K=8192, api="op"),
        # single-sequence decode: the MLP blocks of 8 layers of Llama-2-7B
        _case("mlp", name="mlp_m1_7b", M=1, hidden=4096, inter=11008, layers=8),
        # the same with a batch that is no power of two
        _case("mlp", name="mlp_m24_7b", M=24, hidden=4096, inter=11008, layers=8),
        # a large decode batch (or a short prompt) through the down projections of 8 layers
        _case("linear", name="linear_m96_down", M=96, N=4096, K=11008, layers=8),
        # ragged in every dimension, group size 64, zero point 2, bf16 results: a weight that is no tuned shape
        _case("gemm", name="gemm_m333_ragged_g64", M=333, N=5000, K=4160, group=64, zero_point=2, dtype="bf16"),
        # a chunk of a prompt through two MLP blocks
        _case("mlp", name="mlp_m512_7b", M=512, hidden=4096, inter=11008, layers=2),
        # a full prompt through one MLP block
        _case("mlp", name="mlp_m4096_7b", M=4096, hidden=4096, inter=11008),
        # square prefill GEMM whose tiles do not fill a whole number of waves
        _case("gemm", name="gemm_m2048_8192", M=2048, N=8192, K=8192),
        # the largest: a 4096-token prompt through the gate+up projection of Llama-3-70B
        _case("gemm", name="gemm_m4096_gate_up_70b", M=4096, N=57344, K=8192),
        # loading a checkpoint: one fp16 projection quantised, packed, planned and used for the first time
        _case("load", name="load_11008x4096", M=1, N=11008, K=4096),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "gemm", "gemm", "mlp", "load"])
    group = rng.choice([128, 128, 128, 64, 32, 256])
    dtype = rng.choice(["f16", "bf16"])
    M = _log_int(rng, 1, 4096)
    K = group * _log_int(rng, max(1, 512 // group), 16384 // group)
    if kind == "mlp":
        inter = group * _log_int(rng, max(1, 1024 // group), 14336 // group)
        hidden = min(K, group * (8192 // group))
        return _case("mlp", M=M, hidden=hidden, inter=inter, group=group, dtype=dtype, layers=rng.randint(1, 4) if M <= 64 else 1)
    N = _log_int(rng, 256, 16384)
    if rng.random() < 0.6:
        N = max(128, N // 128 * 128)
    if kind == "load":
        return _case("load", M=rng.randint(1, 16), N=N, K=K, group=group, dtype=dtype)
    layers = rng.randint(1, 8) if M <= 128 else 1
    if kind == "linear":
        return _case("linear", M=M, N=N, K=K, group=group, dtype=dtype, layers=layers)
    return _case("gemm", M=M, N=N, K=K, group=group, dtype=dtype, layers=layers, zero_point=rng.choice([1, 1, 2]),
                 api=rng.choice(["plan", "op"]))


# --------------------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _float_weight(g, N, K, std):
    return torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32).mul_(std)


def _linear(g, N, K, case, std=None, out_dtype=None):
    w = _float_weight(g, N, K, K ** -0.5 if std is None else std)
    lin = W2A8Linear.from_float(w, case["group"], out_dtype=out_dtype or _DTYPES[case["dtype"]])
    lin.plan()
    return lin


def prepare(case, seed):
    g = _generator(seed)
    kind, M, L, dt = case["kind"], case["M"], case["layers"], _DTYPES[case["dtype"]]
    if kind == "linear":
        lins = [_linear(g, case["N"], case["K"], case) for _ in range(L)]
        xs = [torch.randn(M, case["K"], generator=g, device="cuda").to(dt) for _ in range(L)]
        return {"kind": kind, "layers": lins, "xs": xs}
    if kind == "mlp":
        hidden, inter = case["hidden"], case["inter"]
        # (SiLU(gate) * up of unit normals has a standard deviation of about 0.6; between blocks a model normalises)
        blocks = [W2A8LlamaMLP(_linear(g, 2 * inter, hidden, case, out_dtype=torch.float16),
                               _linear(g, hidden, inter, case, std=1.5 * inter ** -0.5)) for _ in range(L)]
        xs = [torch.randn(M, hidden, generator=g, device="cuda").to(dt) for _ in range(L)]
        return {"kind": kind, "blocks": blocks, "xs": xs}
    if kind == "gemm":
        N, K, G = case["N"], case["K"], case["group"]
        plans, weights, acts = [], [], []
        for _ in range(L):
            w = torch.randint(0, 256, (N, K // 4), generator=g, device="cuda", dtype=torch.uint8)
            s = torch.empty(K // G, N, device="cuda").uniform_(0.001, 0.01, generator=g).to(torch.float16)
            x = torch.randint(-127, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
            xs = torch.empty(M, device="cuda").uniform_(0.005, 0.02, generator=g)
            acts.append((x, xs))
            weights.append((w, s))
            if case["api"] == "plan":
                plans.append(W2A8Plan(w, s, group_size=G, zero_point=case["zero_point"], out_dtype=dt))
        return {"kind": kind, "api": case["api"], "plans": plans, "weights": weights, "acts": acts,
                "group": G, "zero_point": case["zero_point"], "dtype": dt}
    assert kind == "load"
    return {"kind": kind, "w": _float_weight(g, case["N"], case["K"], case["K"] ** -0.5).to(dt), "group": case["group"],
            "x": torch.randn(M, case["K"], generator=g, device="cuda").to(dt), "dtype": dt}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return [lin(x) for lin, x in zip(state["layers"], state["xs"])]
    if kind == "mlp":
        return [block(x) for block, x in zip(state["blocks"], state["xs"])]
    if kind == "gemm":
        if state["api"] == "plan":
            return [plan.gemm(x, xs) for plan, (x, xs) in zip(state["plans"], state["acts"])]
        return [w2a8_gemm(x, xs, w, s, state["group"], state["zero_point"], state["dtype"])
                for (x, xs), (w, s) in zip(state["acts"], state["weights"])]
    lin = W2A8Linear.from_float(state["w"], state["group"], out_dtype=state["dtype"])
    y = lin(state["x"])
    return {"w_packed": lin.w_packed, "w_scale": lin.w_scale, "y": y}


def _gemm_work(M, N, K, G, x_bytes):
    """(bytes, operations) of one projection: packed weights and fp16 scales, the activations, the 16-bit results."""
    return N * K // 4 + (K // G) * N * 2 + M * K * x_bytes + M * N * 2, 2 * M * N * K


def work(case):
    M, G, L = case["M"], case["group"], case["layers"]
    if case["kind"] == "mlp":
        b1, f1 = _gemm_work(M, 2 * case["inter"], case["hidden"], G, 2)
        b2, f2 = _gemm_work(M, case["hidden"], case["inter"], G, 0)
        return {"bytes": L * (b1 - M * 2 * case["inter"] * 2 + b2), "flops": L * (f1 + f2)}
    if case["kind"] == "load":
        b, f = _gemm_work(M, case["N"], case["K"], G, 2)
        return {"bytes": b + case["N"] * case["K"] * 2, "flops": f}
    b, f = _gemm_work(M, case["N"], case["K"], G, 1 if case["kind"] == "gemm" else 2)
    return {"bytes": L * (b + (4 * M if case["kind"] == "gemm" else 0)), "flops": L * f}


def tolerance(case):
    # four times what was measured against 64-bit arithmetic on the same quantised operands
    if case["kind"] == "mlp":
        # 5e-3 .. 1.3e-2: rounding gate and up to fp16, and the first sums, move int8 codes of the hidden activations
        return {"rel": 4e-2, "max": 0.25}
    if case["kind"] == "gemm":
        # 2e-4 .. 3.4e-4 with fp16 results, 1.7e-3 with bf16 results
        return {"rel": 1.5e-3 if case["dtype"] == "f16" else 7e-3, "max": 0.02}
    # sums of normally distributed products cancel: 4e-4 .. 2.4e-3 with fp16 results, 1.7e-3 .. 2.9e-3 with bf16 results
    return {"rel": 1e-2, "max": 0.06}


# --------------------------------------------------------------------------------------------------------------
# The same in 64 bits.  The integer codes of weights and activations are the format itself (their rule is defined in
# fp32, as are the token scales; group scales are stored as fp16); sums, SiLU and scaling are float64.
def _codes_of(w, group):
    """Codes - 1 [N, K] in -1..2 and the stored fp16 scales [K/G, N] of a float weight [N, K]."""
    N, K = w.shape
    g = w.float().view(N, K // group, group)
    scale = (g.abs().amax(dim=2).clamp_min(1e-9).double() / 1.5).float()
    codes = torch.round(g / scale[:, :, None]).clamp_(-1, 2)
    return codes.view(N, K), scale.t().to(torch.float16).contiguous()


def _unpacked(w_packed, zero_point):
    shifts = torch.tensor([6, 4, 2, 0], device=w_packed.device, dtype=torch.uint8)
    return ((w_packed[:, :, None] >> shifts) & 3).view(w_packed.shape[0], -1).to(torch.float32) - zero_point


def _quantized(x):
    """Codes and scales of activations; the scale's and the quotient's rule is fp32."""
    x = x.float()
    s = (x.abs().amax(dim=1).double() / 127).float()
    s = torch.where(s > 0, s, torch.ones_like(s))
    return torch.round(x / s[:, None]).clamp_(-127, 127), s


def _product(x_q, x_scale, codes, w_scale, group, columns=4096):
    """float64 x_scale * sum over groups of w_scale * (x_q . codes), a block of output features at a time."""
    xd = x_q.double()
    out = []
    for lo in range(0, codes.shape[0], columns):
        c = codes[lo:lo + columns].double()
        c = c * w_scale[:, lo:lo + columns].t().double().repeat_interleave(group, dim=1)
        out.append(xd @ c.t())
    return torch.cat(out, dim=1) * x_scale.double()[:, None]


def exact(case, seed):
    """What `run` returns, in float64 (None for the packed bytes of `load`, which are whole values)."""
    g = _generator(seed)
    kind, M, L, dt, G = case["kind"], case["M"], case["layers"], _DTYPES[case["dtype"]], case["group"]

    def weight(N, K, std=None):
        return _codes_of(_float_weight(g, N, K, K ** -0.5 if std is None else std), G)

    def activations(K):
        return _quantized(torch.randn(M, K, generator=g, device="cuda").to(dt).to(torch.float16))

    if kind == "linear":
        weights = [weight(case["N"], case["K"]) for _ in range(L)]
        return [_product(*activations(case["K"]), *w, G) for w in weights]
    if kind == "mlp":
        hidden, inter = case["hidden"], case["inter"]
        weights = [(weight(2 * inter, hidden), weight(hidden, inter, 1.5 * inter ** -0.5)) for _ in range(L)]
        out = []
        for gate_up, down in weights:
            gu = _product(*activations(hidden), *gate_up, G)
            h = torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]
            out.append(_product(*_quantized(h), *down, G))
        return out
    if kind == "gemm":
        N, K, out = case["N"], case["K"], []
        for _ in range(L):
            w = torch.randint(0, 256, (N, K // 4), generator=g, device="cuda", dtype=torch.uint8)
            s = torch.empty(K // G, N, device="cuda").uniform_(0.001, 0.01, generator=g).to(torch.float16)
            x = torch.randint(-127, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
            xs = torch.empty(M, device="cuda").uniform_(0.005, 0.02, generator=g)
            out.append(_product(x, xs, _unpacked(w, case["zero_point"]), s, G))
        return out
    codes, scale = _codes_of(_float_weight(g, case["N"], case["K"], case["K"] ** -0.5).to(dt), G)
    return {"w_packed": None, "w_scale": scale.double(), "y": _product(*activations(case["K"]), codes, scale, G)}
