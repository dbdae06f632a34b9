"""The work a user of this library has it do, as a list of cases that can be timed.

A case is one pass through the public entry points: a routed projection of a diffusion transformer
(`PackedLinear`, `SharedProjection`, `ProtectedFFNOutput`, with or without the element-wise
neighbours in its kernels, through a prepared plan), the preparation of a weight (`compress`), or
one denoise step of a model with all its routed projections.  Shapes are those of the workload table
and the benchmark of this repository; `draw` takes others from the same ranges, odd and ragged sizes
among them.  Activations are N(0, 1) with 1 % of the channels twenty times larger, weights N(0, 0.02),
as in the benchmark.
"""
import importlib
import math

import torch

_PACKAGE = "slidesparse-diffusion_b200"
ss = importlib.import_module(_PACKAGE)
backend = importlib.import_module(_PACKAGE + ".backend")
denoiser = importlib.import_module(_PACKAGE + ".denoiser")
reconstruction = importlib.import_module(_PACKAGE + ".reconstruction")
routing = importlib.import_module(_PACKAGE + ".routing")

DEVICE = "cuda:0"
BATCH = 2                 # classifier-free guidance: conditional and unconditional half


def listed():
    return [
        # the benchmark's eager call: a square hidden-sized projection of few rows, where the call itself counts
        dict(name="small 256x1152-1152", op="plain", mode=4, m=256, k=1152, n=1152),
        # text stream of an MMDiT block (2 x 333 tokens: ragged), LayerNorm + modulation in the front-end
        dict(name="mmdit text qkv norm 666", op="norm", mode=6, m=666, k=2432, n=7296),
        # DiT-XL/2 at 512x512: Q|K|V of a block with its adaLN
        dict(name="dit qkv norm 2048", op="norm", mode=4, m=2048, k=1152, n=3456),
        # the single 2:4 projection of the benchmark (hidden 1152 FFN-in)
        dict(name="pixart fc1 4096", op="plain", mode=4, m=4096, k=1152, n=4608),
        # PixArt at 1024x1024: FFN-out with the GELU before it and the gated residual after it
        dict(name="pixart fc2 gelu gate 8192", op="gate", mode=8, m=8192, k=4608, n=1152),
        # fused Q|K|V of the 3072-wide double stream through a prepared plan
        dict(name="flux qkv plan 1536", op="plan", mode=6, m=1536, k=3072, n=9216),
        # its FFN-out: long K, few output channels
        dict(name="flux fc2 1536", op="plain", mode=8, m=1536, k=12288, n=3072),
        # single-stream output projection: dense attention columns as addend, FFN columns read in place
        dict(name="flux single out 1536", op="addend", mode=6, m=1536, k=12288, n=3072),
        # FFN-in of the image stream of an MMDiT block, unfused
        dict(name="sd35 fc1 2048", op="plain", mode=6, m=2048, k=2432, n=9728),
        # the largest projection of the benchmark sweep
        dict(name="flux fc1 16384", op="plain", mode=8, m=16384, k=3072, n=12288),
        # weight preparation with curvature compensation and joint rounding, 3072-wide Q|K|V
        dict(name="compress 9216x3072", op="compress", mode=6, k=3072, n=9216),
        # a denoise step of the class-conditional model at full depth: forward on the guidance pair,
        # guidance, sampler update
        dict(name="dit denoise step", op="step", mode=4, blocks=28),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["plain", "norm", "gate", "plan", "addend", "compress", "step"], [8, 3, 3, 2, 2, 1, 1])[0]
    mode = rng.choice([4, 6, 8])
    if op == "step":
        return dict(op=op, mode=mode, blocks=rng.randint(2, 28))
    if op == "compress":
        return dict(op=op, mode=mode, k=rng.choice([768, 1152, 1536, 2432, 3072]), n=rng.randint(512, 9216))
    while True:
        m, k, n = _log_int(rng, 16, 16384), _log_int(rng, 512, 16384), _log_int(rng, 512, 16384)
        # most widths of a model are multiples of 8; a plain projection takes any
        if op != "plain" or rng.random() < 0.8:
            k, n = k // 8 * 8, n // 8 * 8
        if op == "norm":
            m += m % BATCH
        if op == "gate":
            m = max(1, round(m / (32 * BATCH))) * 32 * BATCH      # whole groups of 32 rows per batch element
        if m * (k + n if op == "addend" else k) * n <= 16384 * 3072 * 12288:
            return dict(op=op, mode=mode, m=m, k=k, n=n)


def _activation(gen, m, k):
    x = torch.randn(m, k, generator=gen, device=DEVICE)
    outliers = torch.randperm(k, generator=gen, device=DEVICE)[:max(1, k // 100)]
    x[:, outliers] *= 20
    return x.to(torch.bfloat16)


def _linear(gen, k, n):
    layer = torch.nn.Linear(k, n, device=DEVICE, dtype=torch.bfloat16)
    layer.requires_grad_(False)
    layer.weight.normal_(0, 0.02, generator=gen)
    layer.bias.normal_(0, 0.1, generator=gen)
    return layer


def _vectors(gen, n, spread):
    return (torch.randn(BATCH, n, generator=gen, device=DEVICE) * spread).to(torch.bfloat16)


def prepare(case, seed):
    op, mode, m, k, n = (case.get(key) for key in ("op", "mode", "m", "k", "n"))
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    state = dict(op=op)
    if op == "step":
        model = denoiser.build("dit-xl-512", DEVICE, seed=seed, blocks=case["blocks"])
        model.select(model.pack(mode))
        model.fuse_neighbours()
        state["loop"] = denoiser.DenoiseLoop(model, graph=True)
        state["inputs"] = state["loop"].inputs(seed)
    elif op == "compress":
        samples = _activation(gen, 2 * k, k).float()
        state["curvature"] = reconstruction.factor_hessian(samples.T @ samples / samples.shape[0])
        state["weight"] = _linear(gen, k, n).weight.float()
        state["mode"], state["tail"] = mode, bool(k % mode)
    elif op == "addend":
        # n columns of attention output stay dense in front of the k columns of the FFN
        layer = _linear(gen, n + k, n)
        ffn = routing.pack_members([layer], mode, protected_prefix=n)
        state["call"] = ss.ProtectedFFNOutput(ffn, layer.weight[:, :n].contiguous())
        state["x"] = _activation(gen, m, n + k)
    else:
        packed = routing.pack_members([_linear(gen, k, n)], mode)
        x = _activation(gen, m, k)
        if op == "plan":
            packed = ss.PackedLinear(packed.packed, packed.metadata, packed.scales, packed.bias, k, n, mode,
                                     frontend="graph_native")
            packed.configure_for(m)
            state["call"] = ss.SharedProjection(packed, [n // 8 * 3, n - n // 8 * 3])
        else:
            state["call"] = packed
        if op in ("norm", "gate"):
            x = x.view(BATCH, m // BATCH, k)
        if op == "norm":
            state["shift"], state["scale"] = _vectors(gen, k, 0.1), _vectors(gen, k, 0.1)
        if op == "gate":
            state["gate"] = _vectors(gen, n, 0.5)
            state["residual"] = torch.randn(BATCH, m // BATCH, n, generator=gen, device=DEVICE).to(torch.bfloat16)
        state["x"] = x
    return state


def run(state):
    op = state["op"]
    if op == "step":
        return state["loop"].run(steps=1, inputs=state["inputs"])
    if op == "compress":
        done = reconstruction.compress(state["weight"], state["curvature"], state["mode"], allow_tail=state["tail"])
        return {key: done[key] for key in ("qweight", "scales", "zeros", "compensated", "proxy_loss")}
    if op == "norm":
        return state["call"].forward_fused(state["x"], backend.Prologue.norm_modulate(state["shift"], state["scale"]))
    if op == "gate":
        return state["call"].forward_fused(state["x"], backend.Prologue.gelu(), gate=state["gate"],
                                           residual=state["residual"])
    return state["call"](state["x"])


def _projection_work(mode, m, k, n):
    """Activations, packed weights (values and metadata of the slid width) and scales read once, the
    output written once; a multiplication and an addition per weight that the pattern keeps."""
    slid = -(-k // mode) * (mode // 2 - 1) * 4
    return 2 * m * k + n * slid * 5 // 8 + 8 * n + 2 * m * n, 2 * m * n * k * (mode - 2) // mode


def work(case):
    op, mode, m, k, n = (case.get(key) for key in ("op", "mode", "m", "k", "n"))
    if op == "compress":
        # the triangle of the factor and the weight in; values, scales, zeros, compensated weight and loss
        # out; each column's error reaches every later column of its row
        return dict(bytes=2 * k * k + (4 + 1 + 1 + 4) * n * k + 8 * n, flops=n * k * k)
    if op == "step":
        spec = denoiser.SPECS["dit-xl-512"]
        tokens, hidden, blocks = BATCH * spec.tokens, spec.hidden, case["blocks"]
        total = [0, 0]
        for width_in, width_out in ((hidden, 3 * hidden), (hidden, 4 * hidden), (4 * hidden, hidden)):
            b, f = _projection_work(mode, tokens, width_in, width_out)
            # activations between the projections need not leave the chip: weights count alone
            total[0] += b - 2 * tokens * (width_in + width_out)
            total[1] += f
        total[0] += 2 * hidden * hidden * 7                         # output projection and adaLN weights
        total[1] += 2 * tokens * hidden * hidden + 4 * tokens * (tokens // BATCH) * hidden + 2 * BATCH * hidden * 6 * hidden
        return dict(bytes=blocks * total[0] + 2 * 4 * 4 * 64 * 64, flops=blocks * total[1])
    b, f = _projection_work(mode, m, k, n)
    if op == "norm":
        b += 2 * 2 * BATCH * k
    if op == "gate":
        b += 2 * m * n + 2 * BATCH * n
    if op == "addend":
        b += 2 * m * n + 2 * n * n
        f += 2 * m * n * n
    return dict(bytes=b, flops=f)


def tolerance(case):
    # the preparation of a weight is fixed operation by operation; the others end in BF16 (or, the
    # denoise step, pass through it)
    return "exact" if case["op"] == "compress" else {"rel": 1e-2}
