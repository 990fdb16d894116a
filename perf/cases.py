"""The work a user of flare_b200 has it do, as measurable cases.

Every case is a plain dict; ``op`` says which public function runs and the rest are its sizes and options:

* ``mixer``          flare_multihead_mixer: a forward pass (``grad`` false) or forward and backward through autograd
* ``causal_prefill`` flare_causal_prefill over a whole prompt from an empty state
* ``causal_decode``  flare_causal_decode: one token on a state that a prompt has filled
* ``causal_step``    flare_causal_mixer, forward and backward
* ``triple``         triple_attention, forward and backward
* ``causal_linear``  causal_linear, forward

Values are drawn as in the repository's benchmark: q, k, v ~ N(0, D^-1/2) (variance), gradients ~ N(0, 1).
``heads`` is the memory layout of k, v and the output gradient: "split" is the 'b n (h d) -> b h n d' view of a
[B, N, H*D] activation that the FLARE modules pass, "dense" a [B, H, N, D] tensor.
"""
import math

import torch

import flare_b200 as fb

_DT = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}


def _mixer(name, B, H, N, M, D, dtype, grad=True, heads="split", autocast=False, mask=False):
    c = dict(op="mixer", B=B, H=H, N=N, M=M, D=D, dtype=dtype, grad=grad, heads=heads, autocast=autocast, mask=mask)
    return dict(c, name=name) if name else c


def _causal(op, name, B, H, N, M, D):
    c = dict(op=op, B=B, H=H, N=N, M=M, D=D, dtype="bf16")
    return dict(c, name=name) if name else c


def _triple(name, B, H, N, dtype):
    c = dict(op="triple", B=B, H=H, N=N, D=32, dtype=dtype)
    return dict(c, name=name) if name else c


def _linear(name, B, H, N, Dv, dtype):
    c = dict(op="causal_linear", B=B, H=H, N=N, Dk=128, Dv=Dv, dtype=dtype)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small mesh through a trained surrogate: latency is all that counts
        _mixer("mesh_infer", 1, 8, 1024, 64, 16, "bf16", grad=False),
        # the fp32 mixer of the reference's CPU-runnable configuration (trainers default to full precision)
        _mixer("fp32_step", 2, 8, 4096, 64, 16, "fp32"),
        # a layer of the PDE surrogate on a batch of 85 x 85 grids, under the trainer's autocast
        _mixer("pde_layer_step", 4, 8, 7225, 64, 16, "bf16", autocast=True),
        # a layer of the long-range-arena classifier: padded sequences, half precision
        _mixer("lra_step", 32, 8, 4096, 128, 16, "fp16", autocast=True, mask=True),
        # automotive aerodynamics point clouds with the narrow trunk (64 channels over 8 heads)
        _mixer("narrow_cloud_step", 1, 8, 500_000, 512, 8, "bf16", autocast=True),
        # a rank's share of the 3-D point-cloud encoder layer: wide trunk, 512 latents, ragged shard
        _mixer("encoder_step", 1, 8, 300_007, 512, 32, "bf16", autocast=True),
        # the million-token mixer of the benchmark
        _mixer("million_step", 1, 8, 1 << 20, 256, 32, "bf16", heads="dense"),
        # the causal decoder block: prompt, one token of generation, training
        _causal("causal_prefill", "causal_prefill", 4, 16, 8192, 128, 64),
        _causal("causal_decode", "causal_decode", 4, 16, 1, 128, 64),
        _causal("causal_step", "causal_step", 4, 16, 8192, 128, 64),
        # triple attention at the long end of its benchmark
        _triple("triple_step", 1, 8, 500_000, "fp16"),
        # causal linear attention at its benchmark's shape
        _linear("causal_linear", 8, 8, 2048, 32, "bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("mesh", "fp32", "layer", "layer", "padded", "cloud", "cloud", "narrow", "prefill", "decode", "train",
                       "triple", "linear"))
    if kind in ("mesh", "layer"):
        D = rng.choice((16, 16, 32))
        M = rng.choice((32, 64, 128, 256))
        B = rng.choice((1, 1, 2) if kind == "mesh" else (1, 2, 4, 8))
        N = _log(rng, 500, 20_000)
        return _mixer(None, B, 8, N, M, D, rng.choice(("bf16", "fp16")), grad=kind == "layer", autocast=kind == "layer")
    if kind == "fp32":
        return _mixer(None, rng.choice((1, 2, 4)), rng.choice((4, 8)), _log(rng, 500, 20_000), rng.choice((32, 64, 128)),
                      rng.choice((8, 16, 32)), "fp32")
    if kind == "padded":
        return _mixer(None, rng.choice((4, 8, 16, 32)), 8, _log(rng, 256, 4096), rng.choice((64, 128)), rng.choice((16, 32)),
                      rng.choice(("bf16", "fp16")), autocast=True, mask=True)
    if kind == "cloud":
        M = rng.choice((64, 128, 256, 512, 1024))
        N = _log(rng, 30_000, min(1_000_000, 260_000_000 // M))
        return _mixer(None, 1, 8, N, M, rng.choice((16, 32)), rng.choice(("bf16", "fp16")), autocast=True)
    if kind == "narrow":
        M = rng.choice((64, 128, 256, 512, 1024, 2048))
        N = _log(rng, 5_000, min(1_000_000, 250_000_000 // M))
        return _mixer(None, 1, 8, N, M, 8, rng.choice(("bf16", "fp16")), autocast=True)
    if kind == "prefill":
        return _causal("causal_prefill", None, rng.choice((1, 2, 4)), rng.choice((8, 16)), _log(rng, 200, 8192),
                       rng.choice((64, 128)), rng.choice((32, 64)))
    if kind == "decode":
        return _causal("causal_decode", None, _log(rng, 1, 32), rng.choice((8, 16)), 1, rng.choice((64, 128)), rng.choice((32, 64)))
    if kind == "train":
        return _causal("causal_step", None, rng.choice((1, 2, 4)), rng.choice((8, 16)), _log(rng, 200, 8192),
                       rng.choice((64, 128)), rng.choice((32, 64)))
    if kind == "triple":
        return _triple(None, 1, 8, _log(rng, 1000, 500_000), rng.choice(("bf16", "fp16")))
    return _linear(None, rng.choice((1, 2, 4, 8)), rng.choice((4, 8)), _log(rng, 256, 8192), rng.choice((32, 64)),
                   rng.choice(("bf16", "fp16")))


def _randn(gen, shape, std, dtype, heads="dense"):
    if heads == "split":
        B, H, N, D = shape
        t = torch.randn(B, N, H, D, generator=gen, device="cuda", dtype=torch.float32).mul_(std).to(dtype)
        return t.permute(0, 2, 1, 3)
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(std).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, dt = case["op"], _DT[case["dtype"]]
    B, H, N = case["B"], case["H"], case["N"]
    s = dict(case=case)
    if op == "triple":
        D = case["D"]
        s["x"] = [_randn(gen, (B, H, N, D), D ** -0.25, dt).requires_grad_(True) for _ in range(5)]
        s["do"] = _randn(gen, (B, H, N, D), 1.0, dt)
        return s
    if op == "causal_linear":
        s["q"], s["k"] = (_randn(gen, (B, H, N, case["Dk"]), case["Dk"] ** -0.25, dt) for _ in range(2))
        s["v"] = _randn(gen, (B, H, N, case["Dv"]), case["Dv"] ** -0.25, dt)
        return s
    M, D = case["M"], case["D"]
    std = D ** -0.25
    heads = case.get("heads", "split")
    # under autocast the latents are the module's fp32 parameter; k and v come out of 16-bit projections
    s["q"] = _randn(gen, (H, M, D), std, torch.float32 if case.get("autocast") else dt)
    s["k"] = _randn(gen, (B, H, N, D), std, dt, heads)
    s["v"] = _randn(gen, (B, H, N, D), std, dt, heads)
    if case.get("grad") or op == "causal_step":
        for n in ("q", "k", "v"):
            s[n].requires_grad_(True)
        s["dy"] = _randn(gen, (B, H, N, D), 1.0, dt, heads)
    if case.get("mask"):
        lens = torch.randint(N // 4, N + 1, (B, 1), generator=gen, device="cuda")
        s["mask"] = torch.arange(N, device="cuda")[None, :] < lens
    if op == "causal_decode":
        prompt = [_randn(gen, (B, H, 256, D), std, dt, heads) for _ in range(2)]
        s["state"] = fb.flare_causal_prefill(s["q"], prompt[0], prompt[1], 1.0)[1]
    return s


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "mixer":
        q, k, v = state["q"], state["k"], state["v"]
        if case["autocast"]:
            with torch.autocast("cuda", _DT[case["dtype"]]):
                y = fb.flare_multihead_mixer(q, k, v, 1.0, key_mask=state.get("mask"))
        else:
            y = fb.flare_multihead_mixer(q, k, v, 1.0, key_mask=state.get("mask"))
        if not case["grad"]:
            return y
        return (y.detach(), *torch.autograd.grad(y, (q, k, v), state["dy"]))
    if op == "causal_prefill":
        return fb.flare_causal_prefill(state["q"], state["k"], state["v"], 1.0)
    if op == "causal_decode":
        return fb.flare_causal_decode(state["q"], state["k"], state["v"], state["state"], 1.0), state["state"]
    if op == "causal_step":
        q, k, v = state["q"], state["k"], state["v"]
        y = fb.flare_causal_mixer(q, k, v, 1.0)
        return (y.detach(), *torch.autograd.grad(y, (q, k, v), state["dy"]))
    if op == "triple":
        rank3, o = fb.triple_attention(*state["x"])
        return (rank3.detach(), o.detach(), *torch.autograd.grad(o, state["x"], state["do"]))
    return fb.causal_linear(state["q"], state["k"], state["v"])


def work(case):
    op = case["op"]
    e = 4 if case["dtype"] == "fp32" else 2
    B, H, N = case["B"], case["H"], case["N"]
    if op == "triple":
        D = case["D"]
        # STATE and dSTATE, O and five gradients: eight products of 2 D^3 a token; 6 tensors read, 6 written
        return dict(bytes=12 * B * H * N * D * e + 2 * 4 * B * H * D ** 3, flops=16 * B * H * N * D ** 3)
    if op == "causal_linear":
        Dk, Dv = case["Dk"], case["Dv"]
        return dict(bytes=B * H * N * (2 * Dk + 2 * Dv) * e, flops=4 * B * H * N * Dk * Dv)
    M, D = case["M"], case["D"]
    W, T = B * H * N * M, B * H * N * D * e
    lat = H * M * D * (4 if case.get("autocast") else e)
    rec = B * H * M * (D + 2) * 4
    if op == "mixer":
        if case["grad"]:      # k, v, dy in; y, dk, dv out; q in, dq out
            return dict(bytes=6 * T + 2 * lat, flops=24 * W * D)
        return dict(bytes=3 * T + lat, flops=8 * W * D)
    if op == "causal_prefill":
        return dict(bytes=3 * T + lat + rec, flops=6 * W * D)
    if op == "causal_decode":  # the state is read and written
        return dict(bytes=3 * T + lat + 2 * rec, flops=6 * W * D)
    return dict(bytes=6 * T + 2 * lat, flops=18 * W * D)


def tolerance(case):
    # what two correct implementations differ by: fp32 sums and exponentials; weights and results rounded to 16 bits
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
