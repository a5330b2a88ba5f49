"""Workloads of the MoE expert block, one pass each through the public entry points.

A case names a layer (one of the configurations in strata_b200/synth.py, or that shape with another weight format), the
number of tokens of the pass and the entry point:

  forward  MoeLayer.forward on activations resident on the GPU: router, grouping, experts, shared expert, combine
  host     MoeLayer.forward_host on pinned host activations, the result back in pinned host memory
  latent   LatentMoe.forward: the block whose experts work on a latent narrower than the model
  exact    the bit-exact DeepSeek arithmetic through the stage calls: route, group, gather, experts, join

Weights are random bytes with the scale distributions of strata_b200/synth.py, activations N(0, 1) in BF16, the router
N(0, 0.02^2); all of it comes from the seed.
"""
import math

import numpy as np
import torch

from strata_b200 import MoeContext, MoeLayer, synth
from strata_b200.api import LatentMoe

_FORMATS = {"mxfp4": synth.FMT_MXFP4, "nvfp4": synth.FMT_NVFP4, "int4": synth.FMT_INT4, "bf16": synth.FMT_BF16}


def listed():
    return [
        # one user's token through a DeepSeek-V4-Flash layer: the smallest call, 75 MB of weights
        _case("mxfp4_decode_1", "c0", "mxfp4", 1),
        # eight users decoding together: the headline decode step
        _case("mxfp4_decode_8", "c0", "mxfp4", 8),
        # the numerical mode that reproduces the reference's DeepSeek arithmetic bit for bit, a few users decoding
        _case("mxfp4_exact_4", "c0", "mxfp4", 4, "exact"),
        # the plain-BF16 layers of a Laguna model in a small decode batch
        _case("bf16_decode_19", "c1_sigmoid", "bf16", 19),
        # a large continuous-decoding batch of a Laguna NVFP4 layer with its always-on shared expert
        _case("nvfp4_shared_256", "c1_sigmoid", "nvfp4", 256),
        # a small decode batch of a GLM INT4 layer
        _case("int4_decode_4", "c2", "int4", 4),
        # a short prompt of a ragged length on the same layer
        _case("int4_prompt_333", "c2", "int4", 333),
        # a prefill chunk of 4096 tokens on the same layer
        _case("int4_prefill_4096", "c2", "int4", 4096),
        # the same chunk handed over and taken back in host memory
        _case("int4_host_4096", "c2", "int4", 4096, "host"),
        # 896 experts under a Zipf-skewed router, a large decode batch
        _case("mxfp4_skewed_256", "c4", "mxfp4", 256),
        # a Kimi-K3 LatentMoE layer, four users decoding
        _case("latent_decode_4", "kimi", "mxfp4", 4, "latent"),
        # the largest call: a prefill of 16384 tokens on 256 experts
        _case("mxfp4_prefill_16384", "c3", "mxfp4", 16384),
    ]


def _case(name, layer, weights, tokens, entry="forward"):
    return {"name": name, "layer": layer, "weights": weights, "tokens": tokens, "entry": entry}


# (layer, weights, entry, fewest tokens, most tokens)
_RANGES = [
    ("c0", "mxfp4", "forward", 1, 4096),
    ("c1_sigmoid", "nvfp4", "forward", 1, 4096),
    ("c1", "nvfp4", "forward", 1, 4096),
    ("c2", "int4", "forward", 1, 4096),
    ("c3", "mxfp4", "forward", 1, 16384),
    ("c4", "mxfp4", "forward", 1, 1024),
    ("c1_sigmoid", "bf16", "forward", 1, 128),
    ("c2", "int4", "host", 16, 4096),
    ("kimi", "mxfp4", "latent", 1, 256),
    ("c0", "mxfp4", "exact", 1, 16),
]


def draw(rng):
    layer, weights, entry, lo, hi = _RANGES[rng.randrange(len(_RANGES))]
    tokens = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))
    return {"layer": layer, "weights": weights, "tokens": min(max(tokens, lo), hi), "entry": entry}


def _config(case, seed=0):
    return synth.CONFIGS[case["layer"]].with_(fmt=_FORMATS[case["weights"]], T=case["tokens"], seed=seed)


_context = None


def _ctx():
    """One context per process, as in a program that serves a model: its layers share the workspaces."""
    global _context
    if _context is None:
        _context = MoeContext(0)
    return _context


def _random_layer(cfg, gen, dev):
    """A synth.SynthLayer with every tensor drawn on the GPU."""
    def normal(shape, std, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=dev).normal_(0.0, std, generator=gen)

    def bits(n, size):
        return torch.randint(0, 256, (n, size), dtype=torch.uint8, device=dev, generator=gen)

    layer = synth.SynthLayer(cfg, dev, expert_begin=0, expert_end=cfg.E)
    layer.x = normal((cfg.T, cfg.Hx), 1.0)
    layer.router_w = normal((cfg.E, cfg.Hx), 0.02)
    if cfg.zipf_s > 0:
        rank = torch.randperm(cfg.E, device=dev, generator=gen).to(torch.float32) + 1.0
        layer.bias = -cfg.zipf_s * 0.25 * torch.log(rank)
    if cfg.I_shared:
        for role in synth.ROLES:
            layer.shared[role] = normal((cfg.Hx, cfg.I_shared) if role == "down" else (cfg.I_shared, cfg.Hx), 0.02)
    if cfg.H_model:
        layer.latent = {"down": normal((cfg.H, cfg.H_model), cfg.H_model ** -0.5), "up": normal((cfg.H_model, cfg.H), 0.02),
                        "norm": 1.0 + normal((cfg.H,), 0.03, torch.float32)}
    for role in synth.ROLES:
        packed_bytes, scale_bytes = synth.expert_bytes(cfg, role)
        if cfg.fmt == synth.FMT_BF16:
            layer.packed[role] = normal((cfg.E, packed_bytes // 2), 0.02).view(torch.uint8)
            layer.scales[role] = torch.zeros(cfg.E, 0, dtype=torch.uint8, device=dev)
            continue
        layer.packed[role] = bits(cfg.E, packed_bytes)
        if cfg.fmt == synth.FMT_INT4:   # BF16 scales, 0.02 / 4.61 times 1 .. 1.1
            u = torch.rand(cfg.E, scale_bytes // 2, device=dev, generator=gen)
            layer.scales[role] = ((0.02 / 4.61) * (1.0 + 0.1 * u)).to(torch.bfloat16).view(torch.uint8)
        elif cfg.fmt == synth.FMT_NVFP4:
            table = torch.from_numpy(synth.e4m3_encode_table()).to(dev)
            layer.scales[role] = table[bits(cfg.E, scale_bytes).int()]
        else:
            layer.scales[role] = synth.MXFP4_SCALE_BYTE - 1 + bits(cfg.E, scale_bytes) % 3
    return layer


def prepare(case, seed):
    ctx = _ctx()
    dev = ctx.device
    cfg = _config(case, seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    weights = _random_layer(cfg, gen, dev)
    block = (LatentMoe if case["entry"] == "latent" else MoeLayer)(ctx, cfg, max_tokens=cfg.T)
    block.load_synth(weights)
    state = {"entry": case["entry"], "cfg": cfg, "block": block, "weights": weights, "x": weights.x}
    if case["entry"] == "forward":
        state["out"] = torch.empty(cfg.T, cfg.H, dtype=torch.float32, device=dev)
    elif case["entry"] == "host":
        state["x"] = weights.x.cpu().pin_memory()
        state["out"] = torch.empty(cfg.T, cfg.H, dtype=torch.float32, pin_memory=True)
    elif case["entry"] == "exact":
        state["rows"] = weights.x.float()
    return state


def run(state):
    block, x = state["block"], state["x"]
    if state["entry"] == "forward":
        return block.forward(x, state["out"])
    if state["entry"] == "host":
        return block.forward_host(x, state["out"])
    if state["entry"] == "latent":
        return block.forward(x, want_routing=True)
    ids, weights = block.route(x)
    _, offsets, perm, inv = block.group(ids, want_inv=True)
    rows = block.gather_rows(state["rows"], perm, state["cfg"].k)
    y = block.experts_grouped_dsv4(rows, offsets, weights.view(-1)[perm.long()])
    return ids, weights, block.combine_dsv4(y, inv, x.shape[0])


def _active_experts(cfg):
    """Expected number of experts that at least one of the pass's tokens selects."""
    if cfg.zipf_s == 0:
        return cfg.E * (1.0 - (1.0 - cfg.k / cfg.E) ** cfg.T)
    rng = np.random.RandomState(0)
    bias = -cfg.zipf_s * 0.25 * np.log(rng.permutation(cfg.E) + 1.0)
    hit = np.zeros(cfg.E, bool)
    for _ in range(cfg.T):
        score = 1.0 / (1.0 + np.exp(-rng.standard_normal(cfg.E) * 0.02 * cfg.Hx ** 0.5)) + bias
        hit[np.argpartition(-score, cfg.k)[:cfg.k]] = True
    return float(hit.sum())


def work(case):
    cfg = _config(case)
    T, out_width = cfg.T, cfg.H_model or cfg.H
    expert = sum(sum(synth.expert_bytes(cfg, role)) for role in synth.ROLES)
    x_bytes = 4 if case["entry"] == "exact" else 2
    moved = T * cfg.Hx * x_bytes + T * out_width * 4 + cfg.E * cfg.Hx * 2 + _active_experts(cfg) * expert
    moved += 3 * cfg.I_shared * cfg.Hx * 2
    flops = 6.0 * cfg.H * cfg.I * T * cfg.k + 2.0 * T * cfg.E * cfg.Hx + 6.0 * T * cfg.I_shared * cfg.Hx
    if cfg.H_model:
        moved += 2 * cfg.H * cfg.H_model * 2
        flops += 4.0 * T * cfg.H * cfg.H_model
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["entry"] == "exact":
        return "exact"
    # 16-bit activations against 4-bit or BF16 weights with 32-bit sums: the SwiGLU output and, for large batches, the
    # expert rows are rounded to 11 bits on the way (unit roundoff 4.9e-4)
    return {"rel": 1e-3, "max": 1e-2}
