"""The work that a user of cssm_b200 has it do, as timed cases: whole classifiers (CSSM-SHViT s1 in
bfloat16, SimpleCSSM in float32) and single mixer blocks, from one image to full batches, through the
package's public entry points.

A case is a dict of plain values.  "kind" is "shvit" (the image classifier), "simple" (stem + one
block + readout) or "block" (a mixer block on its own); the other keys are sizes and options.
All passes are forward passes: the framework has no backward direction."""
from __future__ import annotations

import json
import math

import torch

from cssm_b200 import (AdditiveCSSM, CSSMSHViT, DeltaNetCSSM, GatedCSSM, GatedDeltaNetCSSM, NoGateCSSM,
                       SimpleCSSM, synth)

DEV = "cuda"


# ------------------------------------------------------------------------------- cases ----
def _shvit(B, hw=224, T=1, **kw):
    return dict(kind="shvit", B=B, hw=hw, T=T, **kw)


def _simple(mixer, B, T, E=64, ks=11, gate="factored", pos="spatiotemporal", stem="image1", last=False,
            qkv_conv=1, **kw):
    return dict(kind="simple", mixer=mixer, B=B, T=T, E=E, ks=ks, gate=gate, pos=pos, stem=stem, last=last,
                qkv_conv=qkv_conv, **kw)


def _block(mixer, B, T, H, W, C, ks=11, gate="factored", pos="spatiotemporal", bf16=False, dk=4, qkv_conv=1, **kw):
    return dict(kind="block", mixer=mixer, B=B, T=T, H=H, W=W, C=C, ks=ks, gate=gate, pos=pos, bf16=bf16,
                dk=dk, qkv_conv=qkv_conv, **kw)


def listed():
    return [
        # throughput serving / evaluation of the ImageNet-shaped classifier: the batch of bench.py
        _shvit(512, name="shvit_b512"),
        # one picture at a time: an interactive service, where launches and host work count
        _shvit(1, name="shvit_b1"),
        # the last, ragged batch of an evaluation at a larger test resolution: planes of 16x16 and 8x8
        _shvit(33, hw=256, name="shvit_256_b33"),
        # the constructor's own defaults: eight time steps, kernel sizes 15/15/5/3, spatial short convs
        _shvit(48, T=8, name="shvit_t8_b48"),
        # the smallest training-time configuration: 1x1 kernel, T = 1, dense gates, batch 8
        _simple("gated", 8, 1, ks=1, gate="dense", stem="image2", name="simple_gated_t1_b8"),
        # stroke images repeated over eight steps: the configuration the fused block was built for
        _simple("gated", 128, 8, name="simple_gated_t8_b128"),
        # the same task with the matrix delta rule, 5x5 qkv conv and mrope
        _simple("gdn", 128, 8, pos="mrope", qkv_conv=5, name="simple_gdn_t8_b128"),
        # 32-frame clips of 32x32 pixels
        _simple("gdn", 128, 32, stem="clip", name="simple_gdn_clip_b128"),
        # SimpleCSSM's default width, kernel size and gates on the planes of 224-pixel images
        _block("gated", 16, 8, 56, 56, 32, ks=15, gate="dense", name="gated_56_c32"),
        # GatedDeltaNetCSSM as its constructor gives it (key dim 2, per-channel gates), 28x28 planes
        _block("gdn", 12, 8, 28, 28, 64, gate="channel", pos="none", dk=2, name="gdn_28_dk2"),
        # DeltaNetCSSM's default per-channel gates on short clips of 32x32 planes
        _block("deltanet", 24, 12, 32, 32, 64, gate="channel", name="deltanet_32"),
        # the single-state additive mixer on 64x64 planes
        _block("additive", 12, 8, 64, 64, 64, gate="factored", name="additive_64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("shvit", "shvit", "simple", "simple", "block", "block", "block"))
    if kind == "shvit":
        hw = rng.choice((224, 224, 224, 160, 192, 256, 288))
        T = rng.choice((1, 1, 1, 4, 8))
        most = (512 if T == 1 else 96 / T * 4) * (1.0 if hw == 224 else 0.25) * (224 / hw) ** 2
        return _shvit(_log_int(rng, 1, max(2, most)), hw=hw, T=T)
    if kind == "simple":
        mixer = rng.choice(("gated", "gated", "gdn", "gdn", "deltanet", "add_kqv_1", "no_gate"))
        stem = rng.choice(("image1", "image1", "image2", "clip"))
        T = rng.choice((4, 8, 12, 16, 32)) if stem == "clip" else rng.choice((1, 2, 4, 8))
        E = rng.choice((32, 64, 64))
        return _simple(mixer, _log_int(rng, 1, 96), T, E=E, ks=rng.choice((1, 3, 7, 11, 15)),
                       gate=rng.choice(("factored", "factored", "dense")),
                       pos=rng.choice(("none", "spatiotemporal", "mrope", "temporal")), stem=stem,
                       last=mixer in ("gated", "gdn") and rng.random() < 0.3,
                       qkv_conv=rng.choice((1, 3, 5)))
    mixer = rng.choice(("gated", "gated", "gdn", "gdn", "deltanet", "additive", "nogate"))
    gates = {"gated": ("factored", "dense"), "nogate": ("none",), "gdn": ("factored", "dense", "channel", "scalar")}
    side = rng.choice(("any", "any", "square", "fft"))
    if side == "fft":
        H = W = rng.choice((32, 64))
    elif side == "square":
        H = W = rng.choice((7, 8, 14, 16, 20, 28, 40, 48, 56))
    else:
        H, W = rng.randint(7, 56), rng.randint(7, 56)
    dk = rng.choice((2, 4))
    if mixer == "gdn" and H * W > 2304 and (H, W) != (64, 64):
        H, W = min(H, 48), min(W, 48)
    C = rng.choice((16, 32, 48, 64, 96))
    T = rng.choice((1, 2, 4, 5, 8, 12))
    most = 8.0e6 / (T * H * W * C)              # an eighth of a 64x64 batch of 128 over eight steps, or less
    return _block(mixer, _log_int(rng, 1, max(1.5, most)), T, H, W, C, ks=rng.choice((1, 3, 5, 7)),
                  gate=rng.choice(gates.get(mixer, ("factored", "dense", "channel"))),
                  pos=rng.choice(("none", "spatiotemporal", "mrope")), bf16=mixer == "gated" and rng.random() < 0.4,
                  dk=dk, qkv_conv=rng.choice((1, 1, 3)))


# ----------------------------------------------------------------------- models, weights ----
def _shvit_model(c):
    if c["T"] == 1:
        return CSSMSHViT(embed_dims=(64, 128, 256, 384), depths=(1, 2, 2, 1), num_timesteps=1,
                         kernel_sizes=(1, 1, 1, 1), short_conv_spatial_size=0)
    return CSSMSHViT(embed_dims=(64, 128, 256, 384), depths=(1, 2, 2, 1), num_timesteps=c["T"])


def _shvit_variables(m, hw):
    """A random tree of the model's parameters and BatchNorm statistics, made on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(20)

    def n(*shape, std=1.0, mean=0.0):
        return mean + std * torch.randn(shape, generator=g, device=DEV)

    def norm(c):
        return {"scale": n(c, std=0.1, mean=1.0), "bias": n(c, std=0.1)}

    def dense(ci, co):
        return {"kernel": n(ci, co, std=ci ** -0.5), "bias": n(co, std=0.1)}

    def dw(k, c):
        return {"kernel": n(k, k, 1, c, std=1.0 / k), "bias": n(c, std=0.1)}

    def convbn(ci, co):
        return ({"conv": {"kernel": n(3, 3, ci, co, std=(9 * ci) ** -0.5)}, "bn": norm(co)},
                {"bn": {"mean": n(co, std=0.2), "var": n(co, std=0.3).exp()}})

    E = m.embed_dims
    params, stats = {}, {}
    (p0, s0), (p1, s1) = convbn(3, E[0] // 2), convbn(E[0] // 2, E[0])
    params["patch_embed"], stats["patch_embed"] = {"ConvBN_0": p0, "ConvBN_1": p1}, {"ConvBN_0": s0, "ConvBN_1": s1}
    side = -(-hw // 4)
    for s in range(4):
        if s > 0:
            p, st = convbn(E[s - 1], E[s])
            params[f"downsample{s}"], stats[f"downsample{s}"] = {"ConvBN_0": p}, {"ConvBN_0": st}
            side = -(-side // 2)
        hid = int(E[s] * m.mlp_ratio)
        for b in range(m.depths[s]):
            blk = {"norm1": norm(E[s]), "norm2": norm(E[s]),
                   "mlp": {"fc1": dense(E[s], hid), "fc2": dense(hid, E[s])}}
            if m.use_cssm_stages[s]:
                mix = GatedCSSM(channels=E[s], kernel_size=m.kernel_sizes[s], gate_type=m.gate_type,
                                short_conv_size=m.short_conv_size,
                                short_conv_spatial_size=m.short_conv_spatial_size)
                blk["cssm"] = mix.init(30 + 4 * s + b, (1, 1, side, side, E[s]), bias_scale=0.1)["params"]
                blk["pos_conv"] = dw(3, E[s])
                blk["mlp"]["dwconv"] = {"dwconv": dw(3, hid)}
            else:
                blk["dwconv"], blk["pwconv"] = {"dwconv": dw(7, E[s])}, dense(E[s], E[s])
            params[f"stage{s}_block{b}"] = blk
    params["norm"], params["head"] = norm(E[3]), dense(E[3], m.num_classes)
    return {"params": params, "batch_stats": stats}


def _simple_model(c):
    gdn = dict(delta_key_dim=4, qkv_conv_size=c["qkv_conv"]) if c["mixer"] == "gdn" else {}
    return SimpleCSSM(cssm_type=c["mixer"], embed_dim=c["E"], kernel_size=c["ks"], gate_type=c["gate"],
                      pos_embed=c["pos"], seq_len=c["T"], num_classes=2,
                      stem_mode="pathtracker" if c["stem"] == "clip" else "default",
                      stem_layers=2 if c["stem"] == "image2" else 1, pool_type="max", **gdn)


def _block_model(c):
    kw = dict(channels=c["C"], kernel_size=c["ks"])
    if c["mixer"] == "nogate":
        return NoGateCSSM(**kw)
    kw.update(rope_mode=c["pos"], gate_type=c["gate"])
    if c["mixer"] == "gated":
        return GatedCSSM(**kw)
    if c["mixer"] == "gdn":
        return GatedDeltaNetCSSM(delta_key_dim=c["dk"], qkv_conv_size=c["qkv_conv"], **kw)
    if c["mixer"] == "deltanet":
        return DeltaNetCSSM(**kw)
    return AdditiveCSSM(single_state=True, **kw)


def _input_shape(c):
    if c["kind"] == "shvit":
        return (c["B"], c["hw"], c["hw"], 3)
    if c["kind"] == "simple":
        return (c["B"], c["T"], 32, 32, 3) if c["stem"] == "clip" else (c["B"], 128, 128, 1)
    return (c["B"], c["T"], c["H"], c["W"], c["C"])


# A program keeps one model and feeds it batch after batch, so the states of one case share theirs;
# the model of the case before is let go.
_MODEL = {}


def _model(c):
    key = json.dumps({k: v for k, v in c.items() if k != "name"}, sort_keys=True)
    if key not in _MODEL:
        _MODEL.clear()
        if c["kind"] == "shvit":
            m = _shvit_model(c)
            v = _shvit_variables(m, c["hw"])
        else:
            m = _simple_model(c) if c["kind"] == "simple" else _block_model(c)
            v = m.init(10, _input_shape(c), bias_scale=0.1)
        bound = m.bind(v, DEV)
        if c["kind"] == "simple":
            bound.block.plan(bound.block_desc(bound.desc(_input_shape(c))))
        else:
            bound.plan(bound.desc(_input_shape(c)) if c["kind"] == "block" else m.desc(_input_shape(c)))
        _MODEL[key] = bound
    return _MODEL[key]


# -------------------------------------------------------------------------------- passes ----
def prepare(case, seed):
    bound = _model(case)
    g = torch.Generator(device=DEV).manual_seed(seed)
    shape = _input_shape(case)
    if case["kind"] == "simple" and case["stem"] == "clip":
        # black frames with coloured dots on random walks
        few = torch.from_numpy(synth.dot_clips(min(case["B"], 16), T=case["T"], seed0=seed)).to(DEV)
        pick = torch.randint(0, few.shape[0], (case["B"],), generator=g, device=DEV)
        x = few[pick].roll(int(seed) % 7, 3)
    elif case["kind"] == "simple":
        # dashed strokes, ~6 % of the pixels set; a few drawings, shifted to make a batch
        few = torch.from_numpy(synth.stroke_batch(4, seed0=seed)).to(DEV)
        x = torch.empty(shape, device=DEV)
        shift = torch.randint(0, 128, (case["B"], 2), generator=g, device=DEV).tolist()
        for b, (dy, dx) in enumerate(shift):
            x[b] = few[b % few.shape[0]].roll((dy, dx), (0, 1))
    else:
        x = torch.randn(shape, generator=g, device=DEV)
        if case["kind"] == "shvit" or case["bf16"]:
            x = x.to(torch.bfloat16)
    return {"model": bound, "x": x.contiguous(), "last": case.get("last", False)}


def run(state):
    if state["last"]:
        return state["model"](state["x"], last_frame_only=True)
    return state["model"](state["x"])


# --------------------------------------------------------------- what a pass cannot avoid ----
def _mixer_flops(mixer, B, T, H, W, C, dk=4, qkv_conv=1, kt=4, ksp=3):
    """Operations of one block: projections, short convs, transforms (2.5 N log2 N each way for a real
    plane of N pixels) and the per-bin recurrence."""
    px, bins = B * T * H * W, B * T * H * (W // 2 + 1)
    fft = 2.5 * math.log2(H * W)
    if mixer == "gated":
        return px * C * (2 * 3 * C + 2 * ksp * ksp + 2 * kt + 2 * fft) + bins * C * 20
    if mixer == "gdn":
        return px * C * (2 * 5 * C + 2 * qkv_conv ** 2 + 6 * kt + 4 * fft) + bins * C * dk * 32
    if mixer == "deltanet":
        return px * C * (2 * 4 * C + 4 * fft) + bins * C * 50
    if mixer in ("additive", "add_kqv_1"):
        return px * C * (2 * 2 * C + 2 * fft) + bins * C * 20
    return px * C * (2 * C + 2 * fft) + bins * C * 8


def _gate_weights(c, C, H, W):
    n = {"gated": 3, "gdn": 4, "deltanet": 5, "additive": 3, "add_kqv_1": 3}.get(c["mixer"], 0)
    Wf = W // 2 + 1
    return n * C * {"factored": H + Wf, "dense": H * Wf, "channel": C, "scalar": 1, "none": 0}[c["gate"]]


def work(case):
    """Inputs, weights and outputs once each, and the operations of the pass."""
    c = case
    B, T = c["B"], c["T"]
    if c["kind"] == "block":
        H, W, C = c["H"], c["W"], c["C"]
        n = B * T * H * W * C
        weights = 4 * ((6 if c["mixer"] in ("gdn", "deltanet") else 4) * C * C + _gate_weights(c, C, H, W))
        return {"bytes": n * ((2 if c["bf16"] else 4) + 4) + weights,
                "flops": _mixer_flops(c["mixer"], B, T, H, W, C, c["dk"], c["qkv_conv"])}
    if c["kind"] == "simple":
        E = c["E"]
        side = {"image1": 64, "image2": 32, "clip": 32}[c["stem"]]
        frames = B * T if c["stem"] == "clip" else B
        px_in = frames * (1024 * 3 if c["stem"] == "clip" else 128 * 128)
        stem = {"clip": 2 * 3 * E * 1024, "image1": 2 * 9 * E * 16384,
                "image2": 2 * 9 * E * 16384 + 2 * 9 * E * E * 4096}[c["stem"]] * frames
        weights = 4 * (6 * E * E + _gate_weights(c, E, side, side))
        return {"bytes": 4 * px_in + weights + 8 * B,
                "flops": stem + _mixer_flops(c["mixer"], B, T, side, side, E, 4, c["qkv_conv"])}
    E, depths, side = (64, 128, 256, 384), (1, 2, 2, 1), -(-c["hw"] // 4)
    flops = B * (2 * 27 * 32 * (2 * side) ** 2 + 2 * 9 * 32 * 64 * side * side)
    weights = 2 * (27 * 32 + 9 * 32 * 64)
    for s in range(4):
        if s > 0:
            side = -(-side // 2)
            flops += B * 2 * 9 * E[s - 1] * E[s] * side * side
            weights += 2 * 9 * E[s - 1] * E[s]
        px = B * side * side
        for _ in range(depths[s]):
            flops += px * E[s] * 2 * 8 * E[s]
            weights += 2 * 8 * E[s] * E[s]
            if s < 2:
                flops += px * E[s] * (2 * 49 + 2 * E[s])
                weights += 2 * E[s] * E[s]
            else:
                flops += px * E[s] * 2 * 9 * 5 + _mixer_flops("gated", B, T, side, side, E[s], ksp=0 if T == 1 else 3)
                weights += 2 * 3 * E[s] * E[s]
    return {"bytes": 2 * B * c["hw"] ** 2 * 3 + weights + 4 * (E[3] + B) * 1000,
            "flops": flops + B * 2 * E[3] * 1000}


def tolerance(case):
    """bfloat16 activations: 1e-2.  float32 with sums of up to a few thousand terms, a recurrence over
    T and normalisations of spectra behind them: 3e-5."""
    if case["kind"] == "shvit":
        return {"rel": 1e-2}
    return {"rel": 3e-5}
