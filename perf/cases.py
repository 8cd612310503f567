"""Performance cases: what users of this package run, timed through the functions they call.

A case is a dict of plain values.  ``prepare`` makes its inputs on the GPU from a seed, ``run`` is one pass through the
public functions of custom_helper_op_b200: the forward alone (``train`` false: what a depth-inference program calls) or
the forward and the gradients that torch.autograd asks for (``train`` true: a training step's share of this package).
Shapes are those of the package's configurations (custom_helper_op_b200/synth.py), with ragged neighbours of them.
"""
import math

import numpy as np
import torch

from custom_helper_op_b200 import synth
from custom_helper_op_b200.python.ops import custom_helper_ops as ops

SWEEPS = ("cost_volume", "cost_aggregate", "cost_volume_v3")   # fronto-parallel planes: base_plane + offsets
CONVS = ("sparse_conv3d_fast", "sparse_conv3d_transpose_fast")
DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def _sweep(name, op, B, N, H, W, D, C, dtype="float32", reduce="MEAN", groups=1, train=True, inverse=False, spacing=0.0):
    return dict(name=name, op=op, B=B, N=N, H=H, W=W, D=D, C=C, dtype=dtype, reduce=reduce, groups=groups, train=train,
                inverse=inverse, spacing=spacing)


def _conv(name, op, B, H, W, D, Cin, Cout, dtype, strides, train=True):
    """H, W, D: the fine grid; Cin: channels on the fine side of the convolution (its input, or the transposed form's output)."""
    return dict(name=name, op=op, B=B, H=H, W=W, D=D, Cin=Cin, Cout=Cout, dtype=dtype, sh=strides[0], sw=strides[1],
                sd=strides[2], train=train)


def listed():
    return [
        # a small training step (quarter resolution of 256x320, few channels): launches and host work dominate
        _sweep("volume_small_train", "cost_volume", 1, 2, 64, 80, 32, 8),
        # the plane-sweep network's own shape: 1/4 of 512x640, 192 planes, three images
        _sweep("volume_mvsnet_train", "cost_volume", 1, 2, 128, 160, 192, 32),
        # depth inference on a pair of odd-sized images with three source views
        _sweep("volume_ragged_infer", "cost_volume", 2, 3, 117, 149, 67, 16, train=False),
        # one item of the large batch: six source views, 1/4 of 1184x1600, planes uniform in inverse depth, half-width features
        _sweep("volume_large_train", "cost_volume", 1, 6, 296, 400, 256, 32, dtype="bfloat16", inverse=True),
        # the channel-averaged volume with the layers' default reduction
        _sweep("aggregate_min_train", "cost_aggregate", 1, 2, 128, 160, 192, 32, reduce="MIN"),
        # coarse stage of the cascade: per-pixel hypotheses, group correlation
        _sweep("cascade_coarse_train", "cost_volume_v2", 1, 4, 288, 384, 48, 32, dtype="bfloat16", groups=8, spacing=8.0),
        # fine stage of the cascade at inference: full resolution, few hypotheses and channels
        _sweep("cascade_fine_infer", "cost_volume_v2", 1, 4, 1152, 1536, 8, 8, dtype="bfloat16", groups=8, spacing=1.0,
               train=False),
        # best-matching groups instead of aligned ones
        _sweep("group_match_train", "cost_volume_v3", 1, 2, 128, 160, 192, 32, groups=8),
        # warped features of every view, for networks that aggregate them themselves
        _sweep("features_ragged_train", "feature_aggregate", 1, 3, 131, 173, 96, 16),
        # regularisation over a band of nine planes around the coarse depth
        _conv("band_conv_train", "sparse_conv3d_fast", 1, 256, 320, 9, 16, 16, "bfloat16", (1, 1, 1)),
        # the same layer in float32 on an odd-sized image
        _conv("band_conv_f32_train", "sparse_conv3d_fast", 1, 189, 251, 7, 16, 16, "float32", (1, 1, 1)),
        # the up-sampling layer of the band's U-shaped network
        _conv("band_up_train", "sparse_conv3d_transpose_fast", 1, 256, 320, 9, 16, 16, "bfloat16", (2, 2, 2)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        op = rng.choice(("cost_volume",) * 4 + ("cost_volume_v2",) * 3 + ("cost_aggregate", "cost_aggregate", "cost_volume_v3",
                        "feature_aggregate") + CONVS[:1] * 3 + CONVS[1:] * 2)
        train = rng.random() < 0.7
        dtype = rng.choice(("float32", "bfloat16"))
        H = _log(rng, 48, 1152 if op == "cost_volume_v2" else 320)
        W = int(H * rng.uniform(1.1, 1.5))
        if op in CONVS:
            D = rng.randint(5, 17)
            stride = rng.choice(((2, 2, 2), (2, 2, 1))) if op == CONVS[1] else rng.choice(((1, 1, 1),) * 3 + ((2, 2, 2), (2, 2, 1)))
            case = _conv("", op, rng.choice((1, 1, 2)), H, W, D, rng.choice((8, 16, 32)), rng.choice((8, 16, 32)), dtype, stride, train)
        else:
            C = rng.choice((8, 16, 16, 32, 32, 64 if op == "cost_volume" else 32))
            N = rng.choice((1, 2, 2, 3, 4, 4, 5, 6))
            B = rng.choice((1, 1, 1, 2, 3))
            reduce = rng.choice(("MEAN", "MIN" if op in ("cost_aggregate", "cost_volume_v2") else "MEAN"))
            groups = 1
            spacing = 0.0
            D = _log(rng, 16, 256)
            if op == "cost_volume_v2":
                groups = rng.choice((C, C // 2, C // 4))
                D = _log(rng, 8, 64)
                spacing = math.exp(rng.uniform(0.0, math.log(8.0)))
            if op == "cost_volume_v3":
                groups = C // 4
                dtype = "float32"
            case = _sweep("", op, B, N, H, W, D, C, dtype, reduce, groups, train, rng.random() < 0.4, spacing)
        del case["name"]
        biggest = work(listed()[3])
        mine = work(case)
        if mine["bytes"] <= biggest["bytes"] and mine["flops"] <= biggest["flops"] / 2:
            return case


def _smooth(g, B, H, W, centre=700.0, amp=200.0):
    """centre + four random low-frequency sinusoids of total amplitude amp: a smooth depth map [B,H,W]."""
    dev = g.device
    u = torch.rand((B, 4, 4), generator=g, device=dev)
    a = 0.2 + 0.8 * u[..., 0]
    a = a / a.sum(1, keepdim=True) * amp
    ys = (torch.arange(H, device=dev) / H).view(1, 1, H, 1)
    xs = (torch.arange(W, device=dev) / W).view(1, 1, 1, W)
    f, h, p = (u[..., k].view(B, 4, 1, 1) for k in (1, 2, 3))
    return centre + (a.view(B, 4, 1, 1) * torch.sin(2 * math.pi * ((0.5 + 1.5 * f) * xs + (0.5 + 1.5 * h) * ys + p))).sum(1)


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = DTYPES[c["dtype"]]
    B, H, W, D = c["B"], c["H"], c["W"], c["D"]

    def normal(*shape, dtype=torch.float32, scale=1.0):
        return (torch.randn(shape, generator=g, device=dev) * scale).to(dtype)

    if c["op"] in CONVS:
        coarse = (-(-H // c["sh"]), -(-W // c["sw"]), -(-D // c["sd"]))
        up = c["op"] == CONVS[1]
        images = normal(B, *coarse, c["Cout"], dtype=dt, scale=0.1) if up else normal(B, H, W, D, c["Cin"], dtype=dt, scale=0.1)
        filters = normal(3, 3, 3, c["Cin"], c["Cout"], dtype=dt, scale=0.1)
        index = torch.round((_smooth(g, B, H, W) - 500.0) * 63.0 / 400.0)
        base = torch.clamp(index - D // 2, 0, 64 - D).to(torch.int32)[..., None].contiguous()
        grad = normal(B, H, W, D, c["Cin"], dtype=dt) if up else normal(B, *coarse, c["Cout"], dtype=dt)
        return dict(case=c, images=images.requires_grad_(c["train"]), filters=filters.requires_grad_(c["train"]),
                    default=torch.zeros((), dtype=dt, device=dev), base=base, grad=grad if c["train"] else None)

    N, C = c["N"], c["C"]
    Rs, Ts = synth.random_cameras(np.random.default_rng(seed), B, N, H, W)
    s = dict(case=c, ref=normal(B, H, W, C, dtype=dt), src=normal(B, N, H, W, C, dtype=dt),
             Rs=torch.from_numpy(Rs).to(dev, torch.float32), Ts=torch.from_numpy(Ts).to(dev, torch.float32))
    if c["op"] == "cost_volume_v2":
        steps = (torch.arange(D, device=dev) - D / 2.0) * c["spacing"]
        s["depth"] = (_smooth(g, B, H, W)[..., None] + steps).contiguous()
    else:
        if c["inverse"]:
            offs = 1.0 / torch.linspace(1.0 / 400.0, 1.0 / 1200.0, D, device=dev, dtype=torch.float64)
            s["depth"] = torch.zeros((B, H, W, 1), device=dev)
        else:
            offs = torch.arange(D, device=dev, dtype=torch.float64) * (510.0 / max(D - 1, 1))
            s["depth"] = torch.full((B, H, W, 1), 425.0, device=dev)
        s["offsets"] = offs.to(torch.float32).repeat(B, 1)
    if c["train"]:
        shape = {"cost_volume": (B, H, W, D, C), "cost_aggregate": (B, H, W, D), "cost_volume_v3": (B, H, W, D, 1),
                 "cost_volume_v2": (B, H, W, D, c["groups"]), "feature_aggregate": (B, H, W, D, N, C)}[c["op"]]
        s["grad"] = torch.randn(shape, generator=g, device=dev)
    for k in ("ref", "src", "depth"):
        s[k].requires_grad_(c["train"])
    return s


def _forward(s):
    c = s["case"]
    op = c["op"]
    if op == "sparse_conv3d_fast":
        return (ops.sparse_conv3d_fast(s["images"], s["filters"], s["default"], s["base"], strides=(c["sh"], c["sw"], c["sd"])),)
    if op == "sparse_conv3d_transpose_fast":
        return (ops.sparse_conv3d_transpose_fast(s["images"], s["filters"], s["default"], s["base"], (c["H"], c["W"], c["D"]),
                                                 strides=(c["sh"], c["sw"], c["sd"])),)
    if op == "cost_volume_v2":
        return ops.cost_volume_v2(s["ref"], s["src"], s["depth"], s["Rs"], s["Ts"], reduce_method=c["reduce"], groups=c["groups"])
    if op == "cost_volume_v3":
        return ops.cost_volume_v3(s["ref"], s["src"], s["depth"], s["offsets"], s["Rs"], s["Ts"], reduce_method=c["reduce"],
                                  groups=c["groups"])
    if op == "feature_aggregate":
        return ops.feature_aggregate(s["src"], s["depth"], s["offsets"], s["Rs"], s["Ts"])
    f = ops.cost_volume if op == "cost_volume" else ops.cost_aggregate
    return f(s["ref"], s["src"], s["depth"], s["offsets"], s["Rs"], s["Ts"], reduce_method=c["reduce"])


def run(state):
    c = state["case"]
    if not c["train"]:
        with torch.no_grad():
            return list(_forward(state))
    out = _forward(state)
    if c["op"] in CONVS:
        wrt = (state["images"], state["filters"])
    elif c["op"] == "feature_aggregate":
        wrt = (state["src"], state["depth"])
    else:
        wrt = (state["ref"], state["src"], state["depth"])
    grads = torch.autograd.grad(out[0], wrt, state["grad"])
    return [t.detach() for t in out] + list(grads)


def work(case):
    c = case
    e = 2 if c["dtype"] == "bfloat16" else 4
    B, H, W, D = c["B"], c["H"], c["W"], c["D"]
    if c["op"] in CONVS:
        fine = B * H * W * D
        coarse = B * -(-H // c["sh"]) * -(-W // c["sw"]) * -(-D // c["sd"])
        weights = 27 * c["Cin"] * c["Cout"] * e
        once = (fine * c["Cin"] + coarse * c["Cout"]) * e
        macs = coarse * 27 * c["Cin"] * c["Cout"]
        # forward: images, weights, base planes in, output out; gradient: the upstream values in, two gradients out
        if c["train"]:
            return {"bytes": 2 * once + 2 * weights + B * H * W * 4, "flops": 6.0 * macs}
        return {"bytes": once + weights + B * H * W * 4, "flops": 2.0 * macs}
    N, C = c["N"], c["C"]
    vox = B * H * W * D
    feats = B * H * W * C * (N + (c["op"] != "feature_aggregate")) * e
    per_voxel = {"cost_volume": C, "cost_aggregate": 1, "cost_volume_v3": 1, "cost_volume_v2": c["groups"],
                 "feature_aggregate": N * C}[c["op"]]
    mask = 1 if c["reduce"] == "MEAN" else {"cost_volume": C, "cost_aggregate": 1, "cost_volume_v3": 3,
                                             "cost_volume_v2": c["groups"]}.get(c["op"], 1)
    if c["op"] == "feature_aggregate":
        mask = N
    depth = (vox if c["op"] == "cost_volume_v2" else B * H * W) * 4
    nbytes = feats + depth + vox * (per_voxel + mask) * 4
    # a bilinear sample is three multiply-adds a channel; a squared difference or a product with the reference one more
    per = C * (C // (C // c["groups"]) + 3) if c["op"] == "cost_volume_v3" else 4 * C
    flops = 2.0 * vox * N * per
    if c["train"]:
        nbytes += vox * per_voxel * 4 + feats + depth
        # the sample again, its derivative along two image axes, the scatter to four corners, the reference's share
        flops += 2.0 * vox * N * 11 * C
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "bfloat16" and (case["train"] or case["op"] in CONVS):
        return {"rel": 4e-3}   # results rounded to bfloat16
    if case["op"] in CONVS and case["train"]:
        return {"rel": 2e-5}   # filter gradients are 32-bit sums over all voxels
    if case["train"]:
        return {"rel": 2e-5, "max": 2e-3}   # depth gradients are cancelling sums over planes, channels and views
    return {"rel": 1e-5, "max": 1e-3}
