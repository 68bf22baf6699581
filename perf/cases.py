"""Performance cases of vtpack_b200: what programs that use this framework have it do, through its public
entry points, with the sizes, data types and options they use it with.

* ``layer``     one DGE encoder layer (``Block.forward``) with given gates, as in the layer benchmark
* ``deit``      eval forward of a DeiT+DGE classifier: one image, ordinary batches, a full GPU batch, other resolutions
* ``pvt``       eval forward of a PVT+DGE classifier
* ``train``     one training-mode DeiT+DGE layer with sparse training: forward and backward
* ``bilinear``  the deformable PVT's bilinear-sampling attention: forward and its three gradients

Weights are random (normal, std 0.02, cut at two sigma; router bias 0), images and tokens N(0,1): trained
checkpoints and ImageNet are not part of the repository.
"""
import math

import torch

from vtpack_b200.layers import bilinear_attention
from vtpack_b200.models.dge import deit_dge, pvt_dge

SPLITS = [4, 2, 1]
DEIT = {"tiny": (192, 3), "small": (384, 6), "base": (768, 12)}           # channels, heads
PVT = {"tiny": pvt_dge.pvt_dge_s124_tiny_256, "small": pvt_dge.pvt_dge_s124_small_256}
PVT_STAGES = [(64, 4, 8, 8), (128, 8, 8, 4), (320, 16, 4, 2), (512, 32, 4, 1)]   # channels, stride, MLP ratio, reduction
PVT_DEPTHS = {"tiny": (2, 2, 2, 2), "small": (3, 4, 6, 3)}
DTYPE = {"bf16": torch.bfloat16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp32": 4}
CLASSES = 1000


def listed():
    return [
        # the smallest call: one DeiT-Ti layer in fp32 on two images, the reference's own data type
        dict(name="layer_tiny_fp32_b2", kind="layer", size="tiny", grid=16, batch=2, dtype="fp32", fine=0.33),
        # one image through the smallest model: what an interactive service waits for
        dict(name="deit_tiny_b1", kind="deit", size="tiny", img=256, batch=1, dtype="bf16", images="fp32", replay=False),
        # a small dynamic batch of a service, an odd number of images
        dict(name="deit_small_b7", kind="deit", size="small", img=256, batch=7, dtype="bf16", images="fp32", replay=False),
        # the headline workload: bulk inference, replayed as a CUDA graph
        dict(name="deit_small_b256", kind="deit", size="small", img=256, batch=256, dtype="bf16", images="fp32", replay=True),
        # the largest DeiT, an odd batch, images that arrive in bf16
        dict(name="deit_base_b33", kind="deit", size="base", img=256, batch=33, dtype="bf16", images="bf16", replay=False),
        # high resolution: 1025 keys per image
        dict(name="deit_small_512px_b24", kind="deit", size="small", img=512, batch=24, dtype="bf16", images="fp32", replay=False),
        # evaluation in the reference's data type
        dict(name="deit_small_fp32_b12", kind="deit", size="small", img=256, batch=12, dtype="fp32", images="fp32", replay=False),
        # a pyramid model on a few images, and in bulk
        dict(name="pvt_tiny_b3", kind="pvt", size="tiny", img=256, batch=3, dtype="bf16", images="fp32", replay=False),
        dict(name="pvt_small_b96", kind="pvt", size="small", img=256, batch=96, dtype="bf16", images="fp32", replay=False),
        # a training step of one DeiT-S layer with the sampled grains only
        dict(name="train_small_b48", kind="train", size="small", grid=16, batch=48, dtype="bf16"),
        # deformable attention, first stage: 64 x 64 map, 64 channels per head, 9 points; forward + backward
        dict(name="bilinear_point_bf16", kind="bilinear", mode="point", maps=32, height=64, width=64, channels=64, points=9,
             dtype="bf16"),
        # the channel mode in fp32 on a ragged map
        dict(name="bilinear_channel_fp32", kind="bilinear", mode="channel", maps=10, height=20, width=27, channels=48,
             points=4, dtype="fp32"),
    ]


# Upper bounds of a drawn case's operations: those of the largest listed case of its kind and data type.
_MAX_FLOPS = {("layer", "bf16"): 1.4e11, ("layer", "fp32"): 3e10, ("deit", "bf16"): 1.6e12, ("deit", "fp32"): 7.5e10,
              ("pvt", "bf16"): 4.5e11, ("pvt", "fp32"): 5e10, ("train", "bf16"): 7.5e10, ("train", "fp32"): 7.5e10,
              ("bilinear", "bf16"): 2.3e9, ("bilinear", "fp32"): 2.3e9}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) if hi > lo else int(lo)


def draw(rng):
    kind = rng.choices(["layer", "deit", "pvt", "train", "bilinear"], [2, 8, 4, 3, 3])[0]
    dtype = "bf16" if rng.random() < 0.75 else "fp32"
    if kind == "bilinear":
        case = dict(kind=kind, mode=rng.choice(["point", "channel"]), maps=1, height=_log_int(rng, 7, 64),
                    width=_log_int(rng, 7, 64), channels=rng.choice([32, 48, 64, 96, 128]), points=rng.randint(1, 9), dtype=dtype)
        return dict(case, maps=_log_int(rng, 1, _cap(case, "maps", 64)))
    if kind == "layer":
        case = dict(kind=kind, size=rng.choice(list(DEIT)), grid=rng.choice([16, 16, 24, 32]), batch=1, dtype=dtype,
                    fine=round(rng.uniform(0.0, 1.0), 2))
        return dict(case, batch=_log_int(rng, 1, _cap(case, "batch", 256)))
    if kind == "train":
        case = dict(kind=kind, size=rng.choice(["tiny", "small"]), grid=rng.choice([16, 16, 24]), batch=1, dtype=dtype)
        return dict(case, batch=_log_int(rng, 2, _cap(case, "batch", 96)))
    sizes = DEIT if kind == "deit" else PVT
    case = dict(kind=kind, size=rng.choice(list(sizes)), img=rng.choice([256, 256, 256, 384, 512] if kind == "deit" else [256, 256, 384]),
                batch=1, dtype=dtype, images=rng.choice(["fp32", "fp32", "bf16"]), replay=rng.random() < 0.3)
    return dict(case, batch=_log_int(rng, 1, _cap(case, "batch", 256)))


def _cap(case, axis, most):
    """The largest value of an axis that keeps the case within the operations of the listed ones."""
    return max(1, min(most, int(_MAX_FLOPS[case["kind"], case["dtype"]] / work(dict(case, **{axis: 1}))["flops"])))


# ------------------------------------------------------------------------------------------------ inputs
def _fill(module, gen):
    """Random weights: matrices normal with std 0.02 cut at two sigma, LayerNorm gains around 1, small biases,
    router bias 0 (every grain is picked)."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if not p.is_floating_point():
                continue
            if p.dim() > 1:
                p.normal_(0.0, 0.02, generator=gen).clamp_(-0.04, 0.04)
            elif name.endswith("gate.bias"):
                p.zero_()
            elif name.endswith("weight"):
                p.normal_(1.0, 0.05, generator=gen)
            else:
                p.normal_(0.0, 0.02, generator=gen)
    return module


def _layer(case, gen, dtype):
    dim, heads = DEIT[case["size"]]
    with torch.device("cuda"):
        block = deit_dge.Block(dim, heads, mlp_ratio=4, qkv_bias=True, split_sizes=SPLITS)
    return _fill(block, gen).to(dtype)


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    dtype = DTYPE[case["dtype"]]
    kind = case["kind"]

    def randn(*shape, dt=dtype):
        return torch.randn(*shape, device="cuda", generator=gen).to(dt)

    if kind == "bilinear":
        B, H, W, C, P = (case[k] for k in ("maps", "height", "width", "channels", "points"))
        point = case["mode"] == "point"
        # one query per pixel, its points a few pixels around it as the model's offsets put them
        ys, xs = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
        centre = torch.stack([xs, ys], dim=-1).reshape(1, H * W, 1, 2).float()
        grid = (centre + 3.0 * torch.randn(B, H * W, P, 2, device="cuda", generator=gen)).to(dtype)
        ops = [randn(B, H, W, C), grid, randn(B, H * W, P if point else C)]
        if point:
            ops[2] = ops[2].softmax(dim=-1)
        return dict(kind=kind, mode=case["mode"], operands=[t.requires_grad_(True) for t in ops],
                    grad=randn(B, H * W, C if point else P))
    if kind in ("layer", "train"):
        B, grid = case["batch"], case["grid"]
        block = _layer(case, gen, dtype)
        x = randn(B, grid * grid + 1, DEIT[case["size"]][0])
        if kind == "train":
            block.dge.sparse_train = True
            return dict(kind=kind, block=block.train(), x=x.requires_grad_(True), grad=randn(*x.shape), seed=seed)
        R = grid // 4
        # router logits that put the fraction `fine` of the regions on the finest grain, the rest on the other two
        logits = torch.randn(B, R, R, 3, device="cuda", generator=gen)
        fine = torch.rand(B, R, R, device="cuda", generator=gen) < case["fine"]
        logits[..., 0] = torch.where(fine, 1e4, -1e4)
        return dict(kind=kind, block=block.eval(), x=x, gate=logits)
    with torch.device("cuda"):
        if kind == "deit":
            dim, heads = DEIT[case["size"]]
            model = deit_dge.VisionTransformer(img_size=case["img"], patch_size=16, embed_dim=dim, depth=12, num_heads=heads,
                                               mlp_ratio=4, qkv_bias=True, num_classes=CLASSES, split_sizes=SPLITS)
        else:
            model = PVT[case["size"]]()
    model = _fill(model, gen).to(dtype).eval()
    images = randn(case["batch"], 3, case["img"], case["img"], dt=DTYPE[case["images"]])
    logits = torch.empty(case["batch"], CLASSES, device="cuda") if case["replay"] and kind == "deit" else None
    return dict(kind=kind, model=model, images=images, logits=logits, replay=case["replay"])


# -------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "bilinear":
        out = bilinear_attention(*state["operands"], state["mode"])
        return (out,) + torch.autograd.grad(out, state["operands"], state["grad"])
    if kind == "train":
        block, x = state["block"], state["x"]
        torch.cuda.manual_seed(state["seed"])              # the gate's Gumbel noise
        block.zero_grad(set_to_none=True)
        x.grad = None
        out = block(x)
        out.backward(state["grad"])
        return out.detach(), x.grad, {name: p.grad for name, p in block.named_parameters() if p.requires_grad}
    with torch.no_grad():
        if kind == "layer":
            return state["block"](state["x"], forced_gate=state["gate"])
        if not state["replay"]:
            return state["model"](state["images"])
        if kind == "deit":
            return state["model"].forward_graph(state["images"], state["logits"])
        return state["model"].forward_graph(state["images"])


# ------------------------------------------------------------------------------------- work and tolerance
def _block_flops(tokens, keys, queries, C, mlp, reduced):
    """One encoder layer on one image: q and out projections, reduction, kv projection, attention, MLP."""
    return 2.0 * (2 * queries * C * C + reduced * tokens * C * C + 2 * keys * C * C + 2 * queries * keys * C
                  + 2 * queries * C * mlp * C)


def work(case):
    """Operations of the contractions, and the bytes of inputs (weights among them) and outputs once each."""
    kind, e = case["kind"], BYTES[case["dtype"]]
    if kind == "bilinear":
        B, H, W, C, P = (case[k] for k in ("maps", "height", "width", "channels", "points"))
        n, point = B * H * W, case["mode"] == "point"
        # forward: input, grid, weight, output; backward: those and the output gradient read, three gradients written
        small, out = n * (P if point else C), n * (C if point else P)
        values = (n * C + 2 * n * P + small) * 3 + 2 * out
        return {"bytes": float(values * e), "flops": 30.0 * n * P * C}
    if kind in ("layer", "train"):
        C, G, B = DEIT[case["size"]][0], case["grid"], case["batch"]
        N, R = G * G + 1, (G // 4) ** 2
        fine = case["fine"] if kind == "layer" else 1.0 / 3.0
        q = 1 + R * (16 * fine + 2.5 * (1.0 - fine))               # the other two grains give 4 or 1 queries each
        params = 12 * C * C + 16 * C
        flops = B * _block_flops(N, N, q, C, 4, 0)
        if kind == "layer":
            return {"bytes": float(e * (2 * B * N * C + params)), "flops": flops}
        # backward: two products for each of the forward; tokens and their gradients, parameters and theirs
        return {"bytes": float(e * (4 * B * N * C + 2 * params)), "flops": 3.0 * flops}
    B, img = case["batch"], case["img"]
    flops, params = 0.0, 0.0
    if kind == "deit":
        C, G = DEIT[case["size"]][0], img // 16
        N, q = G * G + 1, 1 + 5.5 * (G // 4) ** 2                  # about 5.5 queries per region with random weights
        flops = B * (2.0 * G * G * 768 * C + 12 * _block_flops(N, N, q, C, 4, 0) + 2.0 * C * CLASSES)
        params = 12 * (12 * C * C + 16 * C) + 768 * C + N * C + C * CLASSES
    else:
        prev = 3
        for (C, stride, mlp, sr), depth in zip(PVT_STAGES, PVT_DEPTHS[case["size"]]):
            G = img // stride
            N = G * G + (1 if sr == 1 else 0)
            keys = N if sr == 1 else (G // sr) ** 2
            q = N - G * G + 7 * (G // 4) ** 2
            k = prev * (16 if prev == 3 else 4)
            flops += B * (2.0 * G * G * k * C + depth * _block_flops(N, keys, q, C, mlp, 1 if sr > 1 else 0))
            params += k * C + N * C + depth * (4 + 2 * mlp + (sr * sr if sr > 1 else 0)) * C * C
            prev = C
        flops += B * 2.0 * prev * CLASSES
        params += prev * CLASSES
    return {"bytes": float(B * 3 * img * img * BYTES[case["images"]] + e * params + 4 * B * CLASSES), "flops": flops}


def tolerance(case):
    """bf16: rounding of every intermediate, over twelve layers and the gates that near-ties flip; fp32: sums in another order."""
    if case["dtype"] == "bf16":
        return {"rel": 0.02 if case["kind"] != "layer" else 0.01}
    return {"rel": 2e-5}
