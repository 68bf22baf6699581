"""GPU parity of the bilinear-sampling attention ops (point and channel mode, forward and the three
gradients) against the reference's autograd function (committed fixture) and the CPU restatement."""
import os

import numpy as np
import pytest
import torch

from oracle import bilinear_oracle as BO
from tests.gpu_util import rel_err

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def op():
    from vtpack_b200 import _lib
    from vtpack_b200.layers import bilinear_attention
    _lib.lib()
    return bilinear_attention


def _run(op, inp, grid, weight, grad_out, mode, dtype=torch.float32):
    a, g, w = (t.to(DEV, dtype).requires_grad_(True) for t in (inp, grid, weight))
    y = op(a, g, w, mode)
    return (y.detach(),) + torch.autograd.grad(y, (a, g, w), grad_out.to(DEV, dtype))


@pytest.mark.parametrize("mode", ["point", "channel"])
def test_bilinear_attention_matches_reference(op, golden_dir, mode):
    z = np.load(os.path.join(golden_dir, "bilinear_attention_fp32.npz"))
    inp, grid, weight, grad_out = BO.make_bilinear_inputs(seed=BO.GOLDEN_SEEDS[mode], mode=mode, **BO.GOLDEN_CASE)
    y, gi, gg, gw = _run(op, inp, grid, weight, grad_out, mode)
    for name, t in (("out", y), ("grad_input", gi), ("grad_grid", gg), ("grad_weight", gw)):
        ref = torch.from_numpy(z[f"{mode}_{name}"])
        assert t.shape == ref.shape, name
        assert rel_err(t, ref) < 1e-5, name


@pytest.mark.parametrize("mode", ["point", "channel"])
@pytest.mark.parametrize("B,H,W,C,G,P", [(6, 16, 16, 64, 256, 9), (2, 32, 32, 64, 1024, 4), (3, 7, 5, 33, 35, 1),
                                         (1, 8, 8, 256, 64, 3)])
def test_bilinear_attention_shapes(op, mode, B, H, W, C, G, P):
    """Deformable-PVT shapes (heads folded into the batch, 64 channels per head, one query per pixel)
    and ragged ones (C not a multiple of the warp, a single point, the widest supported C)."""
    inp, grid, weight, grad_out = BO.make_bilinear_inputs(B, H, W, C, G, P, seed=B * 100 + C + P, mode=mode)
    fwd = getattr(BO, f"bilinear_attention_{mode}wise_forward")
    bwd = getattr(BO, f"bilinear_attention_{mode}wise_backward")
    refs = (fwd(inp.double(), grid.double(), weight.double()),) + bwd(grad_out.double(), inp.double(), grid.double(),
                                                                      weight.double())
    for name, t, ref in zip(("out", "grad_input", "grad_grid", "grad_weight"),
                            _run(op, inp, grid, weight, grad_out, mode), refs):
        assert rel_err(t, ref) < 2e-5, name
    # bf16: same inputs rounded once; outputs within bf16 resolution of the float64 result on them
    rb = lambda t: t.bfloat16().double()      # noqa: E731
    refs16 = (fwd(rb(inp), rb(grid), rb(weight)),) + bwd(rb(grad_out), rb(inp), rb(grid), rb(weight))
    got16 = _run(op, inp, grid, weight, grad_out, mode, torch.bfloat16)
    assert rel_err(got16[0].float(), refs16[0]) < 2e-2
    assert rel_err(got16[2].float(), refs16[2]) < 2e-2 and rel_err(got16[3].float(), refs16[3]) < 2e-2
    assert rel_err(got16[1].float(), refs16[1]) < 6e-2          # sums of bf16 atomics


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mode", ["point", "channel"])
@pytest.mark.parametrize("C,shift", [(8, 0), (32, 0), (48, 0), (72, 0), (128, 0), (192, 0), (48, 2), (20, 0), (48, 1)])
def test_bilinear_attention_channel_layouts(op, dtype, mode, C, shift):
    """Every lane layout (4 to 32 lanes per query with 16-byte vectors, whole or part-filled; channel pairs; single
    channels), an instance count that leaves groups of the last warp idle, and operands that start `shift` elements
    behind a 16-byte boundary.  fp32 bound: sums of at most 4 P + log2(C) terms, 2^-24 each; bf16 bounds as above."""
    B, H, W, G, P = 3, 5, 6, 11, 5
    inp, grid, weight, grad_out = BO.make_bilinear_inputs(B, H, W, C, G, P, seed=C + shift, mode=mode)

    def place(t):                              # a contiguous operand at the given offset
        buf = torch.zeros(t.numel() + shift, dtype=dtype, device=DEV)
        buf[shift:] = t.to(DEV, dtype).flatten()
        return buf[shift:].view(t.shape).requires_grad_(True)

    a, gr, w, go = map(place, (inp, grid, weight, grad_out))
    y = op(a, gr, w, mode)
    got = (y.detach(),) + torch.autograd.grad(y, (a, gr, w), go.detach())
    r = [t.to(dtype).double() for t in (inp, grid, weight, grad_out)]
    want = (getattr(BO, f"bilinear_attention_{mode}wise_forward")(*r[:3]),) + \
        getattr(BO, f"bilinear_attention_{mode}wise_backward")(r[3], *r[:3])
    bounds = (2e-5,) * 4 if dtype == torch.float32 else (2e-2, 6e-2, 2e-2, 2e-2)
    for name, t, ref, bound in zip(("out", "grad_input", "grad_grid", "grad_weight"), got, want, bounds):
        assert rel_err(t.float(), ref) < bound, name


@pytest.mark.parametrize("mode", ["point", "channel"])
@pytest.mark.parametrize("C", [64, 48, 20])
@pytest.mark.parametrize("kind", ["noise", "offset 100", "offset 1000", "smooth", "vertical edge", "horizontal edge"])
def test_bilinear_attention_gradients_of_maps_with_common_parts(op, kind, C, mode):
    """fp32 gradients of the points and weights where neighbouring pixels share most of their value, where they differ a lot across an
    edge and where taps outside the map are zero: every component within 2^-24 times the roundings on its way, of the sum of
    what it is formed from.  Derivatives: a difference, its product, up to eight channels of a lane, five steps of shuffles, the
    fractions, products and sum of the two rows, the scale; weight gradients: three roundings a corner weight, four products
    and sums, the channels (point mode) or the points (channel mode)."""
    B, H, W, P = 2, 20, 17, 5
    inp, grid, weight, grad_out = BO.make_bilinear_inputs(B, H, W, C, H * W, P, seed=C, mode=mode)
    if kind.startswith("offset"):
        inp += float(kind.split()[1])
    elif kind == "smooth":
        ys, xs = torch.meshgrid(torch.arange(H) / 7.0, torch.arange(W) / 9.0, indexing="ij")
        inp = 5.0 + torch.sin(xs + ys)[None, :, :, None] + 1e-3 * inp
    elif kind == "vertical edge":
        inp[:, :, W // 2:] += 1000.0
    elif kind == "horizontal edge":
        inp[:, H // 2:] += 1000.0
    r = [t.double() for t in (inp, grid, weight, grad_out)]
    want = getattr(BO, f"bilinear_attention_{mode}wise_backward")(r[3], *r[:3])
    (lt, rt, lb, rb), _, _, tx, ty = BO._taps(*r[:2])
    tx, ty = tx[..., None], ty[..., None]
    up, sc = (r[3], r[2]) if mode == "point" else (r[2], r[3])
    up, sc = up[:, :, None, :].abs(), sc.abs()
    of_x = (up * ((rt - lt).abs() * (1 - ty) + (rb - lb).abs() * ty)).sum(-1) * sc
    of_y = (up * ((lb - lt).abs() * (1 - tx) + (rb - rt).abs() * tx)).sum(-1) * sc
    value = (1 - tx) * (1 - ty) * lt.abs() + tx * (1 - ty) * rt.abs() + (1 - tx) * ty * lb.abs() + tx * ty * rb.abs()
    of_w = (value * up).sum(-1) if mode == "point" else (value * sc[..., None]).sum(2)
    _, _, gg, gw = _run(op, inp, grid, weight, grad_out, mode)
    for name, got, ref, of, roundings in (("x", gg[..., 0], want[1][..., 0], of_x, 20), ("y", gg[..., 1], want[1][..., 1], of_y, 20),
                                          ("weight", gw, want[2], of_w, 20)):
        assert bool(((got.double().cpu() - ref).abs() <= roundings * 2.0 ** -24 * of).all()), name


@pytest.mark.parametrize("G", [10, 150])
def test_bilinear_attention_points_outside_and_non_finite(op, G):
    """Points far outside the map, at infinity or NaN read zero and leave zero gradients; nothing is
    dereferenced out of bounds.  Queries of one block and of several.  The input gradient is a sum of atomic adds in any order: two runs
    differ by a rounding a term at most, of the sum of the terms' magnitudes (the gradient of the operands' magnitudes)."""
    inp, grid, weight, grad_out = BO.make_bilinear_inputs(2, 6, 6, 32, G, 4, seed=5, mode="point")
    grid[0, :, 0, :] = 1e30
    grid[0, :, 1, :] = -1e30
    grid[1, :, 2, 0] = float("inf")
    grid[1, :, 3, 1] = float("nan")
    finite = grid.clone()
    finite[~torch.isfinite(finite) | (finite.abs() > 1e6)] = -3.0          # an equivalent all-outside point
    y, gi, gg, gw = _run(op, inp, grid, weight, grad_out, "point")
    y2, gi2, gg2, gw2 = _run(op, inp, finite, weight, grad_out, "point")
    assert torch.isfinite(y).all() and torch.equal(y, y2) and torch.equal(gg, gg2) and torch.equal(gw, gw2)
    assert not bool(gg[0, :, :2].any()) and not bool(gg[1, :, 2:].any()) and not bool(gw[0, :, :2].any())
    of = _run(op, inp, finite, weight.abs(), grad_out.abs(), "point")[1].double()
    assert bool(((gi - gi2).double().abs() <= 2 * (4 * G) * 2.0 ** -24 * of).all())


@pytest.mark.parametrize("dtype,C,G", [(torch.bfloat16, 32, 64), (torch.float32, 64, 16), (torch.float32, 128, 8)])
def test_bilinear_attention_smallest_backward_uses_the_whole_block(op, dtype, C, G):
    """As many queries as one block holds take about what a few more take (64 of them 41 us when one warp worked them all off, 11 now)."""
    from vtpack_b200 import _lib

    def us(G):
        t = [v.to(DEV, dtype) for v in BO.make_bilinear_inputs(1, 8, 8, C, G, 9, seed=1, mode="point")]
        inp, grid, weight, grad_out = t
        grads = [torch.empty_like(v) for v in t[:3]]
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = float("inf")
        for _ in range(8):
            e[0].record()
            for _ in range(20):
                _lib.check(_lib.lib().vtp_bilinear_attention_backward(
                    grad_out.data_ptr(), inp.data_ptr(), grid.data_ptr(), weight.data_ptr(), *(g.data_ptr() for g in grads),
                    0 if dtype == torch.float32 else 1, 0, 1, 8, 8, C, G, 9, torch.cuda.current_stream().cuda_stream))
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 50)
        return best

    assert us(G) < 1.9 * us(G + G // 4)


def test_dpvt_attention_usage(op):
    """The call sequence of the deformable PVT's attention (dpvt.py:92-115): heads folded into the
    batch, reference points on the pixel grid plus learned offsets, softmax weights, "point" mode."""
    B, H, W, C, heads, P = 2, 8, 8, 128, 2, 4
    N, d = H * W, C // heads
    g = torch.Generator().manual_seed(9)
    v = torch.randn(B, N, heads, d, generator=g).permute(0, 2, 1, 3).reshape(-1, H, W, d)
    mh, mw = torch.meshgrid(torch.linspace(0, H - 1, H), torch.linspace(0, W - 1, W), indexing="ij")
    ref_points = torch.stack([mw, mh], dim=-1).reshape(1, N, 1, 2)
    offsets = torch.randn(B * heads, N, P, 2, generator=g) * 1.5
    weight = torch.randn(B * heads, N, P, generator=g).softmax(-1)
    grid = ref_points + offsets
    want = BO.bilinear_attention_pointwise_forward(v.double(), grid.double(), weight.double())
    got = op(v.to(DEV).contiguous(), grid.to(DEV), weight.to(DEV), "point")
    assert got.shape == (B * heads, N, d) and rel_err(got, want) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sparse_bilinear_attention_packed_queries(dtype):
    """Packed (variable number per image) queries: equal to the dense op on each image's slice, and to
    the CPU restatement; an image without queries and unsorted image indices included."""
    from vtpack_b200.layers import bilinear_attention, sparse_bilinear_attention_pointwise_forward
    B, H, W, C, P = 4, 9, 7, 48, 3
    g = torch.Generator().manual_seed(12)
    inp = torch.randn(B, H, W, C, generator=g)
    batches = torch.tensor([0] * 5 + [3] * 11 + [1] * 2 + [3] * 4)          # image 2 has no query
    L = batches.numel()
    grid = torch.rand(L, P, 2, generator=g) * torch.tensor([W + 3.0, H + 3.0]) - 2.0
    weight = torch.randn(L, P, generator=g)
    rb = (lambda t: t.to(dtype).double())
    want = BO.sparse_bilinear_attention_pointwise_forward(rb(inp), rb(grid), rb(weight), batches)
    got = sparse_bilinear_attention_pointwise_forward(inp.to(DEV, dtype), grid.to(DEV, dtype), weight.to(DEV, dtype),
                                                      batches.to(DEV))
    assert got.shape == (L, C) and got.dtype == dtype
    assert rel_err(got.float(), want) < (1e-5 if dtype == torch.float32 else 2e-2)
    sel = batches == 3
    dense = bilinear_attention(inp[3:4].to(DEV, dtype).contiguous(), grid[sel][None].to(DEV, dtype),
                               weight[sel][None].to(DEV, dtype), "point")[0]
    assert torch.equal(got[sel.to(DEV)], dense)


def test_dpvt_attention_module_matches_reference(golden_dir):
    """The deformable attention module (dpvt.py:51-115) over this library's op: output, input
    gradient and all eight parameter gradients against the reference's own module."""
    from oracle import dge_oracle as O
    from vtpack_b200.models.standard.dpvt import Attention
    z = np.load(os.path.join(golden_dir, "dpvt_attention_fp32.npz"))
    c = O.DPVT_ATTENTION
    att = Attention(c["dim"], num_heads=c["heads"], qkv_bias=True, num_points=c["points"])
    att.load_state_dict(O.dpvt_attention_weights(), strict=True)
    att.to(DEV)
    x = O.randn_seeded((c["batch"], c["H"] * c["W"], c["dim"]), c["token_seed"]).to(DEV).requires_grad_(True)
    y = att(x, c["H"], c["W"])
    (y * O.randn_seeded(tuple(y.shape), c["grad_seed"]).to(DEV)).sum().backward()
    assert rel_err(y, torch.from_numpy(z["out"])) < 1e-5
    assert rel_err(x.grad, torch.from_numpy(z["grad_x"])) < 1e-4
    n = 0
    for name, prm in att.named_parameters():
        assert rel_err(prm.grad, torch.from_numpy(z[f"grad.{name}"])) < 1e-4, name
        n += 1
    assert n == 8


@pytest.mark.parametrize("mode", ["point", "channel"])
@pytest.mark.parametrize("dtype,C", [(torch.float32, 12), (torch.float32, 44), (torch.float32, 64), (torch.float32, 96), (torch.float32, 256),
                                     (torch.bfloat16, 24), (torch.bfloat16, 64), (torch.bfloat16, 88), (torch.bfloat16, 136), (torch.bfloat16, 256)])
@pytest.mark.parametrize("H,W,G", [(28, 48, 28 * 48), (29, 37, 29 * 37), (40, 3, 120), (29, 37, 1000)])
def test_bilinear_attention_of_many_queries_is_that_of_the_general_kernel(op, dtype, mode, C, H, W, G):
    """Enough queries for several vectors a lane (one to three, whole or part-filled), as tiles of pixels, on maps that no tiles fill, narrow maps and
    queries that are not the pixels, against the kernel for single channels (operands one element behind a 16-byte boundary), on maps with
    infinities and NaN off the way of all but a few queries.  Both sum the same terms in other orders: apart by two times n 2^-24 of the sum of
    the terms' magnitudes (n terms), and a rounding of the result in bf16 (of every term that reaches a pixel of grad_input)."""
    P, lanes = 3, 2
    B = -(-16 * 32 * 148 // (lanes * G))
    g = torch.Generator(DEV).manual_seed(C + G)
    ys, xs = torch.arange(G, device=DEV) // W % H, torch.arange(G, device=DEV) % W
    t = [torch.randn(B, H, W, C, device=DEV, generator=g),
         torch.stack([xs, ys], -1)[None, :, None].float() + 3 * torch.randn(B, G, P, 2, device=DEV, generator=g),
         torch.randn(B, G, P if mode == "point" else C, device=DEV, generator=g),
         torch.randn(B, G, C if mode == "point" else P, device=DEV, generator=g)]
    t = [v.to(dtype) for v in t]

    def run(t, shift):
        def place(v):
            buf = torch.zeros(v.numel() + shift, dtype=dtype, device=DEV)
            buf[shift:] = v.flatten()
            return buf[shift:].view(v.shape).requires_grad_(True)
        a, gr, w, go = map(place, t)
        y = op(a, gr, w, mode)
        return [v.double() for v in (y.detach(), *torch.autograd.grad(y, (a, gr, w), go.detach()))]
    got, want, size = run(t, 0), run(t, 1), run([t[0].abs(), t[1], t[2].abs(), t[3].abs()], 1)
    sc, up = (t[2], t[3]) if mode == "point" else (t[3], t[2])
    size[2] = 2 * float(t[0].abs().max()) * (sc.double().abs() * up.double().abs().sum(-1, keepdim=True))[..., None]
    x0 = t[1].double().floor().long()
    hits = torch.zeros(B * H * W, device=DEV)
    for dx in (0, 1):
        for dy in (0, 1):
            x, y = x0[..., 0] + dx, x0[..., 1] + dy
            ok = (x >= 0) & (x < W) & (y >= 0) & (y < H)
            at = (torch.arange(B, device=DEV)[:, None, None] * H + y) * W + x
            hits.index_add_(0, at[ok], torch.ones_like(at[ok], dtype=torch.float32))
    hits = hits.view(B, H, W, 1)
    # two results on either side of a rounding boundary are a unit of the last place apart, 2^-7 of a bf16 number at most
    eps = 2.0 ** -7 if dtype is torch.bfloat16 else 0.0
    for name, a, b, of, n in zip(("out", "grad_input", "grad_grid", "grad_weight"), got, want, size, (C + 4 * P + 8, hits + 4, C + 8, C + 4 * P + 8)):
        bound = (2 * n * 2.0 ** -24 + (eps * (hits + 1) if name == "grad_input" else 0)) * of + eps * torch.maximum(a.abs(), b.abs())
        assert bool(((a - b).abs() <= bound + 1e-30).all()), name
    t[0][0, 1, 1, 0], t[0][0, 2, 2, C - 1] = float("inf"), float("nan")
    for name, a, b in zip(("out", "grad_input", "grad_grid", "grad_weight"), run(t, 0), run(t, 1)):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)), name


@pytest.mark.parametrize("mode", ["point", "channel"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,W,G,C", [(36, 28, 48, 28 * 48, 64), (160, 28, 32, 28 * 32, 64), (36, 29, 37, 29 * 37, 64), (2, 29, 37, 29 * 37, 64), (36, 29, 37, 1000, 136), (60, 40, 3, 120, 88),
                                       (2, 7, 9, 60, 48)])
def test_bilinear_attention_is_exact_where_its_sums_are(op, dtype, mode, B, H, W, G, C):
    """Small whole numbers, and points half a pixel from the pixels: every product and sum is a multiple of 1/8 below 2^21, exact in fp32, and
    every sum at a pixel below 32 (at most 100 terms of a quarter), exact in bf16 too.  So all four results are the float64 ones,
    rounded once: a corner left out or weighted wrongly anywhere shows."""
    P = 3
    g = torch.Generator(DEV).manual_seed(C + G)

    def whole(n, *shape):
        return torch.randint(-n, n + 1, shape, device=DEV, generator=g).double()
    ys, xs = torch.arange(G, device=DEV) // W % H, torch.arange(G, device=DEV) % W
    point = mode == "point"
    a = whole(3, B, H, W, C)
    grid = torch.stack([xs, ys], -1)[None, :, None].double() + whole(3, B, G, P, 2) + 0.5
    w, go = whole(1, B, G, P if point else C), whole(1, B, G, C if point else P)
    a64, grid64, w64 = (t.clone().requires_grad_(True) for t in (a, grid, w))
    base = grid64.detach().floor()
    t = grid64 - base
    val = 0.0
    for dx in (0, 1):
        for dy in (0, 1):
            x, y = base[..., 0].long() + dx, base[..., 1].long() + dy
            ok = (x >= 0) & (x < W) & (y >= 0) & (y < H)
            at = (torch.arange(B, device=DEV)[:, None, None] * H + y.clamp(0, H - 1)) * W + x.clamp(0, W - 1)
            share = (t[..., 0] if dx else 1 - t[..., 0]) * (t[..., 1] if dy else 1 - t[..., 1])
            val = val + (a64.view(-1, C)[at] * ok[..., None]) * share[..., None]
    y64 = (val * w64[..., None]).sum(2) if point else (val * w64[:, :, None]).sum(3)
    want = (y64.detach(),) + torch.autograd.grad(y64, (a64, grid64, w64), go)
    assert float(want[1].abs().max()) < 32
    got = _run(op, a, grid, w, go, mode, dtype)
    for name, x, y in zip(("out", "grad_input", "grad_grid", "grad_weight"), got, want):
        assert torch.equal(x, y.to(dtype)), name


@pytest.mark.parametrize("mode", ["point", "channel"])
@pytest.mark.parametrize("dtype,C", [(torch.float32, 256), (torch.float32, 260), (torch.float32, 400), (torch.bfloat16, 512), (torch.bfloat16, 520),
                                     (torch.bfloat16, 776)])
def test_bilinear_attention_of_the_widest_rows(op, dtype, mode, C):
    """The forward of rows of 64 and of more 16-byte vectors, which a warp walks through, against the kernel for single channels (operands one
    element behind a 16-byte boundary): the same terms in other orders, apart by two times n 2^-24 of the sum of their magnitudes
    and a rounding of the result in bf16."""
    B, H, W, P = 3, 9, 11, 4
    g = torch.Generator(DEV).manual_seed(C)
    G = H * W
    t = [torch.randn(B, H, W, C, device=DEV, generator=g), 12 * torch.rand(B, G, P, 2, device=DEV, generator=g) - 1,
         torch.randn(B, G, P if mode == "point" else C, device=DEV, generator=g)]
    t = [v.to(dtype) for v in t]

    def run(t, shift):
        moved = []
        for v in t:
            buf = torch.zeros(v.numel() + shift, dtype=dtype, device=DEV)
            buf[shift:] = v.flatten()
            moved.append(buf[shift:].view(v.shape))
        return op(*moved, mode).double()
    got, want, size = run(t, 0), run(t, 1), run([t[0].abs(), t[1], t[2].abs()], 1)
    n, eps = C + 4 * P + 8, 2.0 ** -7 if dtype is torch.bfloat16 else 0.0
    assert bool(((got - want).abs() <= 2 * n * 2.0 ** -24 * size + eps * torch.maximum(got.abs(), want.abs())).all())
