"""GPU parity of the block and model forwards (one C-ABI call each) against the golden
fixtures made by the reference's Python modules and against the CPU oracle."""
import os

import numpy as np
import pytest
import torch

from tests.gpu_util import O, kernels_of, rel_err

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _block(C, h, sd, dtype):
    from vtpack_b200.models.dge.deit_dge import Block
    blk = Block(C, h, mlp_ratio=4, qkv_bias=True, norm_layer=lambda d: torch.nn.LayerNorm(d, eps=1e-6),
                split_sizes=[4, 2, 1])
    blk.load_state_dict(O.block_weights(sd, 0), strict=True)
    return blk.eval().to(device=DEV, dtype=dtype)


def test_layer_fp32_golden(golden_dir):
    """Benchmark configuration 1: one DeiT-Ti DGE layer, fp32, B=2, injected gate logits; fp32
    tolerance 1e-4 relative."""
    g = np.load(os.path.join(golden_dir, "layer_tiny_fp32.npz"))
    sd = O.make_state_dict(192, 1, 3, seed=0)
    x = O.make_tokens(2, 257, 192, seed=1)
    gate = O.make_gate_logits(2, 4, 4, 3, seed=2)
    blk = _block(192, 3, sd, torch.float32)
    out = blk(x.to(DEV), forced_gate=gate)
    assert blk.dge.states["batches_device"].tolist() == g["batch_lengths"].tolist()
    assert rel_err(out, torch.from_numpy(g["out"])) < 1e-4
    # the op-by-op path through vtpack_b200.layers gives the same (router free-running there)
    blk.dge.router.gate.weight.data.zero_()
    out2 = blk.forward_unfused(x.to(DEV))       # zero gate weights -> all logits equal -> grain 0 everywhere
    ref2 = O.dge_block_forward(x, {**O.block_weights(sd, 0), "dge.router.gate.weight": torch.zeros(3, 192)},
                               3, (4, 2, 1))
    assert rel_err(out2, ref2) < 1e-4


@pytest.mark.parametrize("fine_bias", [-1e4, 0.0, 1e4])
def test_layer_fp32_vs_oracle(fine_bias):
    sd = O.make_state_dict(384, 1, 6, seed=3)
    x = O.make_tokens(3, 257, 384, seed=4)
    gate = O.make_gate_logits(3, 4, 4, 3, seed=5, fine_bias=fine_bias)
    ref = O.dge_block_forward(x, O.block_weights(sd, 0), 6, (4, 2, 1), forced_gate=gate)
    out = _block(384, 6, sd, torch.float32)(x.to(DEV), forced_gate=gate)
    assert rel_err(out, ref) < 1e-4


def test_layer_free_running_gate_fp32():
    sd = O.make_state_dict(192, 1, 3, seed=6)
    x = O.make_tokens(4, 257, 192, seed=7)
    tr = {}
    ref = O.dge_block_forward(x, O.block_weights(sd, 0), 3, (4, 2, 1), trace=tr)
    blk = _block(192, 3, sd, torch.float32)
    out = blk(x.to(DEV))
    assert blk.dge.states["batches_device"].tolist() == tr["batches"].tolist()
    assert rel_err(out, ref) < 1e-4
    assert rel_err(blk.forward_unfused(x.to(DEV)), ref) < 1e-4
    assert torch.equal(blk.dge.states["batches"], tr["batches"])


def test_all_fine_equals_dense_block_fp32():
    sd = O.make_state_dict(192, 1, 3, seed=8)
    x = O.make_tokens(2, 257, 192, seed=9)
    gate = torch.zeros(2, 4, 4, 3)
    gate[..., 0] = 1
    blk = _block(192, 3, sd, torch.float32)
    a = blk(x.to(DEV), forced_gate=gate)
    b = blk(x.to(DEV), dense=True)
    ref = O.dense_block_forward(x, O.block_weights(sd, 0), 3)
    assert rel_err(a, ref) < 1e-4 and rel_err(b, ref) < 1e-4


@pytest.mark.parametrize("C,B,mlp_ratio,special", [
    (256, 1, 0.84375, False),       # 216 hidden channels: a reduction that is not whole k-blocks; two rows of tiles and one row more
    (256, 2, 4.0, True), (256, 5, 1.65625, False), (256, 40, 1.0, False),
    (384, 1, 4.0, False), (384, 12, 4.0, False), (384, 4, 4.0, True),
    (768, 1, 4.0, False), (768, 2, 4.0, True),
])
def test_block_fp32_on_terms_vs_dense_block(C, B, mlp_ratio, special):
    """An fp32 block's Linears and attention take their operands as three bf16 terms, split by the kernels in front of them; the
    dense block's Linears split fp32 rows themselves and its attention runs on CUDA cores.  With every region at the finest grain
    the two blocks are the same function; they differ by the attention's rounding only, some 2^-22 of a row's largest value
    (probabilities with errors of a few 2^-24, sums of 257 of them), carried through two Linears.  Where operands or sums are
    infinite, NaN, near the largest or subnormal the same values have to be infinite or NaN."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.deit_dge import Block
    torch.manual_seed(C + B)
    blk = Block(C, C // 64, mlp_ratio=mlp_ratio, qkv_bias=True, split_sizes=[4, 2, 1]).to(DEV).eval()
    x = torch.randn(B, 257, C, device=DEV)
    if special:
        with torch.no_grad():
            w1, w2 = blk.mlp.fc1.weight, blk.mlp.fc2.weight
            w1[5, 3], w1[64, 7], w1[70] = 2.0 ** 113, -3.4e38, 1e-41        # (a row of subnormal numbers)
            w2[9, 2], w2[10, 1], w2[11, 0] = float("inf"), float("nan"), 2.0 ** 111
            blk.attn.proj.weight[17, 5] = -float("inf")
        x[0, 40, 3] = 1e30
    gate = torch.zeros(B, 4, 4, 3)
    gate[..., 0] = 1
    with torch.no_grad():
        # (the cls row goes through the unpool's sum, ref + (q - comp))
        a, b = blk(x, forced_gate=gate)[:, 1:], blk(x, dense=True)[:, 1:]
    assert _lib.device_status() == 0
    assert bool(torch.isfinite(a).all()) != special
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    fin = torch.isfinite(b)
    assert torch.equal(a[~fin & ~a.isnan()], b[~fin & ~b.isnan()])
    scale = torch.where(fin, b, 0.0).double().abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)
    assert float((torch.where(fin, a - b, 0.0).double().abs() / scale).max()) < 2e-6


@pytest.mark.parametrize("n_grid,heads,special", [(4, 1, ""), (8, 2, ""), (12, 3, "inf key"), (16, 2, "nan value"), (16, 6, "huge"),
                                                  (20, 1, "minus inf"), (24, 2, ""), (32, 1, "huge")])
def test_attention_fp32_on_terms(n_grid, heads, special):
    """The fp32 attention of a block at 17 to 1025 keys (one key behind whole blocks of 64, one to four chunks of up to five
    blocks), 1 to 1025 queries an image, in float64 and, where scores or values are infinite, NaN or overflow the terms'
    sums, as the CUDA-core kernel has them (the dense block)."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.deit_dge import Block
    torch.manual_seed(n_grid)
    C, B, N = 64 * heads, 3, n_grid * n_grid + 1
    blk = Block(C, heads, mlp_ratio=1.0, qkv_bias=True, split_sizes=[4, 2, 1]).to(DEV).eval()
    with torch.no_grad():
        blk.attn.q.weight *= 8          # (scores that spread over some units)
        blk.attn.kv.weight *= 4
    x = torch.randn(B, N, C, device=DEV)
    gate = torch.zeros(B, n_grid // 4, n_grid // 4, 3)
    gate[0, ..., 2], gate[1, ..., 0], gate[2, ..., 1] = 1, 1, 1
    kv = blk.attn.kv
    with torch.no_grad():
        if special == "inf key":
            kv.bias[3] = float("inf")
        elif special == "nan value":
            kv.bias[C + 5] = float("nan")
        elif special == "huge":
            kv.bias[C + 7], kv.bias[2] = 2.0 ** 118, 2.0 ** 97
            blk.attn.q.bias[2] = 1e-3
        elif special == "minus inf":
            kv.bias[1], blk.attn.q.bias[1] = -float("inf"), 9.0
        out = blk(x, forced_gate=gate)
        assert _lib.device_status() == 0
        if special:
            fine = torch.zeros(B, n_grid // 4, n_grid // 4, 3)
            fine[..., 0] = 1
            a, b = blk(x, forced_gate=fine)[:, 1:], blk(x, dense=True)[:, 1:]
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
            fin = torch.isfinite(b)
            scale = torch.where(fin, b, 0.0).double().abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)
            assert float((torch.where(fin, a - b, 0.0).double().abs() / scale).max()) < 1e-5
        else:
            w = {k: v.double().cpu() for k, v in blk.state_dict().items()}
            ref = O.dge_block_forward(x.double().cpu(), w, heads, (4, 2, 1), forced_gate=gate.double(), eps=1e-5)
            assert rel_err(out, ref) < 2e-6


def _block_us(blk, x, gate, n):
    best = float("inf")
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    with torch.no_grad():
        blk(x, forced_gate=gate)
        for _ in range(4):
            e[0].record()
            for _ in range(n):
                blk(x, forced_gate=gate)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 1e3 / n)
    return best


def test_block_fp32_with_a_nan_weight_takes_little_longer():
    """One NaN in fc2's weights makes a column of every row one that is worked out again from the decoded operands: that takes two or
    three times a finite block (by scalar loads, a row at a time: 45 times)."""
    from vtpack_b200.models.dge.deit_dge import Block
    torch.manual_seed(0)
    blk = Block(384, 6, mlp_ratio=4, qkv_bias=True, split_sizes=[4, 2, 1]).to(DEV).eval()
    x, gate = torch.randn(12, 257, 384, device=DEV), torch.randn(12, 4, 4, 3, device=DEV)
    finite = _block_us(blk, x, gate, 20)
    with torch.no_grad():
        blk.mlp.fc2.weight[9, 2] = float("nan")
    assert _block_us(blk, x, gate, 5) < 12 * finite


def test_block_fp32_with_a_nan_among_the_values_takes_little_longer():
    """A NaN in v's bias makes every row of the attention, and of the Linears behind it, one that is worked out again: 14 times a finite
    block (41 times with every lane decoding all keys for itself)."""
    from vtpack_b200.models.dge.deit_dge import Block
    torch.manual_seed(0)
    blk = Block(384, 6, mlp_ratio=4, qkv_bias=True, split_sizes=[4, 2, 1]).to(DEV).eval()
    x, gate = torch.randn(12, 257, 384, device=DEV), torch.randn(12, 4, 4, 3, device=DEV)
    finite = _block_us(blk, x, gate, 20)
    with torch.no_grad():
        blk.attn.kv.bias[384 + 5] = float("nan")
    assert _block_us(blk, x, gate, 5) < 27 * finite


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("what", ["block", "dense block", "pvt stage", "model"])
def test_workspace_on_any_16_byte_boundary(what, dtype, monkeypatch):
    """A workspace has to lie on a 16-byte boundary and be as long as the library says: one that begins 16 bytes behind a 32-byte
    boundary gives the same bits, nothing is refused and nothing is written around it."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import deit_dge, pvt_dge
    torch.manual_seed(5)
    if what == "model":
        net = deit_dge.VisionTransformer(img_size=256, patch_size=16, embed_dim=128, depth=2, num_heads=2, mlp_ratio=2, qkv_bias=True,
                                         num_classes=16, split_sizes=[4, 2, 1])
        args = (torch.randn(2, 3, 256, 256),)
    elif what == "pvt stage":
        net = pvt_dge.Block(128, 2, mlp_ratio=2, qkv_bias=True, sr_ratio=2, split_sizes=[4, 2, 1])
        args = (torch.randn(2, 32 * 32, 128), 32, 32)                         # 256 keys
    else:
        net = deit_dge.Block(128, 2, mlp_ratio=2, qkv_bias=True, split_sizes=[4, 2, 1])
        args = (torch.randn(2, 257, 128),)
    net = net.to(DEV, dtype).eval()
    args = tuple(a.to(DEV, dtype) if torch.is_tensor(a) else a for a in args)
    kwargs = {"dense": True} if what == "dense block" else {}
    with torch.no_grad():
        want = net(*args, **kwargs)
    taken = []

    def shifted(device, nbytes, use="block"):
        buf = torch.full((nbytes + 64 + 32,), 0xA5, dtype=torch.uint8, device=device)
        at = (16 - buf.data_ptr()) % 32
        taken.append((buf, at, nbytes))
        return buf[at:at + nbytes]

    for module in (deit_dge, pvt_dge):
        monkeypatch.setattr(module, "scratch", shifted)
    with torch.no_grad():
        got = net(*args, **kwargs)
    assert _lib.device_status() == 0
    assert taken and torch.equal(got, want)
    for buf, at, nbytes in taken:
        assert (buf.data_ptr() + at) % 32 == 16
        assert bool((buf[:at] == 0xA5).all()) and bool((buf[at + nbytes:] == 0xA5).all())


@pytest.mark.parametrize("B", [33, 256, 257])
def test_block_fp32_items_of_runs_of_images(B):
    """The items of the fp32 attention are listed in three ways, for up to 32, up to 256 and more images: an image's bits are those
    it has in a batch of 16."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.deit_dge import Block
    torch.manual_seed(B)
    blk = Block(64, 1, mlp_ratio=1.0, qkv_bias=True, split_sizes=[4, 2, 1]).to(DEV).eval()
    x = torch.randn(B, 145, 64, device=DEV)
    gate = torch.eye(3)[torch.randint(0, 3, (B, 3, 3))]
    with torch.no_grad():
        whole = blk(x, forced_gate=gate)
        parts = torch.cat([blk(x[i:i + 16].contiguous(), forced_gate=gate[i:i + 16]) for i in range(0, B, 16)])
    assert _lib.device_status() == 0
    assert torch.equal(whole, parts)


def test_block_fp32_more_images_than_one_attention_launch_takes():
    """The fp32 attention on tensor cores lists the items of up to 4000 images in a launch: images on both sides of that number have the
    bits they have in a batch of their own."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.deit_dge import Block
    torch.manual_seed(1)
    blk = Block(64, 1, mlp_ratio=1.0, qkv_bias=True, split_sizes=[4, 2, 1]).to(DEV).eval()
    B = 4007
    x = torch.randn(B, 145, 64, device=DEV)
    gate = torch.eye(3)[torch.randint(0, 3, (B, 3, 3))]
    with torch.no_grad():
        whole = blk(x, forced_gate=gate)
        for i in (0, 2000, 3992, 4000):
            n = min(8, B - i)
            assert torch.equal(blk(x[i:i + n].contiguous(), forced_gate=gate[i:i + n]), whole[i:i + n]), i
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B", [1, 12])
@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("C,sr", [(128, 1), (384, 1), (128, 2)])
def test_block_fp32_weights_written_directly_in_front(C, sr, forced, B):
    """The matrices of an fp32 block are split by CTAs that do not wait for the kernel in front of theirs: a call that follows the kernels
    which write its parameters, without anything between them, uses what they wrote."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import deit_dge, pvt_dge
    torch.manual_seed(C + B)
    if sr == 1:
        blk, n, args = deit_dge.Block(C, C // 64, mlp_ratio=4, qkv_bias=True, split_sizes=[4, 2, 1]), 257, ()
    else:
        blk, n, args = pvt_dge.Block(C, C // 64, mlp_ratio=4, qkv_bias=True, sr_ratio=sr, split_sizes=[4, 2, 1]), 256, (16, 16)
    blk = blk.to(DEV).eval()
    params = [p for p in blk.parameters() if p.is_floating_point()]
    x = torch.randn(B, n, C, device=DEV)
    kw = {"forced_gate": torch.randn(B, 4, 4, 3, device=DEV)} if forced else {}
    sets = [[torch.randn_like(p) * 0.05 for p in params] for _ in range(3)]
    outs, want = [], []
    with torch.no_grad():
        for s in sets:
            for p, v in zip(params, s):
                p.copy_(v)
            torch.cuda.synchronize()
            want.append(blk(x, *args, **kw))
            torch.cuda.synchronize()
        for i in range(120):
            if i % 2:
                torch._foreach_copy_(params, sets[i % 3])
            else:                                             # one kernel a parameter, another one last each time
                k = i // 2 % len(params)
                for p, v in list(zip(params, sets[i % 3]))[k + 1:] + list(zip(params, sets[i % 3]))[:k + 1]:
                    p.copy_(v)
            outs.append(blk(x, *args, **kw))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert not torch.equal(want[0], want[1])
    for i, out in enumerate(outs):
        assert torch.equal(out, want[i % 3]), i


def test_layer_512px_skewed_fp32():
    """32x32 grid (N=1025, 64 regions); even images all-coarse, odd all-fine."""
    sd = O.make_state_dict(128, 1, 2, img_size=512, seed=10)
    x = O.make_tokens(4, 1025, 128, seed=11)
    gate = torch.zeros(4, 8, 8, 3)
    gate[0::2, ..., 2] = 1e4
    gate[1::2, ..., 0] = 1e4
    ref = O.dge_block_forward(x, O.block_weights(sd, 0), 2, (4, 2, 1), forced_gate=gate)
    blk = _block(128, 2, sd, torch.float32)
    out = blk(x.to(DEV), forced_gate=gate)
    assert blk.dge.states["batches_device"].tolist() == [65, 1025, 65, 1025]
    assert rel_err(out, ref) < 1e-4


@pytest.mark.parametrize("cuda_cores,fold", [(True, False), (False, False), (False, True)])
def test_layer_bf16_vs_fp32_oracle(cuda_cores, fold):
    """bf16 device path vs fp32 math on the bf16-rounded weights and input; with the
    tcgen05 kernels both with explicit LayerNorms and with LayerNorm folded into the GEMMs."""
    from vtpack_b200 import _lib
    sd = O.round_bf16(O.make_state_dict(384, 1, 6, seed=12))
    g = torch.Generator().manual_seed(15)
    for k in ("norm1", "norm2"):     # non-trivial LayerNorm affine so that folding is exercised
        sd[f"blocks.0.{k}.weight"] = (1 + 0.2 * torch.randn(384, generator=g)).bfloat16().float()
        sd[f"blocks.0.{k}.bias"] = (0.2 * torch.randn(384, generator=g)).bfloat16().float()
    x = (O.make_tokens(4, 257, 384, seed=13) + 0.5).bfloat16().float()
    gate = O.make_gate_logits(4, 4, 4, 3, seed=14)
    ref = O.dge_block_forward(x, O.block_weights(sd, 0), 6, (4, 2, 1), forced_gate=gate)
    blk = _block(384, 6, sd, torch.bfloat16)
    blk.fold_layernorm = fold
    blk.flags = _lib.FLAG_CUDA_CORES if cuda_cores else 0
    out = blk(x.bfloat16().to(DEV), forced_gate=gate)
    assert _lib.device_status() == 0
    assert float((out.float().cpu() - ref).abs().max()) < 6e-2      # |x| ~ 4: one bf16 ulp is 3e-2
    assert rel_err(out.float(), ref) < 1.5e-2


def _model(kind, sd, dtype, depth=12, flags=0, img_size=256):
    from vtpack_b200.models.dge import deit_dge
    cfg = O.MODEL_CONFIGS[kind]
    m = deit_dge.VisionTransformer(img_size=img_size, patch_size=16, embed_dim=cfg["embed_dim"], depth=depth,
                                   num_heads=cfg["num_heads"], mlp_ratio=4, qkv_bias=True, split_sizes=[4, 2, 1])
    m.load_state_dict(sd, strict=True)
    m.flags = flags
    return m.eval().to(device=DEV, dtype=dtype)


def test_model_fp32_golden(golden_dir):
    """Full DeiT-Ti+DGE, fp32, free-running router: logits, per-layer query counts."""
    g = np.load(os.path.join(golden_dir, "model_tiny_fp32.npz"))
    sd = O.make_state_dict(192, 12, 3, seed=0)
    m = _model("tiny", sd, torch.float32)
    logits = m(O.make_images(2, 256, seed=1).to(DEV))
    assert g["gate_margin"].min() > 1e-5        # no near-tie in the fixture: counts must match exactly
    assert np.array_equal(m.last_counts.cpu().numpy(), g["batch_lengths"])
    assert rel_err(logits, torch.from_numpy(g["logits"])) < 1e-4
    # MAC accounting of the same forward, from the counts the kernels left on the device
    comp = m.complexity(O.make_images(2, 256, seed=1))
    assert comp["static"].is_cuda and comp["dynamic"].is_cuda
    assert float(comp["static"]) == float(g["comp_static"])
    assert float(comp["dynamic"]) == float(g["comp_dynamic"])


@pytest.mark.parametrize("cuda_cores", [True, False])
def test_model_bf16_logits(cuda_cores):
    """Benchmark configuration 2 at reduced batch: DeiT-Ti+DGE bf16 vs the fp32 oracle on
    bf16-rounded weights; logits max-abs <= 2e-2, top-1 agreement reported."""
    from vtpack_b200 import _lib
    B = 16
    sd = O.round_bf16(O.make_state_dict(192, 12, 3, seed=0))
    img = O.make_images(B, 256, seed=1)
    tr = []
    ref = O.deit_dge_forward(img, sd, 12, 3, (4, 2, 1), trace=tr)
    m = _model("tiny", sd, torch.bfloat16, flags=_lib.FLAG_CUDA_CORES if cuda_cores else 0)
    logits = m(img.to(DEV)).cpu()
    assert _lib.device_status() == 0
    err = float((logits - ref).abs().max())
    agree = float((logits.argmax(-1) == ref.argmax(-1)).float().mean())
    counts_equal = float((m.last_counts.cpu().long() == torch.stack([t["batches"] for t in tr])).float().mean())
    print(f"bf16 logits max-abs err {err:.4f}, top-1 agreement {agree:.3f}, count agreement {counts_equal:.3f}")
    assert err < 2e-2


def test_model_bf16_top1_agreement_1024_images():
    """1024 images through DeiT-Ti+DGE in bf16 against the fp32 oracle on bf16-rounded weights:
    logits within 2e-2 max-abs, and the top-1 class agrees on every image whose oracle top-2 margin
    exceeds twice the largest logit error seen (with random-init weights the 1000 logits of an image
    lie within a few tenths of each other, so a closer call than that is a coin toss for any
    bf16 implementation); the raw agreement is printed."""
    from vtpack_b200 import _lib
    B, chunk = 1024, 256
    sd = O.round_bf16(O.make_state_dict(192, 12, 3, seed=0))
    m = _model("tiny", sd, torch.bfloat16)
    img = O.make_images(B, 256, seed=11)
    ref = torch.cat([O.deit_dge_forward(img[i:i + chunk], sd, 12, 3, (4, 2, 1)) for i in range(0, B, chunk)])
    logits = torch.cat([m(img[i:i + chunk].to(DEV)).cpu() for i in range(0, B, chunk)])
    assert _lib.device_status() == 0
    err = float((logits - ref).abs().max())
    top2 = ref.topk(2, dim=-1).values
    margin = top2[:, 0] - top2[:, 1]
    same = logits.argmax(-1) == ref.argmax(-1)
    clear = margin > 2 * err
    print(f"1024 images: logits max-abs err {err:.4f}, raw top-1 agreement {float(same.float().mean()):.4f}, "
          f"{int(clear.sum())} images with a clear margin, all agree: {bool(same[clear].all())}")
    assert err < 2e-2
    assert bool(same[clear].all())
    assert float(same.float().mean()) > 0.85


@pytest.mark.parametrize("dtype,depth,tol", [(torch.float32, 4, 1e-4), (torch.bfloat16, 12, 2e-2)])
def test_model_512px(dtype, depth, tol):
    """Benchmark configuration 5 shape through the whole-model entry point at reduced batch and width:
    512 x 512 images (32 x 32 grid + cls = 1025 tokens, 64 regions per image, 1025 keys = four
    256-key chunks + one tail key), free-running router.  fp32: logits within 1e-4 relative of
    the oracle wherever the per-layer query counts agree (they must, unless a gate is a near-tie);
    bf16: logits within 2e-2 max-abs of the fp32 oracle on bf16-rounded weights."""
    from vtpack_b200 import _lib
    sd = O.make_state_dict(192, depth, 3, img_size=512, seed=30)
    if dtype == torch.bfloat16:
        sd = O.round_bf16(sd)
    img = O.make_images(3, 512, seed=34)          # smallest top-2 gate margin of the fp32 run: 2.8e-4
    tr = []
    ref = O.deit_dge_forward(img, sd, depth, 3, (4, 2, 1), trace=tr)
    m = _model("tiny", sd, dtype, depth=depth, img_size=512)
    logits = m(img.to(DEV)).cpu()
    assert _lib.device_status() == 0
    counts_ref = torch.stack([t["batches"] for t in tr])
    assert int(counts_ref.min()) >= 65 and int(counts_ref.max()) <= 1025
    if dtype == torch.float32:
        assert torch.equal(m.last_counts.cpu().long(), counts_ref)
        assert rel_err(logits, ref) < tol
    else:
        assert float((logits - ref).abs().max()) < tol


def test_layer_512px_bf16_skewed():
    """Benchmark configuration 5 shape at reduced batch: 32x32 grid (1025 keys = 4 chunks of 256 + 1 tail
    key), even images all-coarse (65 queries), odd images all-fine (1025 queries), bf16."""
    from vtpack_b200 import _lib
    sd = O.round_bf16(O.make_state_dict(384, 1, 6, img_size=512, seed=20))
    x = O.make_tokens(4, 1025, 384, seed=21).bfloat16().float()
    gate = torch.zeros(4, 8, 8, 3)
    gate[0::2, ..., 2] = 1e4
    gate[1::2, ..., 0] = 1e4
    ref = O.dge_block_forward(x, O.block_weights(sd, 0), 6, (4, 2, 1), forced_gate=gate)
    blk = _block(384, 6, sd, torch.bfloat16)
    out = blk(x.bfloat16().to(DEV), forced_gate=gate)
    assert _lib.device_status() == 0
    assert blk.dge.states["batches_device"].tolist() == [65, 1025, 65, 1025]
    assert rel_err(out.float(), ref) < 1.5e-2


@pytest.mark.parametrize("fine_bias", [-1e4, -0.5, 0.7, 1e4])
def test_layer_gate_skew_bf16(fine_bias):
    """Benchmark configuration 4 at reduced batch: gate skew from all-coarse to all-fine."""
    sd = O.round_bf16(O.make_state_dict(384, 1, 6, seed=22))
    x = O.make_tokens(6, 257, 384, seed=23).bfloat16().float()
    gate = O.make_gate_logits(6, 4, 4, 3, seed=24, fine_bias=fine_bias)
    tr = {}
    ref = O.dge_block_forward(x, O.block_weights(sd, 0), 6, (4, 2, 1), forced_gate=gate, trace=tr)
    blk = _block(384, 6, sd, torch.bfloat16)
    out = blk(x.bfloat16().to(DEV), forced_gate=gate)
    assert blk.dge.states["batches_device"].tolist() == tr["batches"].tolist()
    assert rel_err(out.float(), ref) < 1.5e-2


def test_full_size_properties():
    """Benchmark configuration 3 size (DeiT-S, batch 256, bf16): properties that need no oracle run.
    Images are independent, so permuting the batch permutes the logits; every per-image query
    count is 1 + sum of 16 values from {1, 4, 16}, hence within [17, 257] and = 2 (mod 3); with
    every region forced to the finest grain the DGE block is the dense block."""
    from vtpack_b200 import _lib, synthetic
    B = 256
    model = synthetic.build_model("small", DEV, torch.bfloat16)
    img = synthetic.images(B, 256, seed=5).to(DEV)
    logits = model(img).clone()
    counts = model.last_counts.clone()
    assert torch.isfinite(logits).all()
    assert int(counts.min()) >= 17 and int(counts.max()) <= 257
    assert bool(((counts - 2) % 3 == 0).all())
    perm = torch.randperm(B, generator=torch.Generator().manual_seed(6)).to(DEV)
    logits_p = model(img[perm]).clone()
    counts_p = model.last_counts.clone()
    same = (counts_p == counts[:, perm]).float().mean().item()
    assert same > 0.999          # an image computes the same whatever its place in the batch
    keep = (counts_p == counts[:, perm]).all(0)
    assert float((logits_p[keep] - logits[perm][keep]).abs().max()) < 1e-2
    # graph replay gives what the kernel-by-kernel forward gives
    out = torch.empty_like(logits)
    model.forward_graph(img, out)
    model.forward_graph(img, out)
    keep2 = (model.last_counts == counts).all(0)
    assert keep2.float().mean().item() > 0.99
    assert float((out[keep2] - logits[keep2]).abs().max()) < 1e-2
    # all-fine DGE block == dense block
    blk = model.blocks[0]
    x = torch.randn(B, 257, 384, device=DEV, generator=torch.Generator(DEV).manual_seed(7)).bfloat16()
    gate = torch.zeros(B, 4, 4, 3)
    gate[..., 0] = 1.0
    a = blk(x, forced_gate=gate)
    assert blk.dge.states["batches_device"].tolist() == [257] * B
    b = blk(x, dense=True)
    assert rel_err(a.float(), b.float()) < 2e-2
    assert _lib.device_status() == 0


def _pvt_block(C, heads, mr, sr, w, dtype):
    from functools import partial
    from vtpack_b200.models.dge.pvt_dge import Block
    blk = Block(C, heads, mlp_ratio=mr, qkv_bias=True, norm_layer=partial(torch.nn.LayerNorm, eps=1e-6),
                sr_ratio=sr, split_sizes=[4, 2, 1])
    blk.load_state_dict(w, strict=True)
    return blk.eval().to(device=DEV, dtype=dtype)


def test_pvt_block_fp32_golden(golden_dir):
    """PVT+DGE block (spatial reduction 4, 64 keys per image) against the reference's own output."""
    from vtpack_b200 import _lib
    g = np.load(os.path.join(golden_dir, "pvt_block_fp32.npz"))
    w = O.make_pvt_block_weights(64, 8, 4, seed=3)
    blk = _pvt_block(64, 1, 8, 4, w, torch.float32)
    out = blk(O.make_tokens(2, 32 * 32, 64, seed=4).to(DEV), 32, 32)
    assert g["gate_margin"].min() > 1e-5
    assert blk.dge.states["batches_device"].tolist() == g["batch_lengths"].tolist()
    assert rel_err(out, torch.from_numpy(g["out"])) < 1e-4
    assert _lib.device_status() == 0


@pytest.mark.parametrize("C,heads,H,sr,mr,extra", [(64, 1, 64, 8, 8, 0), (128, 2, 32, 4, 8, 0), (320, 5, 16, 2, 4, 0),
                                                   (512, 8, 8, 1, 4, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pvt_block_stages(C, heads, H, sr, mr, extra, dtype):
    """The four stage shapes of PVT+DGE at 256 px (grids 64..8, reductions 8..1, the last with a cls
    token), gates teacher-forced: fp32 within 1e-4 of the oracle; bf16 against the fp32 oracle on
    bf16-rounded weights and inputs."""
    from vtpack_b200 import _lib
    B = 4
    w = O.make_pvt_block_weights(C, mr, sr, seed=7)
    x = O.make_tokens(B, H * H + extra, C, seed=8)
    if dtype == torch.bfloat16:
        w = O.round_bf16(w)
        x = x.bfloat16().float()
    gate = O.make_gate_logits(B, H // 4, H // 4, 3, seed=9)
    tr = {}
    ref = O.dge_block_forward(x, w, heads, (4, 2, 1), forced_gate=gate, trace=tr, grid=(H, H), sr_ratio=sr)
    blk = _pvt_block(C, heads, mr, sr, w, dtype)
    out = blk(x.to(DEV).to(dtype), H, H, forced_gate=gate)
    assert _lib.device_status() == 0
    assert blk.dge.states["batches_device"].tolist() == tr["batches"].tolist()
    err = rel_err(out.float(), ref)
    assert err < (1e-4 if dtype == torch.float32 else 2e-2), err


def _visible_keys(C, sr):
    """Weights of a PVT block whose output shows its keys: tokens small beside their LayerNorm, attention sharp and wide, the MLP
    faint, random LayerNorm gains and biases.  In the oracle, rows of the reducing convolution that are wrong change the largest
    output by (15 shapes of test_pvt_block_reduction_windows) 0.3 to 1.5 of itself where rows or columns of the grid are
    mirrored or rolled, window elements or images exchanged, channels rolled, norm1's gain and bias left out, zeros or noise
    given; by 0.10 to 0.34 where one 4 x 4 region is zero, by 0.027 to 0.12 where one token is."""
    w = O.make_pvt_block_weights(C, 2, sr, seed=7)
    g = torch.Generator().manual_seed(11)
    for n in ("norm1", "attn.norm"):
        w[n + ".weight"] = 1 + 0.5 * torch.randn(C, generator=g)
        w[n + ".bias"] = 0.5 * torch.randn(C, generator=g)
    for n in ("q", "kv", "proj"):
        w[f"attn.{n}.weight"] = w[f"attn.{n}.weight"] * (5 * (C / 64) ** -0.5)
    w["mlp.fc2.weight"] = w["mlp.fc2.weight"] * 0.01
    return O.round_bf16(w)


@pytest.mark.parametrize("C,heads", [(64, 1), (128, 2), (320, 5)])
@pytest.mark.parametrize("H,W,sr", [(12, 24, 3), (24, 8, 2), (16, 16, 4), (60, 20, 5), (32, 48, 8)])
def test_pvt_block_reduction_windows(C, heads, H, W, sr):
    """Windows of the spatial reduction that lie inside a 4 x 4 region, cover several and straddle them, on grids that are not
    square: the rows the pool writes for the convolution (bf16) against the fp32 oracle on the same bf16 weights and tokens, with the
    bound of the stage shapes."""
    from vtpack_b200 import _lib
    w = _visible_keys(C, sr)
    x = (O.make_tokens(3, H * W, C, seed=8) * 2.0 ** -6).bfloat16().float()
    gate = O.make_gate_logits(3, H // 4, W // 4, 3, seed=9)
    tr = {}
    ref = O.dge_block_forward(x, w, heads, (4, 2, 1), forced_gate=gate, trace=tr, grid=(H, W), sr_ratio=sr)
    blk = _pvt_block(C, heads, 2, sr, w, torch.bfloat16)
    out = blk(x.to(DEV).bfloat16(), H, W, forced_gate=gate)
    assert _lib.device_status() == 0
    assert blk.dge.states["batches_device"].tolist() == tr["batches"].tolist()
    err = rel_err(out.float(), ref)
    assert err < 2e-2, err


@pytest.mark.parametrize("C,heads,H,sr,mr,extra", [(64, 1, 64, 8, 8, 0), (128, 2, 32, 4, 8, 0), (320, 5, 16, 2, 4, 0),
                                                   (512, 8, 8, 1, 4, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pvt_stage_in_one_call_equals_block_by_block(C, heads, H, sr, mr, extra, dtype):
    """Three blocks of a stage through ``stage_forward`` (one C-ABI call; in bf16 a block's unpool leaves the
    next block's router decisions, counts and token statistics) against the same blocks called one by one
    (every block runs its own gate and patch-list kernels): identical per-image query counts for every
    block, outputs equal to within the last bit of a few sums whose order differs."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.pvt_dge import stage_forward
    B = 6
    blocks = [_pvt_block(C, heads, mr, sr, O.make_pvt_block_weights(C, mr, sr, seed=20 + i), dtype) for i in range(3)]
    x = O.make_tokens(B, H * H + extra, C, seed=8).to(DEV).to(dtype)
    one = x
    counts_one = []
    for blk in blocks:
        one = blk(one, H, H)
        counts_one.append(blk.dge.states["batches_device"].tolist())
    x_before = x.clone()
    got = stage_forward(blocks, x, H, H)
    assert _lib.device_status() == 0
    assert torch.equal(x, x_before)                       # the caller's tokens are not written
    assert [blk.dge.states["batches_device"].tolist() for blk in blocks] == counts_one
    assert len({tuple(c) for c in counts_one}) > 1        # the blocks did pick different grains
    assert rel_err(got.float(), one.float()) < (1e-6 if dtype == torch.float32 else 4e-3)
    assert blocks[1].dge.get_complexity()["dynamic"] is not None


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pvt_model(golden_dir, dtype):
    """PVT+DGE tiny (4 stages, 8 blocks, patch 4: 4096 -> 64 tokens) through the mirror model: fp32
    against the reference's own logits and query counts; bf16 against the fp32 oracle on bf16-rounded
    weights (logits within 2e-2 max-abs)."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256
    g = np.load(os.path.join(golden_dir, "pvt_model_fp32.npz"))
    cfg = O.PVT_CONFIGS["tiny"]
    sd = O.make_pvt_state_dict(cfg, seed=0)
    img = O.make_images(2, 256, seed=8)
    if dtype == torch.bfloat16:
        sd = O.round_bf16(sd)
        ref = O.pvt_dge_forward(img, sd, cfg)
    else:
        ref = torch.from_numpy(g["logits"])
    m = pvt_dge_s124_tiny_256()
    m.load_state_dict(sd, strict=True)
    m = m.eval().to(device=DEV, dtype=dtype)
    logits = m(img.to(DEV)).cpu()
    assert _lib.device_status() == 0
    if dtype == torch.float32:
        assert g["gate_margin"].min() > 1e-5
        assert [c.tolist() for c in m.last_counts] == g["batch_lengths"].tolist()
        assert rel_err(logits, ref) < 1e-4
    else:
        assert float((logits - ref).abs().max()) < 2e-2


def test_pvt_model_follows_parameter_updates():
    """The eval forward keeps tensors derived from parameters (GEMM-layout weights, fp32 vectors, position rows);
    after parameters change in place — an optimizer step, load_state_dict — the next forward must use the new
    values: compared with a second model, loaded with the changed parameters, that has never run before."""
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256
    sd = O.make_pvt_state_dict(O.PVT_CONFIGS["tiny"], seed=0)
    m = pvt_dge_s124_tiny_256()
    m.load_state_dict(sd, strict=True)
    m = m.eval().to(device=DEV, dtype=torch.bfloat16)
    img = O.make_images(2, 256, seed=8).to(DEV)
    first = m(img).clone()
    with torch.no_grad():
        m.patch_embed1.proj.weight.mul_(1.5)
        m.patch_embed2.norm.bias.add_(0.25)
        m.pos_embed3.add_(0.5)
        m.cls_token.add_(1.0)
        m.head.bias.add_(2.0)
    fresh = pvt_dge_s124_tiny_256()
    fresh.load_state_dict({k: v.float().cpu() for k, v in m.state_dict().items()}, strict=True)
    fresh = fresh.eval().to(device=DEV, dtype=torch.bfloat16)
    got, ref = m(img), fresh(img)
    assert torch.equal(got, ref)
    assert float((got - first).abs().max()) > 0.5


def test_pvt_model_other_input_size_and_pyramid(golden_dir):
    """PVT+DGE tiny in eval mode on 384 px images (position embeddings resized bilinearly) and its
    feature-pyramid variant (num_classes = 0), fp32, against the reference's own outputs."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256
    g = np.load(os.path.join(golden_dir, "pvt_model_384_fp32.npz"))
    sd = O.make_pvt_state_dict(O.PVT_CONFIGS["tiny"], seed=0)
    img = O.make_images(1, 384, seed=10).to(DEV)
    m = pvt_dge_s124_tiny_256()
    m.load_state_dict(sd, strict=True)
    m = m.eval().to(DEV)
    logits = m(img).cpu()
    assert _lib.device_status() == 0
    assert float(g["gate_margin"]) > 1e-5
    assert [c.tolist() for c in m.last_counts] == g["counts"].tolist()
    assert rel_err(logits, torch.from_numpy(g["logits"])) < 1e-4
    m0 = pvt_dge_s124_tiny_256(num_classes=0)
    m0.load_state_dict({k: v for k, v in sd.items() if not k.startswith(("head.", "norm."))}, strict=True)
    feats = m0.eval().to(DEV)(img)
    assert sorted(feats) == ["res2", "res3", "res4", "res5"]
    for k, v in feats.items():
        assert list(v.shape) == g[f"{k}_shape"].tolist(), k
        assert rel_err(v[:, :, ::8, ::8], torch.from_numpy(g[f"{k}_sub"])) < 1e-4, k
        assert abs(float(v.double().sum()) - float(g[f"{k}_sum"])) < 1e-4 * float(v.double().abs().sum()), k


@pytest.mark.parametrize("kind", ["deit", "pvt"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_repeated_forwards_replay_one_capture(kind, dtype):
    """A forward captures the launches between the image kernel and the head once its shape has earned it (here: the
    second one), later ones replay them: images and logits at other addresses, two batch sizes in turn, a larger batch that replaces the scratch
    buffer and changed weights give bit for bit what a first (launch by launch) forward gives."""
    from vtpack_b200 import _lib, synthetic
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256

    def make(seed):
        if kind == "deit":
            m = synthetic.build_model("tiny", DEV, dtype, depth=2, seed=seed)
        else:
            m = pvt_dge_s124_tiny_256()
            m.load_state_dict(O.make_pvt_state_dict(O.PVT_CONFIGS["tiny"], seed=seed), strict=True)
            m = m.eval().to(device=DEV, dtype=dtype)
        m._plans.earn = 2
        return m

    def first(seed, img):                                    # a model that has never run before
        m = make(seed)
        return m(img), [c.clone() for c in m.last_counts]

    def same(m, ref, img):
        out = m(img)
        assert torch.equal(out, ref[0])
        assert all(torch.equal(a, b) for a, b in zip(m.last_counts, ref[1]))
        return out

    m = make(0)
    imgs = {b: [O.make_images(b, 256, seed=b + k).to(DEV) for k in range(2)] for b in (1, 3)}
    refs = {b: [first(0, i) for i in v] for b, v in imgs.items()}
    kept = None
    for _ in range(3):
        for b in imgs:
            for k in range(2):
                out = same(m, refs[b][k], imgs[b][k].clone())
                kept = out if kept is None else kept         # an earlier result is not overwritten
    assert torch.equal(kept, refs[1][0][0])
    big = O.make_images(40, 256, seed=9).to(DEV)
    m(big)                                                   # may replace the scratch buffers
    for _ in range(3):
        same(m, refs[3][0], imgs[3][0])
    m.load_state_dict(make(5).state_dict())
    ref5 = first(5, imgs[3][1])
    for _ in range(3):
        same(m, ref5, imgs[3][1])
    assert _lib.device_status() == 0


@pytest.mark.parametrize("kind", ["deit", "pvt"])
def test_replayed_forward_follows_settings_and_streams(kind):
    """What the launches take by value (softmax scale, LayerNorm epsilon) may change between calls of a model whose
    launches have been captured, in ``forward`` and in ``forward_graph``, and the calls may come from different streams."""
    from vtpack_b200 import synthetic
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256

    def make():
        if kind == "deit":
            return synthetic.build_model("tiny", DEV, torch.bfloat16, depth=2, seed=0)
        m = pvt_dge_s124_tiny_256()
        m.load_state_dict(O.make_pvt_state_dict(O.PVT_CONFIGS["tiny"], seed=0), strict=True)
        return m.eval().to(device=DEV, dtype=torch.bfloat16)

    def scale(m):
        for blk in (m.blocks if kind == "deit" else m.block1):
            blk.attn.scale *= 4.0

    def eps(m):
        m.norm.eps = 0.1

    img = O.make_images(2, 256, seed=3).to(DEV)
    m, changes = make(), []
    m._plans.earn = 2
    logits = torch.empty(2, 1000, device=DEV)
    graph = (lambda: m.forward_graph(img, logits)) if kind == "deit" else (lambda: m.forward_graph(img))
    for change in (None, scale, eps):
        if change is not None:
            change(m)
            changes.append(change)
        fresh = make()
        for c in changes:
            c(fresh)
        want = fresh(img)
        for _ in range(3):
            assert torch.equal(m(img), want)
            assert torch.equal(graph(), want)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            got = m(img)
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(got, want)
    assert not torch.equal(make()(img), want)


@pytest.mark.parametrize("kind", ["deit", "pvt"])
def test_forward_with_swapped_in_weights_updated_in_place(kind):
    """Weights handed over by functional_call and updated in place between calls (a moving average): every forward, the
    replayed ones among them, uses their current values."""
    from torch.func import functional_call

    from vtpack_b200 import synthetic
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256

    def make():
        if kind == "deit":
            return synthetic.build_model("tiny", DEV, torch.bfloat16, depth=2, seed=0)
        m = pvt_dge_s124_tiny_256()
        m.load_state_dict(O.make_pvt_state_dict(O.PVT_CONFIGS["tiny"], seed=0), strict=True)
        return m.eval().to(device=DEV, dtype=torch.bfloat16)

    img = O.make_images(2, 256, seed=3).to(DEV)
    m, fresh = make(), make()
    m._plans.earn = 2
    ema = {k: v.detach().clone() for k, v in m.named_parameters()}
    for step in range(3):
        if step:
            for t in ema.values():
                if t.is_floating_point():
                    t.mul_(0.9)
        fresh.load_state_dict(ema, strict=False)
        want = fresh._forward_eval(img, use_plans=False)
        for _ in range(3):
            assert torch.equal(functional_call(m, ema, (img,)), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("kind", ["deit", "pvt"])
def test_image_gives_the_same_bits_in_any_batch(kind, dtype):
    """Logits and counts of an image do not depend on how many images are with it: sums are formed in the same order
    whatever the number of tiles a launch has."""
    from vtpack_b200 import synthetic
    from vtpack_b200.models.dge.pvt_dge import pvt_dge_s124_tiny_256
    if kind == "deit":
        m = synthetic.build_model("small", DEV, dtype, depth=3, seed=0)
    else:
        m = pvt_dge_s124_tiny_256()
        m.load_state_dict(O.make_pvt_state_dict(O.PVT_CONFIGS["tiny"], seed=0), strict=True)
        m = m.eval().to(device=DEV, dtype=dtype)
    img = O.make_images(80, 256, seed=3).to(DEV)
    want = m(img)
    counts = [c.clone() for c in m.last_counts]
    for n in (1, 2, 7, 19, 40):
        got = m(img[:n].contiguous())
        assert torch.equal(got, want[:n]), n
        assert all(torch.equal(a, b[:n]) for a, b in zip(m.last_counts, counts))


@pytest.mark.parametrize("C,B,fine", [(192, 9, 0.0), (192, 15, 1.0), (192, 16, 0.5), (192, 20, 1.0), (384, 4, 0.0), (384, 8, 1.0),
                                      (384, 9, 1.0), (768, 2, 0.5), (768, 3, 1.0), (768, 4, 1.0)])
def test_q_and_kv_in_one_launch_same_bits_for_an_image(C, B, fine):
    """q and kv of a block in 128 x 64 tiles (an image alone), 128 x 128 tiles (as many as SMs, or some more where all rows exist: 15 and 16, 8,
    4 images; 192 q columns fill one and a half) and the persistent kernel's, with few and with all rows that the host allows for."""
    from vtpack_b200 import _lib
    torch.manual_seed(C + B)
    sd = O.round_bf16(O.make_state_dict(C, 1, C // 64, seed=B))
    blk = _block(C, C // 64, sd, torch.bfloat16)
    x = torch.randn(B, 257, C, device=DEV).bfloat16()
    gate = torch.zeros(B, 4, 4, 3, device=DEV)
    gate[..., 2] = 1
    gate[..., 0] = torch.where(torch.rand(B, 4, 4, device=DEV) < fine, 2.0, 0.0)
    out = blk(x, forced_gate=gate)
    for b in range(B):
        assert torch.equal(blk(x[b:b + 1].contiguous(), forced_gate=gate[b:b + 1]), out[b:b + 1]), b
    assert _lib.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B", [1, 10, 40, 150])
@pytest.mark.parametrize("C", [64, 128, 320])
def test_q_and_kv_in_one_launch_behind_a_reduction(C, B, dtype):
    """q, which folds norm1 in bf16, and kv of reduced keys, which does not, as one launch (tiles of 64 and 128 columns all at once, the
    persistent kernel's narrow and wide ones) and as two, which is how a block with events between its stages runs: the same bits,
    biases of -0 included."""
    import ctypes

    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import pvt_dge
    torch.manual_seed(C + B)
    blk = pvt_dge.Block(C, C // 64, mlp_ratio=1, qkv_bias=True, sr_ratio=2, split_sizes=[4, 2, 1]).eval()
    with torch.no_grad():
        for p in blk.parameters():
            if p.is_floating_point():
                torch.nn.init.normal_(p, std=0.2)
        blk.attn.kv.bias[: 2 * C: 3] = -0.0
    blk = blk.to(device=DEV, dtype=dtype)
    x = torch.randn(B, 256, C, device=DEV).to(dtype)
    gate = torch.randn(B, 4, 4, 3, device=DEV)
    got = blk(x, 16, 16, forced_gate=gate)
    s = pvt_dge._shape_struct(dtype, B, 16, 16, 0, C, C // 64, C, [4, 2, 1], blk.norm1.eps, 0, blk.attn.scale)
    s.sr_ratio, s.sr_eps = 2, float(blk.attn.norm.eps)
    w, lib = pvt_dge._pack_block(blk, dtype), _lib.lib()
    n = lib.vtp_block_workspace_bytes(ctypes.byref(s))
    ws, out = torch.empty(n, dtype=torch.uint8, device=DEV), torch.empty_like(x)
    counts = torch.empty(B, dtype=torch.int32, device=DEV)
    events = [torch.cuda.Event(enable_timing=True) for _ in range(12)]
    for e in events:
        e.record()
    arr = (ctypes.c_void_p * 12)(*[e.cuda_event for e in events])
    _lib.check(lib.vtp_dge_block_forward_timed(ctypes.byref(s), ctypes.byref(w), x.data_ptr(), out.data_ptr(), gate.data_ptr(),
                                               counts.data_ptr(), ws.data_ptr(), n, arr, 12,
                                               torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert bool(got.isfinite().all()) and torch.equal(got, out)


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("extra", [0, 1])
def test_packed_rows_listed_or_derived_by_the_pool(extra, forced):
    """Many regions and images have the rows of a block's packed queries listed, few have the pool work them out: the same
    bits and counts for an image, in the block that starts and in the one whose counts that one starts."""
    from functools import partial

    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import pvt_dge
    torch.manual_seed(0)
    blocks = [pvt_dge.Block(64, 1, mlp_ratio=2, qkv_bias=True, norm_layer=partial(torch.nn.LayerNorm, eps=1e-6), sr_ratio=8,
                            split_sizes=[4, 2, 1]).eval().to(device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    if extra:                                                # a token in front of the grid: no spatial reduction
        blocks = [pvt_dge.Block(64, 1, mlp_ratio=2, qkv_bias=True, sr_ratio=1, split_sizes=[4, 2, 1]).eval()
                  .to(device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    for b in blocks:
        torch.nn.init.normal_(b.dge.router.gate.weight, std=0.2)
        torch.nn.init.zeros_(b.dge.router.gate.bias)
    G, B = (32, 64) if extra else (64, 40)                   # 64 and 256 regions per image
    x = torch.randn(B, G * G + extra, 64, device=DEV).bfloat16()
    gate = torch.randn(B, G // 4, G // 4, 3, device=DEV) if forced else None

    def run(n):
        if forced:
            y = blocks[0](x[:n].contiguous(), G, G, forced_gate=gate[:n].contiguous())
            return y, [blocks[0].dge.states["batches_device"].clone()]
        y = pvt_dge.stage_forward(blocks, x[:n].contiguous(), G, G)
        return y, [b.dge.states["batches_device"].clone() for b in blocks]

    many, counts = run(B)
    for n in (1, 3):
        few, c = run(n)
        assert torch.equal(few, many[:n]) and all(torch.equal(p, q[:n]) for p, q in zip(c, counts))
    assert len(set(counts[0].tolist())) > 1 and _lib.device_status() == 0


def test_image_with_more_regions_than_a_list_holds():
    """12544 regions do not fit the listing kernel's shared memory: the pool works their rows out.  The image is a smaller
    one, whose 6272 regions are listed, twice: doubled keys leave a softmax average as it is, so its halves are the smaller
    one's result but for the order of fp32 sums over 1568 and 3136 keys (3136 * 2^-24 = 1.9e-4 at worst)."""
    from functools import partial

    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import pvt_dge
    torch.manual_seed(0)
    blk = pvt_dge.Block(64, 1, mlp_ratio=2, qkv_bias=True, norm_layer=partial(torch.nn.LayerNorm, eps=1e-6), sr_ratio=8,
                        split_sizes=[4, 2, 1]).eval().to(DEV)
    H, W = 224, 448
    x, gate = torch.randn(1, H * W, 64, device=DEV), torch.randn(1, H // 4, W // 4, 3, device=DEV)
    small = blk(x, H, W, forced_gate=gate)
    n = int(blk.dge.states["batches_device"])
    big = blk(torch.cat((x, x), 1), 2 * H, W, forced_gate=torch.cat((gate, gate), 1))
    assert int(blk.dge.states["batches_device"]) == 2 * n and _lib.device_status() == 0
    for half in big.split(H * W, 1):
        assert float((half - small).norm() / small.norm()) < 1.9e-4


@pytest.mark.parametrize("fine", [0.0, 0.3, 1.0])
@pytest.mark.parametrize("C,B,grid,sr,ratio", [(64, 8, 64, 8, 8), (128, 33, 32, 4, 8), (192, 79, 16, 1, 4), (320, 96, 16, 2, 4),
                                               (384, 125, 16, 1, 4), (384, 210, 16, 1, 8)])
def test_mlp_in_one_launch(C, B, grid, sr, ratio, fine):
    """fc1 and fc2 as one launch, which large batches take, and as two, which is how a block with events between its stages runs: the
    same bits.  Few rows, some rounds of 256 rows for every pair of CTAs, a last round whose rows are two pairs' each (384: 2125 and
    33410 rows), rows that end inside a warp's, and a wider hidden layer."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import deit_dge, pvt_dge
    torch.manual_seed(C + B)
    if sr > 1:
        blk = pvt_dge.Block(C, C // 64, mlp_ratio=ratio, qkv_bias=True, sr_ratio=sr, split_sizes=[4, 2, 1]).eval()
    else:
        blk = deit_dge.Block(C, C // 64, mlp_ratio=ratio, qkv_bias=True, split_sizes=[4, 2, 1]).eval()
    with torch.no_grad():
        for name, p in blk.named_parameters():
            if p.is_floating_point():
                torch.nn.init.normal_(p, mean=float("norm" in name and name.endswith("weight")), std=0.05)
    blk = blk.to(device=DEV, dtype=torch.bfloat16)
    extra = int(sr == 1)
    x = torch.randn(B, grid * grid + extra, C, device=DEV).bfloat16()
    gate = torch.randn(B, grid // 4, grid // 4, 3, device=DEV)
    gate[..., 0] = torch.where(torch.rand(gate.shape[:3], device=DEV) < fine, 9.0, -9.0)
    if fine == 0.0:
        gate[..., 2] = 9.0

    def plain():
        return blk(x, grid, grid, forced_gate=gate) if sr > 1 else blk(x, forced_gate=gate)
    got = plain()
    s = deit_dge._shape_struct(torch.bfloat16, B, grid, grid, extra, C, C // 64, ratio * C, [4, 2, 1], blk.norm1.eps, 0, blk.attn.scale)
    if sr > 1:
        s.sr_ratio, s.sr_eps = sr, float(blk.attn.norm.eps)
    run, out = _timed_block(s, (pvt_dge if sr > 1 else deit_dge)._pack_block(blk, torch.bfloat16), x, gate)
    apart = range(12)
    run(apart)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert bool(got.isfinite().all()) and torch.equal(got, out)
    # each side is what it is taken for
    assert sum("mlp_tc_kernel" in n for n in kernels_of(plain)) == 1
    assert not any("mlp_tc_kernel" in n for n in kernels_of(lambda: run(apart)))


def _timed_block(s, w, x, gate):
    """A block with events behind the stages of a list: (a function of that list, its output)."""
    import ctypes

    from vtpack_b200 import _lib
    lib = _lib.lib()
    n = lib.vtp_block_workspace_bytes(ctypes.byref(s))
    ws, out = torch.empty(n, dtype=torch.uint8, device=DEV), torch.empty_like(x)
    counts = torch.empty(x.shape[0], dtype=torch.int32, device=DEV)
    events = [torch.cuda.Event(enable_timing=True) for _ in range(12)]
    for e in events:
        e.record()

    def run(stages):
        arr = (ctypes.c_void_p * 12)(*[e.cuda_event if i in stages else None for i, e in enumerate(events)])
        _lib.check(lib.vtp_dge_block_forward_timed(ctypes.byref(s), ctypes.byref(w), x.data_ptr(), out.data_ptr(), gate.data_ptr(),
                                                   counts.data_ptr(), ws.data_ptr(), n, arr, 12,
                                                   torch.cuda.current_stream().cuda_stream))
    return run, out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("C,B,sr", [(384, 125, 1), (192, 3, 1), (64, 5, 8), (64, 8, 8)])
def test_timed_block_without_events_inside_a_pair_runs_what_the_block_runs(dtype, C, B, sr):
    """Stages 4 and 5 (q and kv) and 9 and 10 (fc1 and fc2) share launches in a block's forward; timed with no event between the two the
    block launches the same kernels and gives the same bits, and the events behind the pairs are recorded."""
    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import deit_dge, pvt_dge
    torch.manual_seed(C + B)
    grid, extra = (64, 0) if sr > 1 else (16, 1)
    module = pvt_dge if sr > 1 else deit_dge
    kw = dict(sr_ratio=sr) if sr > 1 else {}
    blk = module.Block(C, C // 64, mlp_ratio=8 if sr > 1 else 4, qkv_bias=True, split_sizes=[4, 2, 1], **kw).eval().to(device=DEV, dtype=dtype)
    x = torch.randn(B, grid * grid + extra, C, device=DEV).to(dtype)
    gate = torch.randn(B, grid // 4, grid // 4, 3, device=DEV)

    def plain():
        return blk(x, grid, grid, forced_gate=gate) if sr > 1 else blk(x, forced_gate=gate)
    s = deit_dge._shape_struct(dtype, B, grid, grid, extra, C, C // 64, (8 if sr > 1 else 4) * C, [4, 2, 1], blk.norm1.eps, 0, blk.attn.scale)
    if sr > 1:
        s.sr_ratio, s.sr_eps = sr, float(blk.attn.norm.eps)
    run, out = _timed_block(s, module._pack_block(blk, dtype), x, gate)
    together = [i for i in range(12) if i not in (4, 9)]
    got = plain()
    run(together)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0 and torch.equal(got, out)
    names = kernels_of(plain)
    assert kernels_of(lambda: run(together)) == names
    apart = kernels_of(lambda: run(range(12)))
    assert len(apart) == len(names) + 1 + any("mlp_tc_kernel" in n for n in names)


@pytest.mark.parametrize("C,G,B,extra,sr", [(64, 20, 49, 0, 1), (128, 12, 133, 1, 1), (192, 20, 49, 1, 1), (320, 20, 49, 1, 1), (384, 28, 25, 1, 1), (384, 4, 1187, 0, 1),
                                            (64, 20, 49, 0, 4), (128, 20, 49, 0, 4), (320, 20, 49, 0, 2), (320, 12, 215, 0, 2),
                                            (320, 12, 301, 0, 2)])
def test_pool_and_unpool_of_many_regions_are_those_of_few(C, G, B, extra, sr):
    """From eight regions a SM on a warp pools and unpools a region, with fewer a block: the same tokens, statistics, rows of a spatial reduction and
    next decisions, so the same bits after two blocks that chain, at every grain; region counts that leave warps of the last block idle, with and
    without extra tokens, and (C = 320) one, one and a bit and one and a half rounds of the pool's blocks, of which the second has a block pool a region."""
    from functools import partial

    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import pvt_dge
    torch.manual_seed(C + G)
    blocks = [pvt_dge.Block(C, C // 64, mlp_ratio=2, qkv_bias=True, norm_layer=partial(torch.nn.LayerNorm, eps=1e-6), sr_ratio=sr,
                            split_sizes=[4, 2, 1]).eval().to(device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    for b in blocks:
        torch.nn.init.normal_(b.dge.router.gate.weight, std=0.3)
        torch.nn.init.zeros_(b.dge.router.gate.bias)
    x = torch.randn(B, G * G + extra, C, device=DEV).bfloat16()
    assert B * (G // 4) ** 2 >= 8 * torch.cuda.get_device_properties(0).multi_processor_count and (B * (G // 4) ** 2) % 4

    def run(rows):
        y = pvt_dge.stage_forward(blocks, rows.contiguous(), G, G)
        return y, [b.dge.states["batches_device"].clone() for b in blocks]
    many, counts = run(x)
    for part in (slice(0, 1), slice(1, 12), slice(B - 5, B)):
        few, c = run(x[part])
        assert torch.equal(few, many[part]) and all(torch.equal(p, q[part]) for p, q in zip(c, counts))
    R = (G // 4) ** 2
    names = kernels_of(lambda: pvt_dge.stage_forward(blocks, x, G, G))
    assert sum("unpool_warp_kernel" in n for n in names) == 2
    assert sum("pool_warp_kernel" in n and "unpool" not in n for n in names) == (0 if B == 215 else 2)
    assert B * extra + B * R < int(counts[1].sum()) < B * extra + 16 * B * R and _lib.device_status() == 0


@pytest.mark.parametrize("C,G,B,extra,sr", [(64, 20, 49, 0, 1), (128, 12, 133, 1, 1), (192, 20, 49, 1, 1), (320, 20, 49, 1, 1), (384, 28, 25, 1, 1),
                                            (64, 20, 49, 0, 4), (320, 20, 49, 0, 2)])
def test_pool_of_many_regions_leaves_the_statistics_itself(C, G, B, extra, sr):
    """With the gate given nothing has left the tokens' statistics, so the pool does: a warp a region for many regions, a block a region
    for few, the same bits of a whole block."""
    from functools import partial

    from vtpack_b200 import _lib
    from vtpack_b200.models.dge import deit_dge, pvt_dge
    torch.manual_seed(C + G)
    kw = dict(mlp_ratio=2, qkv_bias=True, norm_layer=partial(torch.nn.LayerNorm, eps=1e-6), split_sizes=[4, 2, 1])
    blk = pvt_dge.Block(C, C // 64, sr_ratio=sr, **kw) if extra == 0 else deit_dge.Block(C, C // 64, **kw)
    blk = blk.eval().to(device=DEV, dtype=torch.bfloat16)
    x = (torch.randn(B, G * G + extra, C, device=DEV) * torch.rand(B, G * G + extra, 1, device=DEV) + 0.5).bfloat16()
    gate = torch.randn(B, G // 4, G // 4, 3, device=DEV)
    assert B * (G // 4) ** 2 >= 8 * torch.cuda.get_device_properties(0).multi_processor_count

    def run(part):
        args = (x[part].contiguous(), G, G) if extra == 0 else (x[part].contiguous(),)
        return blk(*args, forced_gate=gate[part].contiguous())
    many = run(slice(0, B))
    for part in (slice(0, 1), slice(1, 12), slice(B - 5, B)):
        assert torch.equal(run(part), many[part])
    names = kernels_of(lambda: run(slice(0, B)))
    assert any("pool_warp_kernel" in n and "unpool" not in n for n in names) and any("unpool_warp_kernel" in n for n in names)
    assert not any("warp_kernel" in n for n in kernels_of(lambda: run(slice(0, 1)))) and _lib.device_status() == 0
