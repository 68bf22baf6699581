"""GPU parity of the training path: gradients of the token movers, the ragged products, and a
training-mode DeiT+DGE block, against what the reference's own autograd functions returned on the
same seeded inputs (committed fixtures; tests/golden/make_golden.py)."""
import os

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from tests.gpu_util import O, rel_err

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
TOL = 1e-4          # fp32, relative to the largest reference value


@pytest.fixture(scope="module")
def layers():
    from vtpack_b200 import _lib, layers
    _lib.lib()
    return layers


def _golden(golden_dir, name):
    return {k: torch.from_numpy(v) for k, v in np.load(os.path.join(golden_dir, name)).items()}


@pytest.mark.parametrize("C", [32, 1])
def test_mover_gradients_match_reference(layers, golden_dir, C):
    z = _golden(golden_dir, "train_ops_fp32.npz")
    splits = torch.tensor([4, 2, 1])
    x, indices = O.train_ops_inputs(C)
    x = x.to(DEV).requires_grad_(True)
    patches, lengths = layers.grained_sample_index_to_patch(indices.to(DEV), splits, 4, 1)
    assert torch.equal(lengths, z[f"c{C}_lengths"])
    L = patches.shape[0]
    comp = layers.grained_sample_compress(x, patches, 16, 16, 1)
    assert torch.equal(comp.detach().cpu(), z[f"c{C}_comp"])
    grad_x, = torch.autograd.grad(comp, x, O.randn_seeded((L, C), 11).to(DEV))
    assert torch.equal(grad_x.cpu(), z[f"c{C}_grad_x"])            # a power-of-two scale: exact
    q = O.randn_seeded((L, C), 12).to(DEV).requires_grad_(True)
    ref = x.detach().clone().requires_grad_(True)
    tok = layers.grained_sample_decompress(q, patches, ref, 16, 16, 1, True)
    g2 = O.randn_seeded((2, 257, C), 13).to(DEV)
    grad_q, grad_ref = torch.autograd.grad(tok, (q, ref), g2)
    assert torch.equal(grad_ref, g2)
    assert rel_err(grad_q, z[f"c{C}_grad_q"]) < 1e-6
    # without the reference term the reference tensor receives a zero gradient (grained_sample.py:76-77)
    tok2 = layers.grained_sample_decompress(q, patches, ref, 16, 16, 1, False)
    _, grad_ref2 = torch.autograd.grad(tok2, (q, ref), g2)
    assert not grad_ref2.any()


@pytest.mark.parametrize("B,G,C", [(3, 16, 384), (2, 32, 64)])
def test_mover_gradients_bf16_and_adjoint(layers, B, G, C):
    """Size-independent property: <pool(x), g> == <x, pool_grad(g)> and the same for the unpool (the
    gradient kernels are the adjoints of the forward kernels); bf16 gradients round the fp32 ones."""
    splits = torch.tensor([4, 2, 1])
    gen = torch.Generator().manual_seed(B * G + C)
    indices = torch.randint(0, 3, (B, G // 4, G // 4), generator=gen).to(DEV)
    patches, _ = layers.grained_sample_index_to_patch(indices, splits, 4, 1)
    L, N = patches.shape[0], G * G + 1
    x = torch.randn(B, N, C, generator=gen).to(DEV).requires_grad_(True)
    g = torch.randn(L, C, generator=gen).to(DEV)
    comp = layers.grained_sample_compress(x, patches, G, G, 1)
    gx, = torch.autograd.grad(comp, x, g)
    lhs, rhs = (comp.detach().double() * g.double()).sum(), (x.detach().double() * gx.double()).sum()
    assert abs(float(lhs - rhs)) < 1e-6 * max(1.0, abs(float(lhs)))
    q = torch.randn(L, C, generator=gen).to(DEV).requires_grad_(True)
    gt = torch.randn(B, N, C, generator=gen).to(DEV)
    tok = layers.grained_sample_decompress(q, patches, x.detach(), G, G, 1, False)
    gq, = torch.autograd.grad(tok, q, gt)
    lhs, rhs = (tok.detach().double() * gt.double()).sum(), (q.detach().double() * gq.double()).sum()
    assert abs(float(lhs - rhs)) < 1e-6 * max(1.0, abs(float(lhs)))
    # bf16
    xb = x.detach().bfloat16().requires_grad_(True)
    gxb, = torch.autograd.grad(layers.grained_sample_compress(xb, patches, G, G, 1), xb, g.bfloat16())
    gx_ref, = torch.autograd.grad(layers.grained_sample_compress(x, patches, G, G, 1), x, g.bfloat16().float())
    assert torch.equal(gxb.float(), gx_ref)                             # exact: scale by 1, 1/4 or 1/16
    qb = q.detach().bfloat16().requires_grad_(True)
    tokb = layers.grained_sample_decompress(qb, patches, xb.detach(), G, G, 1, False)
    gqb, = torch.autograd.grad(tokb, qb, gt.bfloat16())
    tokf = layers.grained_sample_decompress(q, patches, x.detach(), G, G, 1, False)
    gqf, = torch.autograd.grad(tokf, q, gt.bfloat16().float())
    # fp32 sums, one rounding.  The fp32 and bf16 rows use different lane layouts of the region kernel, whose
    # partial sums are taken in a different order: the fp32 sums agree to rounding, so the bf16 results agree
    # except where a sum sits on a rounding boundary (one bf16 step, 2^-8 relative)
    assert rel_err(gqb.float(), gqf) < 4e-3
    step = gqf.abs().clamp_min(1e-3) * 2.0 ** -7
    assert bool(((gqb.float() - gqf.bfloat16().float()).abs() <= step).all())
    assert float((gqb != gqf.bfloat16()).float().mean()) < 1e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,G,C", [(3, 16, 384), (2, 32, 64), (5, 16, 192), (2, 16, 32)])
def test_unpool_grad_region_form_matches_the_list_walk(layers, dtype, B, G, C):
    """The gradient of the replicate-unpool for its packed rows in its two forms: a walk over the patch
    list (any list) and one thread block per region (a list made from grain indices).  fp32 sums in a
    different order: equal to fp32 rounding; the autograd function picks the region form when the list
    carries its regions.  Also checks the per-region first rows the Python side derives."""
    import ctypes
    from vtpack_b200 import _lib
    from vtpack_b200.runtime import dtype_code, ptr, stream_ptr
    lib = _lib.lib()
    splits = torch.tensor([4, 2, 1])
    gen = torch.Generator().manual_seed(B * 31 + G + C)
    indices = torch.randint(0, 3, (B, G // 4, G // 4), generator=gen).to(DEV)
    patches, _ = layers.grained_sample_index_to_patch(indices, splits, 4, 1)
    L, N = patches.shape[0], G * G + 1
    idx32, first, splits_l, region_size, Hr, Wr, extra = patches._vtp_regions
    # the first row of every region, read off the list itself: the row whose (y, x) is the region's corner
    pl = patches.cpu()
    corner = (pl[:, 1] >= 0) & (pl[:, 1] % 4 == 0) & (pl[:, 2] % 4 == 0)
    rows = torch.nonzero(corner).reshape(-1)
    rid = pl[rows, 0] * (Hr * Wr) + (pl[rows, 1] // 4) * Wr + pl[rows, 2] // 4
    want = torch.empty(B * Hr * Wr, dtype=torch.long)
    want[rid] = rows
    assert torch.equal(first.cpu().reshape(-1).long(), want)

    g = torch.randn(B, N, C, generator=gen).to(dtype).to(DEV)
    by_list = torch.empty(L, C, dtype=dtype, device=DEV)
    _lib.check(lib.vtp_unpool_grad(ptr(g), dtype_code(dtype), B, N, C, G, 1, ptr(patches._vtp_i32), None, L,
                                   ptr(by_list), stream_ptr(g.device)))
    supported = bool(lib.vtp_region_layout_supported(dtype_code(dtype), C))
    arr = (ctypes.c_int * 3)(4, 2, 1)
    by_region = torch.full((L, C), float("nan"), dtype=dtype, device=DEV)
    rc = lib.vtp_unpool_grad_regions(ptr(g), dtype_code(dtype), B, Hr, Wr, 4, C, 1, ptr(idx32), arr, 3, ptr(first),
                                     ptr(patches._vtp_offsets), L, ptr(by_region), stream_ptr(g.device))
    if not supported:
        assert rc == _lib.ERR_SHAPE          # rows of 4 chunks have no lane layout: the list walk is the general form
        return
    _lib.check(rc)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    # reference: the sum over each patch's tokens in fp64
    want_sum = torch.zeros(L, C, dtype=torch.float64)
    gd = g.double().cpu()
    for p in range(L):
        b, y, x, st = (int(v) for v in pl[p])
        if y < 0:
            want_sum[p] = gd[b, -y - 1]
        else:
            toks = [1 + (y + dy) * G + x + dx for dy in range(st) for dx in range(st)]
            want_sum[p] = gd[b, toks].sum(0)
    tol = 1e-6 if dtype == torch.float32 else 8e-3
    assert rel_err(by_region.double().cpu(), want_sum) < tol
    assert rel_err(by_list.double().cpu(), want_sum) < tol
    if dtype == torch.float32:
        assert rel_err(by_region, by_list) < 1e-6
    # the autograd function takes the region form for this list
    q = torch.zeros(L, C, dtype=dtype, device=DEV, requires_grad=True)
    tok = layers.grained_sample_decompress(q, patches, torch.zeros(B, N, C, dtype=dtype, device=DEV), G, G, 1, False)
    gq, = torch.autograd.grad(tok, q, g)
    assert torch.equal(gq, by_region)
    # ... and the list walk for a list without them
    plain = patches.clone()
    tok = layers.grained_sample_decompress(q, plain, torch.zeros(B, N, C, dtype=dtype, device=DEV), G, G, 1, False)
    gq2, = torch.autograd.grad(tok, q, g)
    assert torch.equal(gq2, by_list)


def test_unpool_grad_region_form_skips_rows_beyond_the_declared_count(layers):
    """First rows supplied by the caller are checked against the declared row count: with grad_q declared 40
    rows shorter than the buffer the test owns, the regions whose patches end beyond that are skipped, the
    rows beyond stay untouched and the status word is set.  Nothing points outside an allocation."""
    import ctypes
    from vtpack_b200 import _lib
    from vtpack_b200.runtime import dtype_code, ptr, stream_ptr
    lib = _lib.lib()
    B, G, C = 2, 16, 384
    indices = torch.zeros(B, 4, 4, dtype=torch.int64, device=DEV)            # every region at the finest grain
    patches, _ = layers.grained_sample_index_to_patch(indices, torch.tensor([4, 2, 1]), 4, 1)
    L, N = patches.shape[0], G * G + 1
    idx32, first, _, _, Hr, Wr, _ = patches._vtp_regions
    g = torch.randn(B, N, C, device=DEV).bfloat16()
    out = torch.full((L, C), 7.0, dtype=torch.bfloat16, device=DEV)
    arr = (ctypes.c_int * 3)(4, 2, 1)
    declared = L - 40
    _lib.device_status()
    _lib.check(lib.vtp_unpool_grad_regions(ptr(g), dtype_code(g.dtype), B, Hr, Wr, 4, C, 1, ptr(idx32), arr, 3,
                                           ptr(first), ptr(patches._vtp_offsets), declared, ptr(out),
                                           stream_ptr(g.device)))
    torch.cuda.synchronize()
    assert _lib.device_status() == _lib.STATUS_BAD_INDEX
    assert bool((out[declared:] == 7.0).all())
    full = torch.empty(L, C, dtype=torch.bfloat16, device=DEV)
    _lib.check(lib.vtp_unpool_grad_regions(ptr(g), dtype_code(g.dtype), B, Hr, Wr, 4, C, 1, ptr(idx32), arr, 3,
                                           ptr(first), ptr(patches._vtp_offsets), L, ptr(full), stream_ptr(g.device)))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    kept = int(first.reshape(-1)[first.reshape(-1) + 16 <= declared].max()) + 16     # rows of the regions that fit
    assert torch.equal(out[:kept], full[:kept])


def test_ragged_products_match_reference(layers, golden_dir):
    z = _golden(golden_dir, "train_ops_fp32.npz")
    h, d, N = 2, 8, 12
    la, lb = torch.tensor([5, 17, 9]), torch.full([3], N, dtype=torch.long)
    L = int(la.sum())
    q = O.randn_seeded((h, L, d), 31).to(DEV).requires_grad_(True)
    k = O.randn_seeded((h, 3 * N, d), 32).to(DEV).requires_grad_(True)
    v = O.randn_seeded((h, 3 * N, d), 33).to(DEV).requires_grad_(True)
    p = O.randn_seeded((h, L, N), 35).to(DEV).requires_grad_(True)
    s = layers.batched_sparse_gemm(q, k, la, lb, False, True)
    o = layers.batched_sparse_gemm(p, v, la, lb, False, False)
    gq, gk = torch.autograd.grad(s, (q, k), O.randn_seeded((h, L, N), 34).to(DEV))
    gp, gv = torch.autograd.grad(o, (p, v), O.randn_seeded((h, L, d), 36).to(DEV))
    for name, t in (("gemm_s", s), ("gemm_o", o), ("gemm_gq", gq), ("gemm_gk", gk), ("gemm_gp", gp), ("gemm_gv", gv)):
        assert t.shape == z[name].shape, name
        assert rel_err(t.detach(), z[name]) < 1e-5, name


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False)])
def test_ragged_products_all_flag_combinations(layers, dtype, ta, tb):
    """The transpose combinations the forward and backward passes use (both operands transposed
    would need the same row count in every image on both sides), ragged lengths (an empty image included) and sizes that are not
    multiples of the tile, against the CPU restatement in float64."""
    h, B, ka = 3, 4, 70
    la = torch.tensor([67, 0, 129, 5])
    gen = torch.Generator().manual_seed(17 + 2 * ta + tb)
    a = torch.randn(h, int(la.sum()), ka, generator=gen).to(dtype)
    if ta:          # op(a_i) is [ka, la]: b_i needs la rows (or la columns when transposed)
        lb = la if not tb else torch.full([B], 33, dtype=torch.long)
        kb = 41 if not tb else None
    else:           # op(a_i) is [la, ka]: b_i needs ka rows (or ka columns when transposed)
        lb = torch.full([B], ka, dtype=torch.long) if not tb else torch.full([B], 33, dtype=torch.long)
        kb = 41 if not tb else ka
    b = torch.randn(h, int(lb.sum()), kb, generator=gen).to(dtype)
    ref = O.batched_sparse_gemm_forward(a.double(), b.double(), la, lb, ta, tb)
    out = layers.batched_sparse_gemm(a.to(DEV), b.to(DEV), la, lb, ta, tb)
    assert out.shape == ref.shape and out.dtype == dtype
    assert rel_err(out.float(), ref) < (1e-5 if dtype == torch.float32 else 8e-3)


@pytest.mark.parametrize("keys,d,las", [(257, 64, [113, 41, 257, 0, 130]), (264, 64, [70, 129]), (65, 64, [33, 7]),
                                        (1025, 32, [300, 5])])
def test_ragged_products_model_shapes_bf16(layers, keys, d, las):
    """The six products of the training-mode attention (forward S = Q K^T and O = P V; backward dP = dO V^T,
    dQ = dS K, dK = dS^T Q, dV = P^T dO) at the model's shapes: 257 keys (rows of 514 bytes: unaligned rows, a
    one-column tail beside the 256-column tile, a reduction of 4 x 64 + 1), query counts below, at and above
    one 128-row tile, an image without queries; also 264 keys (an 8-column tail), 65 and 1025.  bf16 on tensor
    cores against float64 on the bf16-rounded operands."""
    h = 3
    B = len(las)
    la, lb = torch.tensor(las), torch.full([B], keys, dtype=torch.long)
    L = int(la.sum())
    gen = torch.Generator().manual_seed(keys + d + L)
    q = torch.randn(h, L, d, generator=gen).bfloat16()
    k = torch.randn(h, B * keys, d, generator=gen).bfloat16()
    p = torch.randn(h, L, keys, generator=gen).bfloat16()
    cases = [("S = Q K^T", q, k, la, lb, False, True), ("O = P V", p, k, la, lb, False, False),
             ("dK = dS^T Q", p, q, la, la, True, False)]
    for name, a, b, xa, xb, ta, tb in cases:
        ref = O.batched_sparse_gemm_forward(a.double(), b.double(), xa, xb, ta, tb)
        out = layers.batched_sparse_gemm(a.to(DEV), b.to(DEV), xa, xb, ta, tb)
        torch.cuda.synchronize()
        assert out.shape == ref.shape and out.dtype == torch.bfloat16, name
        assert rel_err(out.float(), ref) < 8e-3, name
    # operands that start 2 bytes into their storage (a view) cannot be fetched with aligned 16-byte loads: the
    # call takes the CUDA-core kernel and gives the same product to bf16 rounding
    def shifted(t):
        buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
        view = buf[1:].view(t.shape)
        view.copy_(t)
        assert view.data_ptr() % 16 != 0
        return view
    ref = O.batched_sparse_gemm_forward(q.double(), k.double(), la, lb, False, True)
    out = layers.batched_sparse_gemm(shifted(q), shifted(k), la, lb, False, True)
    assert rel_err(out.float(), ref) < 8e-3
    from vtpack_b200 import _lib
    assert _lib.device_status() == 0


def _train_block(mode):
    from vtpack_b200.models.dge import deit_dge
    cfg = O.TRAIN_BLOCK
    blk = deit_dge.Block(cfg["dim"], cfg["heads"], mlp_ratio=4, qkv_bias=True,
                         norm_layer=lambda d: torch.nn.LayerNorm(d, eps=1e-6), split_sizes=[4, 2, 1])
    blk.load_state_dict(O.train_block_weights(), strict=True)
    blk.to(DEV).train()
    blk.dge.sparse_train = mode == "sparse"
    return blk, cfg


@pytest.mark.parametrize("mode", ["sparse", "dense"])
def test_training_block_matches_reference(golden_dir, mode):
    """Forward value, input gradient, every parameter gradient and the complexity term of one
    training-mode block, with the reference's Gumbel noise injected."""
    z = _golden(golden_dir, "train_block_fp32.npz")
    blk, cfg = _train_block(mode)
    x = O.randn_seeded((cfg["batch"], 257, cfg["dim"]), cfg["token_seed"]).to(DEV).requires_grad_(True)
    g = O.randn_seeded((cfg["batch"], 257, cfg["dim"]), cfg["grad_seed"]).to(DEV)
    real = F.gumbel_softmax
    F.gumbel_softmax = O.gumbel_softmax_fixed([O.make_gumbel_noise((cfg["batch"], 4, 4, 3), cfg["noise_seed"])])
    try:
        y = blk(x)
        comp = blk.dge.get_complexity()
        ((y * g).sum() + 1e-9 * comp["dynamic"].sum()).backward()
    finally:
        F.gumbel_softmax = real
    assert torch.equal(torch.as_tensor(blk.dge.states["batches"]).cpu(), z[f"{mode}_lengths"])
    assert rel_err(comp["dynamic"].detach(), z[f"{mode}_comp_dynamic"]) < 1e-12
    assert rel_err(y.detach(), z[f"{mode}_out"]) < TOL
    assert rel_err(x.grad, z[f"{mode}_grad_x"]) < TOL
    checked = 0
    for name, prm in blk.named_parameters():
        key = f"{mode}_grad.{name}"
        if key in z:
            assert prm.grad is not None, name
            assert rel_err(prm.grad, z[key]) < 5 * TOL, name
            checked += 1
    assert checked == 16          # two LayerNorms, five Linears and the gate: weight and bias each


def test_training_model_step_and_eval_after():
    """A DeiT-Ti+DGE model takes an SGD step in training mode (sparse_train on): gradients reach the
    router and the patch embedding, and the fused eval forward afterwards runs on the updated
    weights (its packed copies are rebuilt)."""
    from vtpack_b200.models.dge import deit_dge
    torch.manual_seed(0)
    m = deit_dge.deit_dge_s124_tiny_patch16_256().to(DEV)
    for blk in m.blocks:
        blk.dge.sparse_train = True
    images = O.make_images(4, 256, seed=3).to(DEV)
    m.eval()
    with torch.no_grad():
        logits_before = m(images).clone()
    m.train()
    target = torch.tensor([1, 2, 3, 4], device=DEV)
    opt = torch.optim.SGD(m.parameters(), lr=1e-2)
    before = m.blocks[0].dge.router.gate.weight.detach().clone()
    logits = m(images)
    assert logits.shape == (4, 1000) and logits.requires_grad
    budget = torch.stack([blk.dge.get_complexity()["dynamic"].mean() for blk in m.blocks]).sum()
    loss = F.cross_entropy(logits, target) + 1e-10 * budget
    loss.backward()
    assert torch.isfinite(loss)
    params = dict(m.named_parameters())
    for name in ("patch_embed.proj.weight", "blocks.0.dge.router.gate.weight", "blocks.11.attn.kv.weight"):
        grad = params[name].grad
        assert grad is not None and torch.isfinite(grad).all() and grad.abs().max() > 0, name
    opt.step()
    assert not torch.equal(before, m.blocks[0].dge.router.gate.weight.detach())
    m.eval()
    with torch.no_grad():
        logits_after = m(images)
    assert torch.isfinite(logits_after).all() and not torch.equal(logits_after, logits_before)


def test_training_pvt_block_matches_reference(golden_dir):
    """A PVT+DGE block with spatial-reduction keys in training mode (sparse_train on): output,
    input gradient and all parameter gradients against the reference's."""
    from functools import partial
    from vtpack_b200.models.dge import pvt_dge
    z = _golden(golden_dir, "train_pvt_block_fp32.npz")
    cfg = O.TRAIN_PVT_BLOCK
    blk = pvt_dge.Block(cfg["dim"], cfg["heads"], mlp_ratio=cfg["mlp_ratio"], qkv_bias=True,
                        norm_layer=partial(torch.nn.LayerNorm, eps=1e-6), sr_ratio=cfg["sr"], split_sizes=[4, 2, 1])
    blk.load_state_dict(O.make_pvt_block_weights(cfg["dim"], cfg["mlp_ratio"], cfg["sr"], seed=cfg["weight_seed"]),
                        strict=True)
    blk.to(DEV).train()
    blk.dge.sparse_train = True
    G = cfg["grid"]
    x = O.randn_seeded((cfg["batch"], G * G, cfg["dim"]), cfg["token_seed"]).to(DEV).requires_grad_(True)
    g = O.randn_seeded((cfg["batch"], G * G, cfg["dim"]), cfg["grad_seed"]).to(DEV)
    real = F.gumbel_softmax
    F.gumbel_softmax = O.gumbel_softmax_fixed([O.make_gumbel_noise((cfg["batch"], G // 4, G // 4, 3), cfg["noise_seed"])])
    prev = torch.backends.cudnn.allow_tf32
    torch.backends.cudnn.allow_tf32 = False          # the reduction convolution in full fp32
    try:
        y = blk(x, G, G)
        (y * g).sum().backward()
    finally:
        F.gumbel_softmax = real
        torch.backends.cudnn.allow_tf32 = prev
    assert torch.equal(blk.dge.states["batches"].cpu(), z["lengths"])
    assert rel_err(y, z["out"]) < TOL
    assert rel_err(x.grad, z["grad_x"]) < TOL
    checked = 0
    for name, prm in blk.named_parameters():
        if f"grad.{name}" in z:
            assert rel_err(prm.grad, z[f"grad.{name}"]) < 5 * TOL, name
            checked += 1
    assert checked == 20          # DeiT block's 16 plus the reduction convolution and its LayerNorm


def test_training_pvt_model_matches_reference(golden_dir):
    """PVT+DGE tiny in training mode (sparse_train on, one injected Gumbel-noise tensor per block):
    the same per-block query counts, logits, loss and parameter gradients as the reference."""
    from vtpack_b200.models.dge import pvt_dge
    z = _golden(golden_dir, "train_pvt_model_fp32.npz")
    cfg, t = O.PVT_CONFIGS["tiny"], O.TRAIN_PVT_MODEL
    m = pvt_dge.pvt_dge_s124_tiny_256()
    m.load_state_dict(O.make_pvt_state_dict(cfg, seed=t["weight_seed"]), strict=True)
    m.to(DEV).train()
    blocks = [b for i in range(4) for b in getattr(m, f"block{i + 1}")]
    for b in blocks:
        b.dge.sparse_train = True
    x = O.make_images(t["batch"], 256, seed=t["image_seed"]).to(DEV)
    real = F.gumbel_softmax
    F.gumbel_softmax = O.gumbel_softmax_fixed(O.train_pvt_model_noises(cfg))
    prev = torch.backends.cudnn.allow_tf32
    torch.backends.cudnn.allow_tf32 = False          # the patch and reduction convolutions in full fp32
    try:
        logits = m(x)
        counts = torch.stack([b.dge.states["batches"].cpu() for b in blocks])
        loss = F.cross_entropy(logits, torch.tensor(t["target"], device=DEV))
        loss.backward()
    finally:
        F.gumbel_softmax = real
        torch.backends.cudnn.allow_tf32 = prev
    assert torch.equal(counts, z["counts"])
    assert rel_err(logits, z["logits"]) < TOL
    assert abs(float(loss.detach()) - float(z["loss"])) < 1e-4
    params = dict(m.named_parameters())
    for name in t["grads"]:
        assert rel_err(params[name].grad, z[f"grad.{name}"]) < 1e-3, name
    # the feature-pyramid variant returns the four stage maps
    m.num_classes = 0
    F.gumbel_softmax = O.gumbel_softmax_fixed(O.train_pvt_model_noises(cfg))
    try:
        with torch.no_grad():
            feats = m(x)
    finally:
        F.gumbel_softmax = real
    assert [tuple(feats[f"res{i}"].shape) for i in (2, 3, 4, 5)] == [(2, 64, 64, 64), (2, 128, 32, 32),
                                                                       (2, 320, 16, 16), (2, 512, 8, 8)]


def _ragged_case(B, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    la = torch.randint(0, 9, (B,), generator=g)
    la[0] = 7
    lb = la.new_full([B], 5)
    a = torch.randn(2, int(la.sum()), 16, generator=g).to(dtype)
    b = torch.randn(2, int(lb.sum()), 16, generator=g).to(dtype)
    return a, b, la, lb


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 8e-3)])
@pytest.mark.parametrize("B", [1, 512, 513])
def test_ragged_product_image_counts(layers, dtype, tol, B):
    """Offsets that travel with the launch (up to 512 images) and offsets in device memory (more): the product and
    both gradients, empty images among them; changing the caller's lengths after the forward changes nothing."""
    a, b, la, lb = _ragged_case(B, dtype, B)
    ref_a, ref_b = a.double().requires_grad_(True), b.double().requires_grad_(True)
    ref = O.batched_sparse_gemm_forward(ref_a, ref_b, la, lb, False, True)
    go = torch.randn(ref.shape, generator=torch.Generator().manual_seed(3)).to(dtype)
    want = torch.autograd.grad(ref, (ref_a, ref_b), go.double())
    x, y = a.to(DEV).requires_grad_(True), b.to(DEV).requires_grad_(True)
    out = layers.batched_sparse_gemm(x, y, la, lb, False, True)
    la.zero_()
    got = torch.autograd.grad(out, (x, y), go.to(DEV))
    for t, r in zip((out,) + got, (ref,) + want):
        assert rel_err(t.float(), r) < tol


@pytest.mark.parametrize("dt", [torch.int32, torch.int64])
@pytest.mark.parametrize("extra,splits", [(0, [4, 2, 1]), (1, [4, 2, 1]), (2, [2, 1])])
def test_region_rows_of_patch_list(layers, dt, extra, splits):
    """The per-region first rows that come with a patch list, against their prefix-sum definition."""
    B, Hr, Wr = 5, 3, 7
    idx = torch.randint(0, len(splits), (B, Hr, Wr), generator=torch.Generator().manual_seed(extra), dtype=dt)
    patches, lengths = layers.grained_sample_index_to_patch(idx.to(DEV), torch.tensor(splits), max(splits), extra)
    idx32, first = patches._vtp_regions[:2]
    per = torch.tensor(splits)[idx.reshape(B, -1).long()] ** 2
    start = torch.cumsum(lengths, 0) - lengths
    want = start[:, None] + extra + torch.cumsum(per, 1) - per
    assert torch.equal(first.cpu().long(), want) and torch.equal(idx32.cpu().long(), idx.reshape(B, -1).long())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,G,C,extra", [(3, 4, 192, 1), (2, 3, 64, 0), (5, 2, 384, 2), (2, 4, 320, 1), (3, 2, 768, 1), (2, 2, 512, 0)])
def test_gated_decompress_is_the_sequence_of_operations(layers, dtype, B, G, C, extra):
    """The gated decompress of the training path as one launch each way against the operations it stands for: output and row gradients
    bit for bit; the gate's gradient, a sum of n = 16 C products (or fewer) in fp32, within n 2^-24 of the sum of their magnitudes and one
    rounding of the result.  Gate values that are not quite 1, every grain, an image of one grain."""
    from vtpack_b200.layers import dge, grained_sample as gs
    g = torch.Generator(DEV).manual_seed(C + B)
    N, W = extra + 16 * G * G, 4 * G
    idx = torch.randint(0, 3, (B, G, G), device=DEV, generator=g)
    idx[0] = 1
    gate = torch.zeros(B, G, G, 3, device=DEV).scatter_(3, idx[..., None], 1.0) * (1 + 0.01 * torch.rand(B, G, G, 3, device=DEV, generator=g))
    patches, _ = gs.grained_sample_index_to_patch(idx, torch.tensor([4, 2, 1]), 4, extra)
    L = patches.shape[0]
    leaves = [torch.randn(L, C, device=DEV, generator=g), torch.randn(L, C, device=DEV, generator=g), gate, torch.randn(B, N, C, device=DEV, generator=g)]
    grad = torch.randn(B, N, C, device=DEV, generator=g).to(dtype)
    enc = dge.DynamicGrainedEncoder(C, [4, 2, 1], sparse_train=True).to(DEV).train()

    def run(fused):
        x, comp, gt, ref = (t.to(dtype).requires_grad_(True) for t in leaves)
        listed = patches if fused else patches.clone()            # (a copy does not say which grains it was made from)
        enc.states.update(comp=comp, gate=gt, input=ref, patches=listed, size=(4 * G, W), num_extra_tokens=extra)
        out = enc.decompress(x)
        assert ("GatedDecompress" in type(out.grad_fn).__name__) == fused
        return out, torch.autograd.grad(out, (x, comp, gt, ref), grad)
    out, (gx, gc, gg, gr) = run(True)
    want, (_, _, wg, wr) = run(False)
    # the sequence pools the gate over its patches, which in fp32 rounds it: 16 additions of a value of about 1
    assert torch.equal(out, want) if dtype is torch.bfloat16 else float((out - want).detach().abs().max()) <= 16 * 2.0 ** -24 * 12
    assert torch.equal(gr, wr)
    first = patches[:, 1] < 0
    val = torch.ones(L, 1, device=DEV, dtype=dtype)
    region = (patches[:, 0] * G + torch.div(patches[:, 1], 4, rounding_mode="floor")) * G + torch.div(patches[:, 2], 4, rounding_mode="floor")
    picked = gate.to(dtype).gather(3, idx[..., None]).reshape(-1)
    val[~first, 0] = picked[region[~first]]
    x, comp, ref = (leaves[i].to(dtype) for i in (0, 1, 3))
    rows = ((x - comp) * val).requires_grad_(True)
    y = gs.grained_sample_decompress(rows, patches, ref, 4 * G, W, extra, True)
    assert torch.equal(out, y)
    r, = torch.autograd.grad(y, rows, grad)
    assert torch.equal(gx, r * val) and torch.equal(gc, -(r * val))
    prod = (r.double() * (x - comp).double())[~first]
    exact = torch.zeros(B * G * G, device=DEV, dtype=torch.double).index_add_(0, region[~first], prod.sum(1))
    size = torch.zeros_like(exact).index_add_(0, region[~first], prod.abs().sum(1))
    got = gg.double().gather(3, idx[..., None]).reshape(-1)
    eps = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -23
    assert bool(((got - exact).abs() <= 16 * C * 2.0 ** -24 * size + eps * exact.abs()).all())
    assert int((gg != 0).sum()) <= B * G * G and float((gg - wg).abs().max()) <= 0.05 * float(wg.abs().max()) + 1e-3
    from vtpack_b200 import _lib
    assert _lib.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lengths,M,heads,d", [([197, 3, 50], 197, 6, 64), ([1, 0, 5], 49, 1, 64), ([17, 64], 64, 2, 64), ([9, 2], 1, 3, 64), ([4, 30], 1100, 2, 64)])
def test_ragged_attention_is_the_sequence_of_operations(layers, dtype, lengths, M, heads, d):
    """The training attention as one node against float64 attention of the same inputs, output and both gradients no further off than the
    separate operations are (plus the two roundings' worth that separates orders of one sum); sums of one key, more keys than a lane
    keeps, images without queries."""
    from vtpack_b200.layers import sparse_ops
    g = torch.Generator(DEV).manual_seed(M)
    B, L, C = len(lengths), sum(lengths), heads * d
    ln = torch.tensor(lengths)
    q0 = torch.randn(L, C, device=DEV, generator=g).to(dtype)
    kv0 = torch.randn(B, M, 2 * C, device=DEV, generator=g).to(dtype)
    w = torch.randn(L, C, device=DEV, generator=g).to(dtype)
    drop, scale = torch.nn.Dropout(0.0), d ** -0.5

    def one(q, kv):
        return sparse_ops.ragged_attention(q, kv, ln, heads, scale, drop)

    def separate(q, kv):
        qh = q.reshape(-1, heads, d).permute(1, 0, 2)
        k, v = (t.reshape(heads, -1, d) for t in kv.reshape(B, M, 2, heads, d).permute(2, 3, 0, 1, 4))
        n = ln.new_full([B], M)
        p = (sparse_ops.batched_sparse_gemm(qh, k, ln, n, False, True) * scale).softmax(-1, dtype=v.dtype)
        return sparse_ops.batched_sparse_gemm(p, v, ln, n, False, False).transpose(0, 1).reshape(-1, C)

    def exact(q, kv):
        k, v = kv.reshape(B, M, 2, heads, d).permute(2, 0, 3, 1, 4)
        rows = [((x.reshape(-1, heads, d).transpose(0, 1) @ k[b].transpose(-1, -2)) * scale).softmax(-1) @ v[b]
                for b, x in enumerate(q.split(lengths))]
        return torch.cat(rows, 1).transpose(0, 1).reshape(-1, C)

    def run(f, dt):
        q, kv = q0.to(dt).requires_grad_(True), kv0.to(dt).requires_grad_(True)
        y = f(q, kv)
        return [t.double() for t in (y.detach(), *torch.autograd.grad(y, (q, kv), w.to(dt)))]
    got, old, want = run(one, dtype), run(separate, dtype), run(exact, torch.float64)
    eps = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -23
    for a, b, e in zip(got, old, want):
        size = float(e.abs().max())
        assert float((a - e).norm()) <= float((b - e).norm()) * 1.1 + eps / 4 * float(e.norm())
        assert float((a - e).abs().max()) <= 1.5 * float((b - e).abs().max()) + 2 * eps * size
    assert one(q0, kv0[:, :, :-2]) is None and sparse_ops.ragged_attention(q0, kv0, ln, heads, scale, torch.nn.Dropout(0.1)) is None


def test_scaled_softmax_of_rows_without_a_value():
    """Scores of -inf, +inf and NaN, and a negative scale, as softmax(scale * s) gives them."""
    from vtpack_b200 import _lib
    from vtpack_b200.runtime import dtype_code, ptr, stream_ptr
    inf, nan = float("inf"), float("nan")
    for n in (3, 70, 1200):
        s = torch.randn(6, n, device=DEV)
        s[0, 1:], s[1], s[2, 0], s[3, 0] = -inf, -inf, nan, inf
        for scale in (0.125, -0.5):
            p = torch.empty_like(s)
            _lib.check(_lib.lib().vtp_scaled_softmax(ptr(s), dtype_code(s.dtype), 6, n, scale, ptr(p), stream_ptr(s.device)))
            want = (s.double() * scale).softmax(-1)
            assert torch.equal(p.isnan(), want.isnan())
            ok = ~want.isnan()
            assert float((p.double() - want)[ok].abs().max()) <= 2.0 ** -20


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [16, 65, 257, 1200])
@pytest.mark.parametrize("spread", [1.0, 8.0])
def test_scaled_softmax_is_no_further_off_than_the_operations_it_stands_for(dtype, n, spread):
    """Error in the 2-norm against float64 of softmax and gradient over 4096 rows, beside that of PyTorch's operations on the same rows.  Both
    round each value as often; over 65536 values and more the two norms scatter by 1 / sqrt(2 * 65536) = 0.3 %, and the sums' orders
    differ.  (Sums over lanes of a warp in one, of a block in the other: 2 % is allowed.)"""
    from vtpack_b200 import _lib
    from vtpack_b200.runtime import dtype_code, ptr, stream_ptr
    g = torch.Generator(DEV).manual_seed(n)
    scale = 0.125
    s = (spread / scale * torch.randn(4096, n, device=DEV, generator=g)).to(dtype)
    dp = torch.randn(4096, n, device=DEV, generator=g).to(dtype)
    p, ds = torch.empty_like(s), torch.empty_like(s)
    args = (dtype_code(dtype), 4096, n, scale)
    ops = (s * scale).softmax(-1, dtype=dtype)
    _lib.check(_lib.lib().vtp_scaled_softmax(ptr(s), *args, ptr(p), stream_ptr(s.device)))
    _lib.check(_lib.lib().vtp_scaled_softmax_grad(ptr(ops), ptr(dp), *args, ptr(ds), stream_ptr(s.device)))
    grad = torch._softmax_backward_data(dp, ops, -1, dtype) * scale
    q, d = ops.double(), dp.double()
    for got, old, want in ((p, ops, (s.double() * scale).softmax(-1)), (ds, grad, scale * q * (d - (q * d).sum(-1, keepdim=True)))):
        assert float((got.double() - want).norm()) <= 1.02 * float((old.double() - want).norm())
