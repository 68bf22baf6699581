"""Counterparts of ``vtpack/layers/sparse_ops.py``: ``batched_sparse_attention(q, k, v, q_lengths,
scale)`` (eval; ``sparse_ops.py:60-78``) and the differentiable ragged product
``batched_sparse_gemm(a, b, a_lengths, b_lengths, is_a_transposed, is_b_transposed)`` of the
training path (``sparse_ops.py:11-57``)."""
import torch
from torch.autograd import Function
from torch.autograd.function import once_differentiable

from .. import _lib
from ..runtime import dtype_code, ptr, require_cuda, stream_ptr


def batched_sparse_attention(q, k, v, q_lengths, scale, flags: int = 0):
    """q [h,L,d], k/v [h,B,N,d], q_lengths int [B] (CPU, as in the reference) -> [h,L,d].

    The operands may be the permuted views the model makes of its Linear outputs; they
    are read through their strides, so the ``.contiguous()`` copies of the reference
    (``sparse_ops.py:64-66``) do not happen.  The result is a [h,L,d] view of an
    [L,h,d] buffer, so the model's ``transpose(0,1).reshape(-1,C)`` is free.
    """
    require_cuda(q, k, v)
    h, L, d = q.shape
    _, B, N, _ = k.shape
    if q.stride(2) != 1:
        q = q.contiguous()
    if k.stride(3) != 1 or v.stride(3) != 1 or k.stride() != v.stride():
        k, v = k.contiguous(), v.contiguous()
    lengths = q_lengths.to("cpu", torch.int64)
    offsets = torch.zeros(B + 1, dtype=torch.int32)
    offsets[1:] = torch.cumsum(lengths, 0)
    assert int(offsets[-1]) == L, "q_lengths do not add up to the number of query rows"
    offsets = offsets.to(q.device, non_blocking=True)
    out = torch.empty(L, h, d, dtype=q.dtype, device=q.device)
    _lib.check(_lib.lib().vtp_sparse_attention(
        ptr(q), q.stride(1), q.stride(0), ptr(k), ptr(v), k.stride(1), k.stride(2), k.stride(0),
        ptr(out), h * d, d, dtype_code(q.dtype), B, N, h, d, ptr(offsets), L,
        int(lengths.max()) if B > 0 else 0, float(scale), int(flags), stream_ptr(q.device)))
    return out.permute(1, 0, 2)


class _Lengths:
    """The per-image row counts of an operand, read once for the forward and the backward products."""

    def __init__(self, lengths):
        self.host = lengths.to("cpu", torch.int64).contiguous().clone()
        values = self.host.tolist()
        self.n, self.total = len(values), sum(values)
        self.max, self.min = (max(values), min(values)) if values else (0, 0)

    def offsets(self, device):
        off = torch.zeros(self.n + 1, dtype=torch.int32)
        off[1:] = torch.cumsum(self.host, 0)
        return off.to(device, non_blocking=True)


_INLINE_IMAGES = 512            # the library passes the offsets of up to this many images with the launch


def _ragged_gemm(a, b, la, lb, ta, tb, out=None):
    """One launch of the ragged product: a [H,La,ka], b [H,Lb,kb] -> the per-image products
    stacked along dim 1 (``batched_sparse_gemm.cu:150-196``), in `out` (dense, of that shape) if it is given."""
    require_cuda(a, b)
    a, b = a.contiguous(), b.contiguous()
    H, B = a.shape[0], la.n
    assert la.total <= a.shape[1] and lb.total <= b.shape[1], "lengths exceed the rows of the operands"
    if tb:
        assert b.shape[1] % B == 0 and lb.min == lb.max, \
            "a transposed b needs the same number of rows in every image"
    out_rows = B * a.shape[2] if ta else la.total
    out_cols = lb.max if tb else b.shape[2]
    if out is None:
        out = torch.empty(H, out_rows, out_cols, dtype=a.dtype, device=a.device)
    lib = _lib.lib()
    head = (ptr(a), ptr(b), ptr(out), dtype_code(a.dtype), H, B, a.shape[1], a.shape[2], b.shape[1], b.shape[2])
    tail = (int(bool(ta)), int(bool(tb)), out_rows, out_cols, stream_ptr(a.device))
    if 0 < B <= _INLINE_IMAGES and la.min >= 0 and lb.min >= 0 and lb.n == B:
        _lib.check(lib.vtp_batched_sparse_gemm_lengths(*head, ptr(la.host), ptr(lb.host), *tail))
    else:
        a_off, b_off = la.offsets(a.device), lb.offsets(a.device)
        _lib.check(lib.vtp_batched_sparse_gemm(*head, ptr(a_off), ptr(b_off), la.max, lb.max, *tail))
    return out


class _BatchedSparseGEMM(Function):
    """Forward and backward are the same kernel with other transpose flags, wired as in
    ``sparse_ops.py:30-55``."""

    @staticmethod
    def forward(ctx, a, b, a_lengths, b_lengths, is_a_transposed, is_b_transposed):
        a, b = a.contiguous(), b.contiguous()
        ctx.ta, ctx.tb = bool(is_a_transposed), bool(is_b_transposed)
        la = _Lengths(a_lengths)
        lb = la if b_lengths is a_lengths else _Lengths(b_lengths)
        ctx.lengths = (la, lb)
        ctx.save_for_backward(a, b)
        return _ragged_gemm(a, b, la, lb, ctx.ta, ctx.tb)

    @staticmethod
    @once_differentiable
    def backward(ctx, grad_output):
        a, b = ctx.saved_tensors
        la, lb = ctx.lengths
        g = grad_output.contiguous()
        if not ctx.ta:
            grad_a = _ragged_gemm(g, b, la, lb, False, not ctx.tb)
        else:
            grad_a = _ragged_gemm(b, g, lb, la, ctx.tb, True)
        if not ctx.tb:
            grad_b = _ragged_gemm(a, g, la, la, not ctx.ta, False)
        else:
            grad_b = _ragged_gemm(g, a, la, la, True, ctx.ta)
        return grad_a, grad_b, None, None, None, None


batched_sparse_gemm = _BatchedSparseGEMM.apply


class _RaggedAttention(Function):
    """softmax(scale * q k^T) v of every image and head, q [L,C] (an image's queries behind those of the one in front), kv [B,M,2C]
    -> [L,C]: the two ragged products with the softmax between them (``deit_dge.py:87-95`` of the reference) and the layout changes
    around them as one node."""

    @staticmethod
    def forward(ctx, q, kv, q_lengths, heads, scale):
        L, C = q.shape
        B, M, _ = kv.shape
        d = C // heads
        la, lb = _Lengths(q_lengths), _Lengths(q_lengths.new_full([B], M))
        qh = q.reshape(L, heads, d).transpose(0, 1).contiguous()
        kvh = kv.reshape(B, M, 2, heads, d).permute(2, 3, 0, 1, 4).contiguous().view(2, heads, B * M, d)
        p = _ragged_gemm(qh, kvh[0], la, lb, False, True)
        _lib.check(_lib.lib().vtp_scaled_softmax(ptr(p), dtype_code(p.dtype), heads * L, M, scale, ptr(p), stream_ptr(p.device)))
        ctx.save_for_backward(qh, kvh, p)
        ctx.lengths, ctx.scale, ctx.shapes = (la, lb), scale, (q.shape, kv.shape)
        return _ragged_gemm(p, kvh[1], la, lb, False, False).transpose(0, 1).reshape(L, C)

    @staticmethod
    @once_differentiable
    def backward(ctx, grad_output):
        qh, kvh, p = ctx.saved_tensors
        la, lb = ctx.lengths
        (L, C), (B, M, _) = ctx.shapes
        heads, _, d = qh.shape
        g = grad_output.reshape(L, heads, d).transpose(0, 1).contiguous()
        grads = torch.empty_like(kvh)
        _ragged_gemm(p, g, la, la, True, False, out=grads[1])
        ds = _ragged_gemm(g, kvh[1], la, lb, False, True)
        _lib.check(_lib.lib().vtp_scaled_softmax_grad(ptr(p), ptr(ds), dtype_code(p.dtype), heads * L, M, ctx.scale, ptr(ds),
                                                      stream_ptr(p.device)))
        _ragged_gemm(ds, qh, la, la, True, False, out=grads[0])
        grad_q = _ragged_gemm(ds, kvh[0], la, lb, False, False).transpose(0, 1).reshape(L, C)
        grad_kv = grads.view(2, heads, B, M, d).permute(2, 3, 0, 1, 4).reshape(B, M, 2 * C)
        return grad_q, grad_kv, None, None, None


def ragged_attention(q, kv, q_lengths, heads, scale, drop):
    """``_RaggedAttention`` where it is what the separate operations are: no dropout of its weights (`drop`, the module for it), rows of one
    supported type on one GPU and lengths that add up; None elsewhere."""
    if (type(drop) is not torch.nn.Dropout or drop.p != 0.0 or drop._forward_hooks or drop._forward_pre_hooks
            or drop._backward_hooks or drop._backward_pre_hooks or not isinstance(scale, (int, float))
            or q.dim() != 2 or kv.dim() != 3 or q.dtype is not kv.dtype or q.dtype not in (torch.float32, torch.bfloat16)
            or not (q.is_cuda and kv.is_cuda) or q.device != kv.device or kv.shape[2] != 2 * q.shape[1]
            or q.shape[1] % heads != 0 or q_lengths.shape != kv.shape[:1] or kv.shape[1] == 0
            or int(q_lengths.sum()) != q.shape[0]):
        return None
    return _RaggedAttention.apply(q, kv, q_lengths, heads, float(scale))
