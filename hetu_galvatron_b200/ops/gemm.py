"""GEMM entry points over the tcgen05 kernel (csrc/gemm_sm100.cu).

``gemm`` computes ``C[M,N] = alpha * A[M,K] @ B[N,K]^T (+bias) (+residual) (+C)``; either operand
may be handed over in its transposed storage (``a_mn`` / ``b_mn``), which is how the input- and
weight-gradient GEMMs of a linear layer read ``dY``, ``W`` and ``X`` without materialising a
transpose (reference: megatron/core/tensor_parallel/layers.py:417,462,534).
"""
from __future__ import annotations

import functools
import warnings

import torch

from . import _lib


def _use_native(*ts) -> bool:
    for t in ts:
        if t is not None and not (t.is_cuda and t.dtype == torch.bfloat16):
            return False
    return True


def _row_major_2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        t = t.reshape(-1, t.shape[-1])
    ld, inner = t.stride()
    if inner != 1 or ld % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


class RopeEpilogue:
    """Rotary embedding applied by the GEMM epilogue to the first ``cols`` output columns (heads of ``dh`` = 64 or 128
    columns, non-interleaved halves): the position of output row r is ``positions[r]`` (int32) or ``r // pos_div +
    pos_offset``. Saves the separate pass over q and k that follows a packed QKV projection."""

    def __init__(self, cols: int, dh: int, inv_freq: torch.Tensor, positions=None, pos_div: int = 1, pos_offset: int = 0):
        self.cols, self.dh, self.inv_freq = int(cols), int(dh), inv_freq
        self.positions = None if positions is None else positions.to(torch.int32).contiguous()
        self.pos_div, self.pos_offset = int(pos_div), int(pos_offset)

    @staticmethod
    def supported(x: torch.Tensor, dh: int, bias) -> bool:
        return x.is_cuda and x.dtype == torch.bfloat16 and dh in (64, 128) and bias is None


@functools.lru_cache(maxsize=1024)
def _workspace_bytes(M: int, N: int, K: int) -> int:
    """Scratch of a product of these sizes whose reductions CTA pairs share, of all tiles or of the last wave's (at most 39 MB); 0: none
    is shared."""
    return _lib.lib().gv_gemm_workspace_bytes(_lib.GemmArgs(M=M, N=N, K=K))


# Products (device, M, N, K) whose scratch once did not fit. They stay unsplit: a product that was split or not as memory happened
# to be free would change its last bits from call to call, and each failed allocation first empties the allocator's cache.
_NO_SCRATCH: set = set()


def _split_scratch(M: int, N: int, K: int, device) -> "torch.Tensor | None":
    need = _workspace_bytes(M, N, K)
    if not need or (device.index, M, N, K) in _NO_SCRATCH:
        return None
    try:
        return torch.empty(need, dtype=torch.uint8, device=device)
    except torch.cuda.OutOfMemoryError:
        _scratch_did_not_fit(device.index, M, N, K, need)
        return None


def _scratch_did_not_fit(device_index: int, M: int, N: int, K: int, need: int) -> None:
    _NO_SCRATCH.add((device_index, M, N, K))
    _lib.torch_ops().no_scratch_for(device_index, M, N, K)
    warnings.warn("no room for %.0f MB of partial sums: products of %d x %d x %d run unsplit from now on" % (need / 1e6, M, N, K))


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False, out: torch.Tensor | None = None,
         out_dtype: torch.dtype | None = None, bias: torch.Tensor | None = None,
         residual: torch.Tensor | None = None, accumulate: bool = False, gelu: bool = False,
         alpha: float = 1.0, rope: "RopeEpilogue | None" = None, swiglu_out: torch.Tensor | None = None,
         gelu_out: torch.Tensor | None = None) -> torch.Tensor:
    """See module docstring. ``a`` is ``[M,K]`` (or ``[K,M]`` when ``a_mn``), ``b`` is ``[N,K]`` (or ``[K,N]``).
    ``rope``: rotate the leading q / k head columns of the output in the epilogue (see ``RopeEpilogue``).
    ``swiglu_out`` [M, N / 2] bf16: ``b`` is [gate rows | up rows]; besides the projection itself the epilogue stores
    silu(gate) * up there (see ``swiglu_epilogue_supported``). ``gelu_out`` [M, N] bf16: the epilogue also stores gelu of the
    projection there (see ``gelu_epilogue_supported``)."""
    a = _row_major_2d(a)
    b = _row_major_2d(b)
    if a_mn:
        K, M = a.shape
    else:
        M, K = a.shape
    if b_mn:
        Kb, N = b.shape
    else:
        N, Kb = b.shape
    if K != Kb:
        raise ValueError(f"gemm: reduction sizes differ ({K} vs {Kb})")
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype or a.dtype, device=a.device)
        if accumulate:
            out.zero_()
    elif out.shape != (M, N):
        out = out.view(M, N)
    native = _use_native(a, b, bias, residual) and out.dtype in (torch.bfloat16, torch.float32) \
        and (K % 8 == 0 or a_mn and b_mn) and out.stride(1) == 1
    if native and (a_mn and M % 8 or b_mn and N % 8 or out.stride(0) % 8):
        native = False
    if native:
        if residual is not None:
            residual = _row_major_2d(residual)
        args = _lib.GemmArgs(
            a.data_ptr(), b.data_ptr(), out.data_ptr(), 0 if bias is None else bias.data_ptr(),
            0 if residual is None else residual.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0),
            0 if residual is None else residual.stride(0), int(a_mn), int(b_mn), int(out.dtype == torch.float32),
            int(accumulate), int(gelu), float(alpha))
        if swiglu_out is not None:
            args.swiglu_out, args.swiglu_ld = swiglu_out.data_ptr(), swiglu_out.stride(0)
        if rope is not None:
            args.rope_cols, args.rope_dh = rope.cols, rope.dh
            args.rope_inv_freq = rope.inv_freq.data_ptr()
            args.rope_pos = _lib.p(rope.positions) or None
            args.rope_pos_div, args.rope_pos_mod, args.rope_pos_offset = rope.pos_div, 0, rope.pos_offset
        elif gelu_out is not None:
            args.gelu_out, args.gelu_ld = gelu_out.data_ptr(), gelu_out.stride(0)
        elif swiglu_out is None:
            scratch = _split_scratch(M, N, K, a.device)
            if scratch is not None:
                args.workspace, args.workspace_bytes = scratch.data_ptr(), scratch.numel()
        _lib.check(_lib.lib().gv_gemm_bf16(args, _lib.stream_ptr()), "gv_gemm_bf16")
        return out
    if rope is not None or swiglu_out is not None or gelu_out is not None:
        raise _lib.KernelError("gemm: the rotary / gated-activation epilogues need the native kernel (bf16 CUDA operands)")
    if a.is_cuda and a.dtype == torch.bfloat16 and not _lib_fallback_allowed():
        raise _lib.KernelError(f"gemm: shape/stride not supported by the sm_100a kernel: M={M} N={N} K={K}")
    # Reference path (CPU ranks, fp32/fp16 runs): plain PyTorch in the accumulation dtype.
    acc_dtype = torch.float32 if a.dtype in (torch.bfloat16, torch.float16) and not a.is_cuda else a.dtype
    am = (a.t() if a_mn else a).to(acc_dtype)
    bm = (b if b_mn else b.t()).to(acc_dtype)
    c = am @ bm
    if alpha != 1.0:
        c = c * alpha
    if bias is not None:
        c = c + bias.to(acc_dtype)
    if gelu:
        c = torch.nn.functional.gelu(c, approximate="tanh")
    if residual is not None:
        c = c + residual.reshape(M, N).to(acc_dtype)
    if accumulate:
        out.add_(c.to(out.dtype))
    else:
        out.copy_(c)
    return out


def swiglu_epilogue_supported(x: torch.Tensor, w_up: torch.Tensor) -> bool:
    """The gated-activation epilogue wants bf16 CUDA operands in natural storage and an FFN width that is a multiple of
    128 (one output tile = 128 gate columns + the 128 up columns of the same hidden units)."""
    return (_use_native(x, w_up) and w_up.dim() == 2 and w_up.shape[0] % 256 == 0 and w_up.shape[1] % 8 == 0
            and w_up.stride(1) == 1 and w_up.stride(0) % 8 == 0 and w_up.data_ptr() % 16 == 0)


def gelu_epilogue_supported(x: torch.Tensor, W: torch.Tensor, bias) -> bool:
    """The GELU epilogue wants bf16 CUDA operands in natural storage, row lengths of multiples of 8."""
    return (_use_native(x, W, bias) and W.dim() == 2 and W.shape[0] % 8 == 0 and W.shape[1] % 8 == 0 and x.numel() > 0)


def head_xent_supported(x: torch.Tensor, W: torch.Tensor) -> bool:
    """The cross-entropy epilogues need bf16 CUDA operands in their natural (K-major) storage."""
    return (_use_native(x, W) and x.dim() == 2 and W.dim() == 2 and x.shape[1] == W.shape[1] and x.shape[1] % 8 == 0
            and W.shape[0] % 8 == 0          # the backward twin stores a [tokens, vocab shard] bf16 gradient (row stride % 8)
            and x.stride(1) == 1 and W.stride(1) == 1 and x.stride(0) % 8 == 0 and W.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and W.data_ptr() % 16 == 0)


def _head_args(x, W, C):
    M, K = x.shape
    N = W.shape[0]
    return _lib.GemmArgs(A=x.data_ptr(), B=W.data_ptr(), C=_lib.p(C), bias=0, residual=0, M=M, N=N, K=K, lda=x.stride(0),
                         ldb=W.stride(0), ldc=N if C is None else C.stride(0), ldr=0, a_mn_major=0, b_mn_major=0, c_f32=0,
                         accumulate=0, act=0, alpha=1.0)


def _head_stats(x, W, labels, vocab_start: int, ignore_index: int, finish: bool):
    M, N = x.shape[0], W.shape[0]
    tiles = (N + 255) // 256
    stats = torch.empty(M, tiles, 2, dtype=torch.float32, device=x.device)
    rows = torch.empty(5, M, dtype=torch.float32, device=x.device)          # max, sum, target, log-sum-exp, loss
    labels = labels.reshape(-1).to(torch.int64).contiguous()
    mx, se, target, lse, loss = rows.unbind(0)
    xa = _lib.XentArgs(mode=1, labels=labels.data_ptr(), vocab_start=int(vocab_start), ignore_index=int(ignore_index),
                       stats=stats.data_ptr(), target=target.data_ptr(), lse=0, gscale=0)
    _lib.check(_lib.lib().gv_gemm_xent(_head_args(x, W, None), xa, _lib.stream_ptr()), "gv_gemm_xent(stats)")
    _lib.check(_lib.lib().gv_xent_merge(stats.data_ptr(), tiles, labels.data_ptr(), int(vocab_start), N, int(ignore_index), mx.data_ptr(),
                                        se.data_ptr(), target.data_ptr(), lse.data_ptr() if finish else 0,
                                        loss.data_ptr() if finish else 0, M, _lib.stream_ptr()), "gv_xent_merge")
    return mx, se, target, lse, loss


def head_xent_stats(x: torch.Tensor, W: torch.Tensor, labels: torch.Tensor, vocab_start: int = 0, ignore_index: int = -100):
    """Language-model head forward without logits: per row (max, sum exp(logit - max), target logit or 0) over this
    rank's vocabulary shard ``W`` [V_local, K], computed in the epilogue of the head GEMM from its fp32 accumulators."""
    return _head_stats(x, W, labels, vocab_start, ignore_index, False)[:3]


def head_xent_loss(x: torch.Tensor, W: torch.Tensor, labels: torch.Tensor, vocab_start: int = 0, ignore_index: int = -100):
    """(loss, log-sum-exp) per row where ``W`` is the whole vocabulary; ignored rows have loss 0."""
    _, _, _, lse, loss = _head_stats(x, W, labels, vocab_start, ignore_index, True)
    return loss, lse


def head_xent_grad(x: torch.Tensor, W: torch.Tensor, labels: torch.Tensor, lse: torch.Tensor, gscale: torch.Tensor,
                   vocab_start: int = 0, ignore_index: int = -100) -> torch.Tensor:
    """d loss / d logits (bf16 [M, V_local]) from recomputed logits: (softmax - onehot) * gscale[row], written by the
    epilogue of the head GEMM; ``lse`` is the log-sum-exp over the whole vocabulary. Rows with an ignored label give 0."""
    M, N = x.shape[0], W.shape[0]
    out = torch.empty(M, N, dtype=torch.bfloat16, device=x.device)
    labels = labels.reshape(-1).to(torch.int64).contiguous()
    lse = lse.float().contiguous()
    gscale = gscale.float().contiguous()
    xa = _lib.XentArgs(mode=2, labels=labels.data_ptr(), vocab_start=int(vocab_start), ignore_index=int(ignore_index),
                       stats=0, target=0, lse=lse.data_ptr(), gscale=gscale.data_ptr())
    _lib.check(_lib.lib().gv_gemm_xent(_head_args(x, W, out), xa, _lib.stream_ptr()), "gv_gemm_xent(grad)")
    return out


def _lib_fallback_allowed() -> bool:
    # Odd shapes (leading dimensions, or K of a K-major operand, not multiples of 8) only occur in tiny unit-test models;
    # they take the PyTorch path instead of failing.
    return True
