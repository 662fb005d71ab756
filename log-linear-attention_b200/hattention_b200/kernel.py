"""Autograd boundary of log-linear attention, with the interface of the reference's
`hattention/kernel.py` (`HAttentionFunction` :32-244, `hattention_kernel` :338-374)."""
from typing import Optional, Tuple

import torch

from .base import HStruct, HType
from . import _lib
from .chunkwise import chunkwise_bwd, chunkwise_fwd
from .recurrent import HState, is_level_major  # noqa: F401  (HState: the reference imports it from both modules)


# Keep the forward call's scratch alive until the backward, which then skips its recomputation: the
# Mamba-2 segment-level states (about 0.2 GB at B=2, T=16384, H=32), and for Gated DeltaNet the chunk
# matrices and every chunk's level states (2.4 GB at B=4, T=8192, H=16, 128 x 128 heads; not kept above
# chunkwise_hgdn.KEEP_WORKSPACE_MAX_BYTES).  The reference keeps only the inputs (kernel.py:125); set to
# False for that memory behaviour.
KEEP_FORWARD_STATES = True


class HAttentionFunction(torch.autograd.Function):
    """Same argument list, validation and saved tensors as the reference's function
    (kernel.py:37-136); the chunkwise=False ("parallel") form is not provided."""

    @staticmethod
    def forward(ctx, q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct, chunk_sizes, chunkwise,
                use_qk_l2norm_in_kernel):
        q, k, v, g, l = (x.contiguous() for x in (q, k, v, g, l))
        if hstruct == HStruct.MAMBA2 and chunkwise:
            if b is not None:
                raise ValueError
            if chunk_sizes[0] != chunk_sizes[1]:
                raise NotImplementedError
            if use_qk_l2norm_in_kernel:
                raise NotImplementedError
            if scale is not None:
                raise NotImplementedError
            kept = [] if KEEP_FORWARD_STATES else None
            o, g_cum, _ = chunkwise_fwd(q=q, k=k, v=v, g=g, l=l, head_first=head_first, level_base=level_base,
                                        htype=htype, chunk_size=chunk_sizes[0], output_final_state=False,
                                        keep_workspace=kept)
            ctx.fwd_workspace = kept[0] if kept else None
            Aw = Au = None
        elif hstruct == HStruct.GDELTA and chunkwise:
            from .chunkwise_hgdn import gdn_forward
            if b is None:
                raise ValueError
            if chunk_sizes[0] != chunk_sizes[1]:
                raise NotImplementedError
            if not use_qk_l2norm_in_kernel:
                raise NotImplementedError
            if scale is None:
                raise NotImplementedError
            kept = [] if KEEP_FORWARD_STATES and any(ctx.needs_input_grad[:6]) else None
            g_cum, o, Aw, Au = gdn_forward(q, k, v, b.contiguous(), g, l, scale, head_first, level_base, htype,
                                           chunk_sizes[0], keep=kept)
            ctx.fwd_workspace = kept if kept else None
        else:
            raise NotImplementedError
        ctx.save_for_backward(q, k, v, b, g_cum, l, Aw, Au)
        ctx.scale = scale
        ctx.dtype = g.dtype
        ctx.head_first = head_first
        ctx.level_base = level_base
        ctx.htype = htype
        ctx.hstruct = hstruct
        ctx.chunk_sizes = chunk_sizes
        return o.to(q.dtype)

    @staticmethod
    def backward(ctx, do):
        q, k, v, b, g_cum, l, Aw, Au = ctx.saved_tensors
        do = do.contiguous()
        if ctx.hstruct == HStruct.MAMBA2:
            dq, dk, dv, dg, dl = chunkwise_bwd(q=q, k=k, v=v, g=g_cum, l=l, do=do, head_first=ctx.head_first,
                                               level_base=ctx.level_base, htype=ctx.htype,
                                               chunk_size=ctx.chunk_sizes[0], fwd_workspace=ctx.fwd_workspace)
            ctx.fwd_workspace = None
            db = None
        else:
            from .chunkwise_hgdn import gdn_backward
            dq, dk, dv, db, dg, dl = gdn_backward(q, k, v, b, g_cum, l, Aw, Au, do, ctx.scale, ctx.head_first,
                                                  ctx.level_base, ctx.htype, ctx.chunk_sizes[0],
                                                  kept=ctx.fwd_workspace)
            ctx.fwd_workspace = None
        return (dq.to(q), dk.to(k), dv.to(v), db.to(b) if b is not None else None, dg.to(ctx.dtype), dl.to(l),
                None, None, None, None, None, None, None, None)


def gdn_native(q, k, v, b, g, l, scale: float, lambda_mul: float):
    """The native Gated DeltaNet node (lambda times lambda_mul unless that is 0), or None for operands that it does not take."""
    from .chunkwise_hgdn import KEEP_WORKSPACE_MAX_BYTES
    return _lib.host().hattention_gdn(q, k, v, b, g, l, scale, lambda_mul, KEEP_WORKSPACE_MAX_BYTES if KEEP_FORWARD_STATES else -1,
                                      _lib.CHECK_STATUS)


def hattention_kernel(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    b: Optional[torch.Tensor],
    g: torch.Tensor,
    l: torch.Tensor,
    scale: Optional[float],
    head_first: bool,
    level_base: int,
    htype: HType,
    hstruct: HStruct,
    chunk_sizes: Optional[Tuple[int, int]] = None,
    chunkwise: bool = True,
    use_qk_l2norm_in_kernel: bool = False,
) -> torch.Tensor:
    """o = log-linear attention(q, k, v, g, l[, b]) with gradients; see kernel.py:338-374."""
    return kernel_call(q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct, chunk_sizes, chunkwise, use_qk_l2norm_in_kernel)


def kernel_call(q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct, chunk_sizes=None, chunkwise=True,
                use_qk_l2norm_in_kernel=False, in_layer=False):
    """hattention_kernel; `in_layer`: the gradients go on into the sums over tokens of a Mamba-2 layer (llattn_mamba2_bwd_layer)."""
    if chunk_sizes is None:
        chunk_sizes = (64, 64)
    if chunkwise and not head_first and level_base == 2 and htype == HType.WEAK and tuple(chunk_sizes) == (64, 64):
        # bf16 operands of the supported shapes: the native nodes; everything else, errors included, below
        o = None
        if hstruct == HStruct.MAMBA2 and b is None and scale is None and not use_qk_l2norm_in_kernel:
            o = _lib.host().hattention_mamba2(q, k, v, g, l, KEEP_FORWARD_STATES, _lib.CHECK_STATUS, in_layer)
        elif hstruct == HStruct.GDELTA and b is not None and scale is not None and use_qk_l2norm_in_kernel:
            o = gdn_native(q, k, v, b, g, l, scale, 0.0)
        if o is not None:
            return o
    return HAttentionFunction.apply(q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct, chunk_sizes,
                                    chunkwise, use_qk_l2norm_in_kernel)


@torch.no_grad()
def hattention_step(hstate: HState, q, k, v, b, g, l, scale, level_base, htype, hstruct,
                    use_qk_l2norm_in_kernel: bool = False):
    """One decoding step, signature of the reference's `hattention_step` (kernel.py:563-633):
    q, k (B,G,K), v (B,H,V), g (B,H), l (B,H,L)[, b (B,H)] -> (o (B,H,V), hstate).  One CUDA kernel per step for
    either structure, the l2norm of the delta-rule structure included, which moves only the levels that hold tokens
    (`llattn_mamba2_layer_step`, `llattn_gdn_layer_step`); states that a caller has stored with the level innermost go
    through `llattn_mamba2_step` / `llattn_gdn_step`."""
    if not (q.ndim == 3 and k.ndim == 3 and v.ndim == 3 and g.ndim == 2 and l.ndim == 3
            and (b is None or b.ndim == 2) and g.dtype == hstate.dtype and q.dtype == k.dtype == v.dtype == l.dtype
            and hstate.base == level_base and hstate.htype == htype and hstate.hstruct == hstruct):
        raise TypeError
    if hstate.dtype != torch.float32:
        raise NotImplementedError("level states are kept in fp32")
    B, G, K = k.shape
    _, H, V = v.shape
    L = l.shape[-1]
    if hstruct == HStruct.MAMBA2:
        if b is not None:
            raise ValueError
        if use_qk_l2norm_in_kernel or scale is not None:
            raise NotImplementedError
    else:
        if b is None:
            raise ValueError
        if use_qk_l2norm_in_kernel:
            if scale is None:
                raise NotImplementedError
        elif scale is not None:
            raise NotImplementedError
    if not v.is_cuda:
        raise RuntimeError("the decode kernels need CUDA tensors (there is no CPU path)")
    if is_level_major(hstate.states):
        q_, k_, v_, l_ = (_lib.aligned(x.to(torch.bfloat16)) for x in (q, k, v, l))
        g_ = g.contiguous()
        if hstruct == HStruct.MAMBA2:
            o = mamba2_layer_step(hstate, q_, k_, v_, g_, l_)
        else:
            o = gdn_layer_step(hstate, q_, k_, v_, b.to(torch.bfloat16).contiguous(), g_, l_, scale if use_qk_l2norm_in_kernel else None)
        return o.to(v.dtype), hstate
    lib = _lib.lib()
    if not hstate.states.is_contiguous():
        hstate.states = hstate.states.contiguous()           # these kernels take the level innermost
    if hstruct == HStruct.GDELTA:
        if use_qk_l2norm_in_kernel:
            from .chunkwise_hgdn import l2norm_fwd
            q, k = l2norm_fwd(q, scale), l2norm_fwd(k)
        if G != H:
            q, k = q.repeat_interleave(H // G, dim=1), k.repeat_interleave(H // G, dim=1)
    carry = hstate.cascade_counts()
    hstate.counts[0] += 1
    with torch.cuda.device(v.device):
        q_, k_, v_, l_ = (x.to(torch.bfloat16).contiguous() for x in (q, k, v, l))
        g_ = g.to(torch.float32).contiguous()
        o = torch.empty(B, H, V, dtype=torch.bfloat16, device=v.device)
        stream = torch.cuda.current_stream().cuda_stream
        if hstruct == HStruct.MAMBA2:
            rc = lib.llattn_mamba2_step(hstate.states.data_ptr(), q_.data_ptr(), k_.data_ptr(), v_.data_ptr(), g_.data_ptr(),
                                        l_.data_ptr(), o.data_ptr(), B, H, G, K, V, L, carry, stream)
            _lib.check(rc, "llattn_mamba2_step")
        else:
            b_ = b.to(torch.bfloat16).contiguous()
            rc = lib.llattn_gdn_step(hstate.states.data_ptr(), q_.data_ptr(), k_.data_ptr(), v_.data_ptr(), b_.data_ptr(),
                                     g_.data_ptr(), l_.data_ptr(), o.data_ptr(), B, H, K, V, L, carry, stream)
            _lib.check(rc, "llattn_gdn_step")
    return o.to(v.dtype), hstate


def _step_levels(hstate: HState):
    """Runs the cascade on the counts and counts the new token: the levels that held tokens, as bits, and the one that receives the merged ones."""
    live = hstate.live_levels()
    carry = hstate.cascade_counts()
    hstate.counts[0] += 1
    return live, carry


def mamba2_layer_step(hstate: HState, q, k, v, g, l) -> torch.Tensor:
    """One launch of `llattn_mamba2_layer_step` on a level-major state, with v, the log decay and lambda given: contiguous bf16 q, k, v, l; fp32 g."""
    B, G, K = k.shape
    _, H, V = v.shape
    dev = v.device.index
    o = torch.empty(B, H, V, dtype=torch.bfloat16, device=v.device)
    live, carry = _step_levels(hstate)
    rc = _lib.lib().llattn_mamba2_layer_step(
        hstate.states.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), None, g.data_ptr(), l.data_ptr(), None, 0, None, 0, None, 0, None,
        o.data_ptr(), B, H, G, K, V, l.shape[-1], live, carry, 2, 0, dev, torch._C._cuda_getCurrentRawStream(dev))
    if rc != 0:
        _lib.check(rc, "llattn_mamba2_layer_step")
    return o


def gdn_layer_step(hstate: HState, q, k, v, b, g, l, scale: Optional[float] = None) -> torch.Tensor:
    """One launch of `llattn_gdn_layer_step` on a level-major state: contiguous bf16 q, k, v, b, l; fp32 g.  With a scale q and k
    are normalised (and q scaled) first."""
    B, G, K = k.shape
    _, H, V = v.shape
    dev = v.device.index
    o = torch.empty(B, H, V, dtype=torch.bfloat16, device=v.device)
    live, carry = _step_levels(hstate)
    rc = _lib.lib().llattn_gdn_layer_step(
        hstate.states.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), b.data_ptr(), g.data_ptr(), l.data_ptr(), o.data_ptr(),
        B, H, G, K, V, l.shape[-1], live, carry, scale is not None, scale or 1.0, 0.0, dev, torch._C._cuda_getCurrentRawStream(dev))
    if rc != 0:
        _lib.check(rc, "llattn_gdn_layer_step")
    return o


def hattention_prefill(q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct,
                       chunk_size: Optional[int] = None, use_qk_l2norm_in_kernel: bool = False):
    """Outputs for a prompt and the level states to continue from, signature of the reference's
    `hattention_prefill` (kernel.py:469-560).  The whole chunks of the prompt go through the chunkwise kernels; the
    tokens behind them keep the fp32 states and products of decode steps, in kernels that take all of them at once.
    Shapes that those kernels do not take and that are shorter than a chunk are stepped token by token."""
    return prefill(q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct, chunk_size, use_qk_l2norm_in_kernel)


@torch.no_grad()
def prefill(q, k, v, b, g, l, scale, head_first, level_base, htype, hstruct, chunk_size: Optional[int] = None,
            use_qk_l2norm_in_kernel: bool = False, lambda_mul: float = 0.0):
    """`hattention_prefill`; lambda_mul != 0 (delta-rule structure): lambda is multiplied by it on the way to the kernels."""
    if chunk_size is None:
        chunk_size = 64
    if head_first:
        raise NotImplementedError
    B, T, G, K = k.shape
    _, _, H, V = v.shape
    L = l.shape[-1]
    if hstruct == HStruct.MAMBA2:
        if b is not None:
            raise ValueError
        if use_qk_l2norm_in_kernel or scale is not None:
            raise NotImplementedError
        chunkwise = T >= chunk_size or (chunk_size == 64 and K in (64, 128) and V == 64)
    else:
        if b is None:
            raise ValueError
        if not use_qk_l2norm_in_kernel or scale is None:
            raise NotImplementedError
        chunkwise = T >= chunk_size or (chunk_size == 64 and K <= 128 and V % 64 == 0 and V <= 384)
    ragged = T % chunk_size != 0
    if (ragged or hstruct == HStruct.GDELTA) and not (q.dtype == k.dtype == v.dtype == l.dtype):
        raise TypeError
    if chunkwise:
        if hstruct == HStruct.MAMBA2:
            from .chunkwise import prompt_forward
            o, states = prompt_forward(q, k, v, g, l, level_base, htype, chunk_size)
        else:
            from .chunkwise_hgdn import prompt_forward
            o, states = prompt_forward(q, k, v, b, g, l, scale, head_first, level_base, htype, chunk_size, lambda_mul)
        hstate = HState.holding(states, level_base, htype, hstruct)
        hstate.set_counts_after(T)
        return o.to(v.dtype), hstate
    if lambda_mul != 0.0:
        l = l * lambda_mul
    o = torch.zeros_like(v)
    hstate = HState(base=level_base, htype=htype, hstruct=hstruct, shape=(B, H, K, V, L), dtype=torch.float32, device=g.device)
    for t in range(T):
        o[:, t], hstate = hattention_step(hstate, q[:, t], k[:, t], v[:, t], b[:, t] if b is not None else None, g[:, t].float(),
                                          l[:, t], scale, level_base, htype, hstruct, use_qk_l2norm_in_kernel)
    return o, hstate
