"""Layer-level log-linear Gated DeltaNet API with the signature of the reference's
`chunk_h_gated_delta_rule` (hattention/gated_delta_rule_apis.py:21-34)."""
import warnings
from typing import Optional

import torch

from . import _lib
from .base import HStruct, HType
from .kernel import gdn_native, hattention_kernel, hattention_step, prefill

SCALE_LAMBDA = True


def _decode(q, k, v, g, l, beta, scale, s):
    """One token through the native call, or None for what it does not take."""
    if q.dtype != torch.bfloat16 or s.base != 2 or s.htype != HType.WEAK or s.hstruct != HStruct.GDELTA:
        return None
    T, heads, K = q.shape[1:] if q.dim() == 4 else (0, 0, 0)
    if T != 1:
        return None
    if T < heads:
        warnings.warn(f"seq_len ({T}) < num_heads ({heads}): inputs may be in head-first format", stacklevel=2)
    if scale is None:
        scale = K ** -0.5
    return _lib.host().gdn_step(s.states, s.counts, q, k, v, beta, g, l, scale, 1.0 / scale if SCALE_LAMBDA else 0.0)


@torch.compiler.disable
def chunk_h_gated_delta_rule(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    g: torch.Tensor,
    l: torch.Tensor,
    beta: torch.Tensor,
    scale: float = None,
    initial_state=None,
    output_final_state: bool = False,
    cu_seqlens: Optional[torch.LongTensor] = None,
    head_first: bool = False,
    use_qk_l2norm_in_kernel: bool = False,
):
    """q,k (B,T,H,K), v (B,T,H,V), g (B,T,H) log decay, l (B,T,H,L), beta (B,T,H) -> (o, final_state).
    Same checks and dispatch as the reference (gated_delta_rule_apis.py:35-132): bf16 only, no varlen, l2norm
    in the kernel is mandatory, scale defaults to K^-1/2 and lambda is divided by it; training call without
    states, prompt call with `output_final_state=True` (-> `hattention_prefill`), and one-token call with an
    `initial_state` (-> `hattention_step`)."""
    if initial_state is not None and output_final_state is not False and cu_seqlens is None and use_qk_l2norm_in_kernel is True \
            and not head_first:
        # a decode step: the native call takes only bf16 operands of a one-token call, which makes the checks below (1.4 of 14.7 us
        # of a step at small batches) its own; it declines before anything is written
        o = _decode(q, k, v, g, l, beta, scale, initial_state)
        if o is not None:
            return o, initial_state
    assert q.dtype == k.dtype == v.dtype
    assert q.dtype != torch.float32, "ChunkGatedDeltaRuleFunction does not support float32. Please use bfloat16."
    assert len(beta.shape) == 3, "beta must be of shape [B, T, H] if head_first=False, or [B, H, T] otherwise."
    assert cu_seqlens is None
    assert use_qk_l2norm_in_kernel is True
    if head_first:
        raise DeprecationWarning("head_first is deprecated; use head_first=False")
    if q.shape[1] < q.shape[2]:
        warnings.warn(f"seq_len ({q.shape[1]}) < num_heads ({q.shape[2]}): inputs may be in head-first format")
    if scale is None:
        scale = k.shape[-1] ** -0.5
    if output_final_state is not False:
        lambda_mul = 1.0 / scale if SCALE_LAMBDA else 0.0
        if initial_state is None:
            if l.dtype != torch.bfloat16 and SCALE_LAMBDA:
                l, lambda_mul = l / scale, 0.0
            return prefill(q=q, k=k, v=v, b=beta, g=g, l=l, scale=scale, head_first=False, level_base=2, htype=HType.WEAK,
                           hstruct=HStruct.GDELTA, use_qk_l2norm_in_kernel=True, lambda_mul=lambda_mul)
        if not (q.ndim == 4 and k.ndim == 4 and v.ndim == 4 and beta.ndim == 3 and g.ndim == 3 and l.ndim == 4
                and q.shape[1] == k.shape[1] == v.shape[1] == beta.shape[1] == g.shape[1] == l.shape[1] == 1):
            raise ValueError
        s = initial_state
        q, k, v, beta, g, l = (x.squeeze(1) for x in (q, k, v, beta, g, l))
        if SCALE_LAMBDA:
            l = l / scale
        o, final_state = hattention_step(hstate=s, q=q, k=k, v=v, b=beta, g=g, l=l, scale=scale, level_base=2, htype=HType.WEAK,
                                         hstruct=HStruct.GDELTA, use_qk_l2norm_in_kernel=True)
        return o.unsqueeze(1), final_state
    if initial_state is not None:
        raise NotImplementedError
    o = gdn_native(q, k, v, beta, g, l, scale, 1.0 / scale if SCALE_LAMBDA else 0.0)
    if o is not None:
        return o, None
    if SCALE_LAMBDA:
        l = l / scale
    o = hattention_kernel(q=q, k=k, v=v, b=beta, g=g, l=l, scale=scale, head_first=False, level_base=2, htype=HType.WEAK,
                          hstruct=HStruct.GDELTA, use_qk_l2norm_in_kernel=True)
    return o, None
