"""What a prompt keeps in fp32: the tokens behind its last whole chunk and the level states that they build have the precision of decode steps,
and the layer's prompt has the rounding points of the torch operators around the scan."""
import pytest
import torch

from oracle import loglinear_oracle as orc

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


# tails of one token, of 63, across the rows of a warp; no whole chunk, one, an odd number, whole segments, several sequences
@pytest.mark.parametrize("B,T,H,N,G", [(1, 1, 2, 128, 1), (2, 63, 2, 64, 1), (1, 65, 2, 128, 2), (3, 80, 2, 128, 1), (2, 209, 4, 64, 2),
                                       (1, 513, 2, 128, 1), (2, 1025, 2, 64, 1), (1, 1600, 2, 128, 1), (1, 2079, 2, 128, 1)])
def test_mamba2_tail_keeps_fp32(B, T, H, N, G):
    from hattention_b200.base import HStruct, HType
    from hattention_b200.kernel import hattention_prefill
    L, T0 = 15, T // 64 * 64
    q, k, v, g, l = orc.make_mamba2_inputs(B, T, H, 64, N, G, L, seed=T)
    q, k, v, l = (x.bfloat16().float() for x in (q, k, v, l))
    want, st = orc.recurrent(q.double(), k.double(), v.double(), g.double(), l.double())
    d = lambda x: x.bfloat16().to(DEV)
    o, hs = hattention_prefill(d(q), d(k), d(v), None, g.float().to(DEV), d(l), None, False, 2, HType.WEAK, HStruct.MAMBA2)
    assert hs.counts == list(st.counts)
    states = torch.stack(st.states, dim=-1)
    if T0 < T:
        # outputs: one rounding to bf16, about 2^-9 / sqrt(3) in the norm (more for few values); the levels before these tokens come from bf16 operands
        assert rel(o[:, T0:], want[:, T0:]) < 2.5e-3
        # levels built by these tokens: fp32 sums of at most 32 exact products times a decay (with bf16 operands 1e-3)
        assert rel(hs.states[..., :7], states[..., :7]) < 1e-6
    if T0:
        assert rel(hs.states[..., 7:], states[..., 7:]) < 4e-3          # bf16 operands of the whole chunks


def test_mamba2_tail_after_a_decay_to_nothing():
    """A log decay of -inf among the tokens behind the last whole chunk empties every level and leaves no NaN."""
    from hattention_b200.base import HStruct, HType
    from hattention_b200.kernel import hattention_prefill
    T, cut = 70, 67
    q, k, v, g, l = orc.make_mamba2_inputs(1, T, 2, 64, 128, 1, 9, seed=0)
    d = lambda x: x.bfloat16().to(DEV)
    g = g.float().to(DEV)
    g[:, cut] = float("-inf")
    o, hs = hattention_prefill(d(q), d(k), d(v), None, g, d(l), None, False, 2, HType.WEAK, HStruct.MAMBA2)
    assert torch.isfinite(o).all() and torch.isfinite(hs.states).all()
    assert (hs.states[..., 7:] == 0).all()


@pytest.mark.parametrize("mode", ["positive", "bounded", None])
@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T", [(1, 200), (2, 130), (1, 40), (2, 128)])
def test_layer_prompt_rounds_like_the_torch_operators(B, T, mode, params):
    from hattention_b200 import mamba_apis
    from hattention_b200.base import HStruct, HType
    torch.manual_seed(T)
    H, G, N, L = 4, 2, 128, 12
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    x, dt, Bm, Cm, dl = bf(B, T, H, 64), bf(B, T, H), bf(B, T, G, N) / 11, bf(B, T, G, N) / 11, bf(B, T, H, L)
    A, Lp, D, bias = -torch.rand(H, device=DEV), bf(H, L).to(params), bf(H).to(params), bf(H).to(params)
    kw = dict(D=D, dt_bias=bias, dt_softplus=True, return_final_states=True, lambda_mode=mode, lambda_level_max=L, lambda_level_base=2,
              lambda_htype=HType.WEAK, lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)
    y, s = mamba_apis.hmamba_chunk_scan_combined(x, dt, A, Bm, Cm, dl, Lp, 64, **kw)
    old = mamba_apis.FUSED_PREP
    mamba_apis.FUSED_PREP = False
    try:
        yt, st = mamba_apis.hmamba_chunk_scan_combined(x, dt, A, Bm, Cm, dl, Lp, 64, **kw)
    finally:
        mamba_apis.FUSED_PREP = old
    assert y.dtype == yt.dtype == params
    # the same operands but for the last bit of the exponentials' fp32 values: a value in a few hundred falls on the other side of a rounding
    assert rel(y, yt) < 5e-4
    assert rel(s.states, st.states) < 5e-4


# tails of one token, of 63; no whole chunk, one, an odd number, a power of two; narrow keys, parts of wide values, several sequences
@pytest.mark.parametrize("B,T,H,Dk,Dv", [(1, 1, 2, 128, 128), (2, 63, 2, 64, 64), (1, 65, 2, 128, 128), (3, 90, 2, 128, 64), (1, 255, 2, 128, 192),
                                         (1, 330, 2, 96, 256), (2, 521, 2, 128, 128), (1, 800, 2, 128, 64), (1, 1050, 1, 128, 384)])
def test_gdn_tail_keeps_fp32(B, T, H, Dk, Dv):
    from hattention_b200.gated_delta_rule_apis import chunk_h_gated_delta_rule
    L, T0 = 13, T // 64 * 64
    q, k, v, b, g, l = orc.make_gdn_inputs(B, T, H, Dk, Dv, L, seed=T)
    q, k, v, b, l = (x.bfloat16().float() for x in (q, k, v, b, l))
    scale = Dk ** -0.5
    d = lambda x: x.bfloat16().to(DEV)
    o, hs = chunk_h_gated_delta_rule(d(q), d(k), d(v), g.float().to(DEV), d(l), d(b), output_final_state=True, use_qk_l2norm_in_kernel=True)
    # the recurrence on the rounded operands that a step takes
    from hattention_b200.chunkwise_hgdn import l2norm_fwd
    qn, kn = l2norm_fwd(d(q), scale).double().cpu(), l2norm_fwd(d(k)).double().cpu()
    want, st = orc.recurrent(qn, kn, v.double(), g.double(), (d(l) / scale).double().cpu(), b=b.double())
    assert o.is_contiguous() and hs.counts == list(st.counts)
    states = torch.stack(st.states, dim=-1)
    if T0 < T:
        # one rounding to bf16 (the chunkwise kernels are at 3.4e-3 here), and the levels below a chunk in fp32
        assert rel(o[:, T0:], want[:, T0:]) < 2.5e-3
        assert rel(hs.states[..., :7], states[..., :7]) < 2e-6
        if T0:
            # the lowest level above them holds the last whole chunk, in fp32; what the others have from the scan is decayed by then
            N = T0 // 64
            low = 7 + (N & -N).bit_length() - 1
            if N % 2:
                assert rel(hs.states[..., low], states[..., low]) < 2e-6
            assert rel(hs.states[..., 7:], states[..., 7:]) < 2e-3


def test_gdn_tail_after_a_decay_to_nothing():
    """A log decay of -inf among the tokens behind the last whole chunk empties every level and leaves no NaN."""
    from hattention_b200.gated_delta_rule_apis import chunk_h_gated_delta_rule
    q, k, v, b, g, l = orc.make_gdn_inputs(1, 70, 2, 128, 64, 9, seed=0)
    d = lambda x: x.bfloat16().to(DEV)
    g = g.float().to(DEV)
    g[:, 67] = float("-inf")
    o, hs = chunk_h_gated_delta_rule(d(q), d(k), d(v), g, d(l), d(b), output_final_state=True, use_qk_l2norm_in_kernel=True)
    assert torch.isfinite(o).all() and torch.isfinite(hs.states).all()
    assert (hs.states[..., 7:] == 0).all()
