"""Prompts of any length and decode steps on level-major states: the padded chunkwise pass and the level-state kernels against
the fp64 token recurrence, and the level-major decode kernels against the level-innermost ones."""
import pytest
import torch

from oracle import loglinear_oracle as orc

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def assert_close(got, want, name, rtol=2e-2, atol=2e-3):
    got, want = got.detach().double().cpu(), want.detach().double().cpu()
    assert got.shape == want.shape
    tol = rtol * want.abs() + atol * max(1.0, want.abs().max().item())
    worst = ((got - want).abs() / tol).max().item()
    assert worst <= 1.0, f"{name}: worst err/tol = {worst:.3f}"


# one token, below / at / above a chunk, an even and an odd number of chunks, segment edges, levels that hold whole segments
@pytest.mark.parametrize("B,T,H,N,G,L", [(2, 1, 2, 128, 1, 4), (1, 40, 2, 64, 2, 7), (2, 65, 2, 128, 1, 9), (1, 192, 2, 128, 2, 12),
                                         (1, 513, 2, 64, 1, 11), (2, 1537, 2, 128, 1, 15), (1, 3333, 2, 128, 1, 15)])
def test_mamba2_prompt(B, T, H, N, G, L):
    from hattention_b200.base import HStruct, HType
    from hattention_b200.kernel import hattention_prefill
    q, k, v, g, l = orc.make_mamba2_inputs(B, T, H, 64, N, G, max(L, 7), seed=T)
    q, k, v, l = (x.bfloat16().float() for x in (q, k, v, l))
    l = l[..., :L]
    want, st = orc.recurrent(q.double(), k.double(), v.double(), g.double(), l.double())
    d = lambda x: x.bfloat16().to(DEV)
    o, hs = hattention_prefill(d(q), d(k), d(v), None, g.float().to(DEV), d(l), None, False, 2, HType.WEAK, HStruct.MAMBA2)
    assert o.is_contiguous() and hs.counts == list(st.counts)
    assert_close(o, want, "outputs")
    assert_close(hs.states, torch.stack(st.states, dim=-1), "level states")


@pytest.mark.parametrize("B,T,H,Dk,Dv,L", [(2, 1, 2, 128, 64, 3), (1, 63, 2, 128, 128, 7), (2, 65, 2, 64, 128, 8), (1, 130, 2, 128, 192, 9),
                                           (1, 700, 2, 128, 256, 11)])
def test_gdn_prompt(B, T, H, Dk, Dv, L):
    from hattention_b200.gated_delta_rule_apis import chunk_h_gated_delta_rule
    q, k, v, b, g, l = orc.make_gdn_inputs(B, T, H, Dk, Dv, L, seed=T)
    q, k, v, b, l = (x.bfloat16().float() for x in (q, k, v, b, l))
    scale = Dk ** -0.5
    qn, kn = orc.gdn_layer_inputs(q.double(), k.double(), scale)
    want, st = orc.recurrent(qn, kn, v.double(), g.double(), l.double() / scale, b=b.double())
    d = lambda x: x.bfloat16().to(DEV)
    o, hs = chunk_h_gated_delta_rule(d(q), d(k), d(v), g.float().to(DEV), d(l), d(b), output_final_state=True, use_qk_l2norm_in_kernel=True)
    assert o.is_contiguous() and hs.counts == list(st.counts)
    assert_close(o, want, "outputs", atol=4e-3)
    assert_close(hs.states, torch.stack(st.states, dim=-1), "level states", atol=4e-3)


def _pair_of_states(hstruct, B, H, K, V, L, position):
    """The same random states stored level-major and level-innermost."""
    from hattention_b200.base import HType
    from hattention_b200.recurrent import HState, is_level_major
    a = HState(2, HType.WEAK, hstruct, (B, H, K, V, L), torch.float32, DEV)
    a.set_counts_after(position)
    for level, count in enumerate(a.counts):
        if count:
            a.states[..., level] = torch.randn(B, H, K, V, device=DEV)
    b = HState.holding(a.states.contiguous(), 2, HType.WEAK, hstruct)
    b.counts = list(a.counts)
    assert is_level_major(a.states) and not is_level_major(b.states)
    return a, b


# few heads / many heads, one live level, all of them, levels that merge far up
@pytest.mark.parametrize("B,H,G,K,V,L,position", [(1, 2, 1, 128, 64, 15, 1), (1, 6, 2, 64, 64, 13, 4090), (5, 64, 1, 128, 64, 20, 21845),
                                                  (1, 2, 1, 96, 16, 9, 128), (2, 3, 3, 256, 128, 12, 1000), (20, 15, 1, 128, 16, 13, 2047)])
@pytest.mark.parametrize("struct", ["MAMBA2", "GDELTA"])
def test_level_major_steps(B, H, G, K, V, L, position, struct):
    from hattention_b200.base import HStruct, HType
    from hattention_b200.kernel import hattention_step
    hstruct = HStruct[struct]
    torch.manual_seed(position)
    a, b = _pair_of_states(hstruct, B, H, K, V, L, position)
    gdn = hstruct == HStruct.GDELTA
    for _ in range(4):
        bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()
        args = (bf(B, G, K), bf(B, G, K), bf(B, H, V), torch.rand(B, H, device=DEV).bfloat16() if gdn else None,
                -torch.rand(B, H, device=DEV), bf(B, H, L), K ** -0.5 if gdn else None, 2, HType.WEAK, hstruct, gdn)
        oa, _ = hattention_step(a, *args)
        ob, _ = hattention_step(b, *args)
        assert a.counts == b.counts
        assert_close(oa, ob, "output", rtol=1e-2, atol=1e-3)
        assert_close(a.states, b.states, "states", rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("mode", ["positive", "bounded", None])
@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
def test_layer_step_rounds_like_the_torch_operators(mode, params):
    """One launch against the sequence of torch operators around the kernel (which a level-innermost state takes)."""
    from hattention_b200.base import HStruct, HType
    from hattention_b200.mamba_apis import hselective_state_update
    torch.manual_seed(0)
    B, H, G, N, L = 2, 4, 2, 128, 12
    a, b = _pair_of_states(HStruct.MAMBA2, B, H, N, 64, L, 700)
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    x, dt, Bm, Cm, dl = bf(B, H, 64), bf(B, H), bf(B, G, N), bf(B, G, N), bf(B, H, L)
    A, Lp, D, bias = -torch.rand(H, device=DEV), bf(H, L).to(params), bf(H).to(params), bf(H).to(params)
    kw = dict(D=D, dt_bias=bias, dt_softplus=True, lambda_mode=mode, lambda_level_max=L, lambda_level_base=2, lambda_htype=HType.WEAK,
              lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)
    for _ in range(3):
        ya, _ = hselective_state_update(a, x, dt, A, Bm, Cm, dl, Lp, **kw)
        yb, _ = hselective_state_update(b, x, dt, A, Bm, Cm, dl, Lp, **kw)
        assert ya.dtype == yb.dtype == params
        assert_close(ya, yb, "output", rtol=1e-2, atol=1e-3)
        assert_close(a.states, b.states, "states", rtol=1e-5, atol=1e-6)
