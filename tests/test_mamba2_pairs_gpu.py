"""The CTAs of the output and gradient kernels take a pair of chunks and up to eight heads of a q / k group.  Small calls have a head a CTA: pairs that read no, one and
several levels, ends of sequences, the most lambda levels.  Calls that fill the chip walk several heads in a CTA, whose rings, sums and places in shared memory are
written again from the second or third head on: group sizes that leave a part of a CTA's heads over, two groups, narrow states, a last half pair, and what only a layer asks of it."""
import pytest
import torch

from oracle import loglinear_oracle as orc
from test_mamba2_gpu import assert_close, rounded_inputs, run_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,N,G,L", [
    (1, 640, 9, 128, 1, 11),       # two segments, the last of one pair
    (2, 1024, 6, 64, 6, 12),       # one head a group
    (1, 1088, 13, 64, 1, 12),      # an odd number of chunks
    (2, 704, 10, 128, 2, 20),      # the most lambda levels, two groups, a last half pair
    (1, 128, 5, 128, 1, 8),        # a single pair: no states at all
    (1, 4096, 3, 128, 1, 13),      # eight segments: pairs that read up to five levels
])
def test_heads_and_levels_of_a_cta_match_oracle(B, T, H, N, G, L):
    q, k, v, g, l, do = rounded_inputs(B, T, H, 64, N, G, L, seed=T + 7 * H)
    o, _ = run_cuda(q, k, v, g, l, do)
    assert_close(o, orc.mamba2_chunkwise(q, k, v, g, l), "o")


@pytest.mark.parametrize("B,T,H,N,G,L", [
    (1, 128, 5, 128, 1, 8),        # a single pair: neither states nor readers
    (2, 256, 3, 64, 1, 9),         # two pairs of one segment, N = 64
    (1, 512, 9, 128, 1, 20),       # four pairs of one segment, spare lambda levels
    (1, 640, 9, 128, 1, 11),       # two segments, the last of one pair
    (2, 1024, 6, 64, 6, 12),       # one head a group
    (2, 704, 10, 128, 2, 20),      # a last half pair, the most lambda levels
    (1, 384, 3, 128, 1, 10),       # three pairs, the last of which nobody reads
    (2, 896, 32, 128, 1, 11),      # the same in a second segment, enough of them for either order of completion (four heads a CTA)
    (1, 1344, 4, 64, 2, 12),       # ... and the last pair a half
    (1, 8832, 1, 128, 1, 15),      # eighteen segments: readers of a fifth high level, for which a second CTA is there
])
def test_gradients_of_a_cta_match_oracle(B, T, H, N, G, L):
    q, k, v, g, l, do = rounded_inputs(B, T, H, 64, N, G, L, seed=T + 5 * H)
    _, grads = run_cuda(q, k, v, g, l, do)
    _, want = orc.mamba2_grads(q, k, v, g, l, do, fn=orc.mamba2_chunkwise_blocked if T > 4096 else orc.mamba2_chunkwise)
    for got, ref, key in zip(grads, want, ("dq", "dk", "dv", "dg", "dl")):
        assert_close(got, ref, key)


def heads_per_cta(B, T, H, N, G, L):
    from hattention_b200 import _lib
    return _lib.lib().llattn_testing_mamba2_heads_per_cta(B, T, H, G, N, 64, L)


@pytest.mark.parametrize("B,T,H,N,G,L,heads", [
    (2, 2112, 13, 128, 1, 20, 4),      # 4 + 4 + 4 + 1 heads, a last half pair, spare lambda levels
    (4, 1984, 10, 64, 2, 12, 5),       # whole groups of five, N = 64, an odd number of chunks
    (2, 4096, 9, 128, 1, 13, 5),       # 5 + 4 heads, pairs that read up to five levels
    (8, 640, 17, 64, 1, 11, 6),        # 6 + 6 + 5 heads, N = 64
    (8, 384, 26, 128, 2, 10, 5),       # 5 + 5 + 3 heads a group, one segment
    (16, 128, 48, 128, 1, 20, 6),      # a single pair, as many heads as L = 20 allows
])
def test_heads_that_follow_in_a_cta_match_oracle(B, T, H, N, G, L, heads):
    assert heads_per_cta(B, T, H, N, G, L) == heads
    q, k, v, g, l, do = rounded_inputs(B, T, H, 64, N, G, L, seed=T + 3 * H)
    o, grads = run_cuda(q, k, v, g, l, do)
    want_o, want = orc.mamba2_grads(q, k, v, g, l, do, fn=orc.mamba2_chunkwise)
    for got, ref, key in zip((o, *grads), (want_o, *want), ("o", "dq", "dk", "dv", "dg", "dl")):
        assert_close(got, ref, key)


@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,heads", [(576, 9, 1), (1024, 2, 1), (2112, 18, 5)])      # (five heads: either team of warps takes a second and one a third)
def test_residual_of_a_layer(T, H, heads, params):
    """y = bf16(o) + D x, in the parameters' dtype, leaves by way of the tile of x: every row of it, and nothing behind the sequence's end."""
    from hattention_b200.base import HStruct, HType
    from hattention_b200.mamba_apis import hmamba_chunk_scan_combined
    dev, L = torch.device("cuda:0"), 12 if T <= 2048 else 13
    assert heads_per_cta(2, T, H, 128, 1, L) == heads
    gen = torch.Generator().manual_seed(T + H)
    r = lambda *s: torch.randn(*s, generator=gen)
    x, Bm, Cm, dl = (t.bfloat16().to(dev) for t in (r(2, T, H, 64), r(2, T, 1, 128) / 128 ** 0.5, r(2, T, 1, 128) / 128 ** 0.5, r(2, T, H, L)))
    dt, A, Lp, D = (r(2, T, H) - 2).bfloat16().to(dev), -torch.exp(r(H)).to(dev), torch.ones(H, L).to(dev, params), r(H).to(dev, params)
    kw = dict(dt_softplus=True, lambda_mode="positive", lambda_level_max=L, lambda_level_base=2, lambda_htype=HType.WEAK, lambda_hstruct=HStruct.MAMBA2,
              lambda_level_fixed=True)
    with torch.no_grad():
        y, _ = hmamba_chunk_scan_combined(x, dt, A, Bm, Cm, dl, Lp, 64, D=D, **kw)
        o, _ = hmamba_chunk_scan_combined(x, dt, A, Bm, Cm, dl, Lp, 64, D=None, **kw)
    want = o.float() + D.float()[:, None] * x.float()
    # the sum and the product are rounded to fp32 (2^-24 of each, on either side), bf16 results once more
    bound = 2.0 ** -22 * (o.float().abs() + (D.float()[:, None] * x.float()).abs()) + (2.0 ** -8 * want.abs() if params == torch.bfloat16 else 0.)
    assert y.dtype == params and ((y.float() - want).abs() <= bound).all()


@pytest.mark.parametrize("B,T,H,N,G,L,heads", [
    (1, 640, 6, 128, 6, 11, 1),        # one head a group
    (2, 2112, 4, 64, 4, 13, 1),        # N = 64, a last half pair
    (1, 64, 3, 128, 3, 8, 1),          # a single chunk
    (4, 1984, 10, 64, 2, 12, 5),       # five heads a group, all in one CTA
    (8, 1088, 12, 128, 4, 12, 3),
])
def test_gradients_of_whole_groups_leave_as_they_are(B, T, H, N, G, L, heads):
    """Where a CTA has all heads of a group dq and dk need no accumulators: the digits are those of the accumulators, which serve results that start off a 16-byte boundary."""
    from hattention_b200 import _lib
    lib, dev = _lib.lib(), torch.device("cuda:0")
    assert heads_per_cta(B, T, H, N, G, L) == heads == H // G
    ins = rounded_inputs(B, T, H, 64, N, G, L, seed=T + H)
    q, k, v, g, l, do = (x.to(dev) for x in ins)
    q, k, v, l, do = (x.bfloat16() for x in (q, k, v, l, do))
    g_cum = torch.cumsum(g.reshape(B, T // 64, 64, H), dim=2).reshape(B, T, H).contiguous()
    ws = torch.empty(lib.llattn_mamba2_bwd_workspace_bytes(B, T, H, G, N, 64, L), dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream().cuda_stream

    def run(offset):
        n = q.numel()
        dq, dk = (torch.full((n + 16,), float("nan"), device=dev).bfloat16() for _ in range(2))
        dv, dg, dl = torch.empty_like(v), torch.empty_like(g), torch.empty(l.shape, device=dev)
        rc = lib.llattn_mamba2_bwd(*(x.data_ptr() for x in (q, k, v, g_cum, l, do)), dq.data_ptr() + 2 * offset, dk.data_ptr() + 2 * offset,
                                   *(x.data_ptr() for x in (dv, dg, dl)), ws.data_ptr(), ws.numel(), B, T, H, G, N, 64, L, stream)
        _lib.check(rc, "llattn_mamba2_bwd")
        _lib.raise_on_status(ws, stream, "llattn_mamba2_bwd")
        for x in (dq, dk):
            assert torch.isnan(x[:offset]).all() and torch.isnan(x[offset + n:]).all()
        return [x[offset:offset + n].reshape(q.shape) for x in (dq, dk)] + [dv, dg, dl]

    whole, summed = run(0), run(4)
    _, want = orc.mamba2_grads(*ins, fn=orc.mamba2_chunkwise)
    for a, b, ref, key in zip(whole, summed, want, ("dq", "dk", "dv", "dg", "dl")):
        assert_close(a, ref, key)
        if key != "dg":                                    # (sums of atomic adds)
            assert torch.equal(a, b), key
