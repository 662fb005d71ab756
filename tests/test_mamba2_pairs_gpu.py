"""The CTAs of the output and gradient kernels take a pair of chunks and up to eight heads of a q / k group: group sizes that leave a part of a CTA's heads over, one head a
group, the most lambda levels that it stages, pairs that read no, one and several levels, and what only a layer asks of it."""
import pytest
import torch

from oracle import loglinear_oracle as orc
from test_mamba2_gpu import assert_close, rounded_inputs, run_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,N,G,L", [
    (1, 640, 9, 128, 1, 11),       # nine heads a group: a CTA of its own for what is over, two segments, the last of one pair
    (2, 1024, 6, 64, 6, 12),       # one head a group
    (1, 1088, 13, 64, 1, 12),      # an odd number of chunks, thirteen heads
    (2, 704, 10, 128, 2, 20),      # the most lambda levels (six heads a CTA at most), a last half pair
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
    (1, 512, 9, 128, 1, 20),       # four pairs of one segment, a ninth head on its own, spare lambda levels
    (1, 640, 9, 128, 1, 11),       # two segments, the last of one pair
    (2, 1024, 6, 64, 6, 12),       # one head a group
    (2, 704, 10, 128, 2, 20),      # a last half pair, the most lambda levels
    (1, 384, 3, 128, 1, 10),       # three pairs, the last of which nobody reads
    (2, 896, 32, 128, 1, 11),      # the same in a second segment, enough of them for either order of completion
    (1, 1344, 4, 64, 2, 12),       # ... and the last pair a half
    (1, 8832, 1, 128, 1, 15),      # eighteen segments: readers of a fifth high level, for which a second CTA is there
])
def test_gradients_of_a_cta_match_oracle(B, T, H, N, G, L):
    q, k, v, g, l, do = rounded_inputs(B, T, H, 64, N, G, L, seed=T + 5 * H)
    _, grads = run_cuda(q, k, v, g, l, do)
    _, want = orc.mamba2_grads(q, k, v, g, l, do, fn=orc.mamba2_chunkwise_blocked if T > 4096 else orc.mamba2_chunkwise)
    for got, ref, key in zip(grads, want, ("dq", "dk", "dv", "dg", "dl")):
        assert_close(got, ref, key)


@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H", [(576, 9), (1024, 2)])
def test_residual_of_a_layer(T, H, params):
    """y = bf16(o) + D x, in the parameters' dtype, leaves by way of the tile of x: every row of it, and nothing behind the sequence's end."""
    from hattention_b200.base import HStruct, HType
    from hattention_b200.mamba_apis import hmamba_chunk_scan_combined
    dev, L = torch.device("cuda:0"), 12
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
