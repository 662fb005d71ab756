"""Sequences that end inside a pair of chunks, and K = 64, on the tcgen05 kernels: the second chunk of the last pair, and half of the
state rows, come from the zero fill of the tensor maps, and nothing may be written there."""
import pytest
import torch

from oracle import loglinear_oracle as orc
from test_mamba2_gpu import assert_close, rounded_inputs, run_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,N,G,L", [
    (2, 64, 2, 64, 2, 7),          # half a pair, two sequences: the other half is not the next sequence's first chunk
    (2, 192, 4, 128, 2, 9),        # one pair and a half
    (2, 576, 2, 128, 1, 11),       # a last segment of half a pair
    (1, 960, 2, 64, 1, 11),        # 15 chunks: all but the last half pair of two segments
    (1, 1024, 4, 64, 2, 12),       # whole segments, half the state rows
    (1, 64 * 67, 2, 128, 1, 14),   # nine segments: four high levels
])
def test_ends_inside_a_pair_match_oracle(B, T, H, N, G, L):
    q, k, v, g, l, do = rounded_inputs(B, T, H, 64, N, G, L, seed=3 * T + N)
    o, grads = run_cuda(q, k, v, g, l, do)
    o_ref, g_ref = orc.mamba2_grads(q, k, v, g, l, do, fn=orc.mamba2_chunkwise_blocked if T > 4096 else orc.mamba2_chunkwise)
    assert_close(o, o_ref, "o")
    for got, want, key in zip(grads, g_ref, ("dq", "dk", "dv", "dg", "dl")):
        assert_close(got, want, key)


@pytest.mark.parametrize("T,N", [(192, 128), (576, 64), (1088, 128)])
def test_layer_backward_keeps_the_rounding_of_the_chunk_kernels(T, N):
    """llattn_mamba2_bwd_layer at an odd chunk count or K = 64 gives the gradients of the mma.sync kernels, from states of either forward."""
    from hattention_b200 import _lib
    from hattention_b200.base import HType
    from hattention_b200.mamba_apis import hmamba_chunk_scan_combined
    from hattention_b200.base import HStruct
    dev, H, L = torch.device("cuda:0"), 2, 13
    gen = torch.Generator().manual_seed(T)
    r = lambda *s: torch.randn(*s, generator=gen)
    x, Bm, Cm, dl, do = (t.bfloat16().to(dev) for t in (r(1, T, H, 64), r(1, T, 1, N) / N ** 0.5, r(1, T, 1, N) / N ** 0.5, r(1, T, H, L), r(1, T, H, 64)))
    dt, A, Lp = (r(1, T, H) - 2).bfloat16().to(dev), -torch.exp(r(H)).to(dev), torch.ones(H, L, device=dev).bfloat16()

    def grads():
        ins = [t.detach().requires_grad_(True) for t in (x, dt, A, Bm, Cm, dl, Lp)]
        y, _ = hmamba_chunk_scan_combined(*ins, 64, dt_softplus=True, lambda_mode="positive", lambda_level_max=L, lambda_level_base=2,
                                          lambda_htype=HType.WEAK, lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)
        return torch.autograd.grad(y, ins, do)

    here = grads()
    try:
        _lib.lib().llattn_testing_use_tensor_core_path(0)
        want = grads()
    finally:
        _lib.lib().llattn_testing_use_tensor_core_path(1)
    for a, b in zip(here, want):
        assert (a.double() - b.double()).norm() <= 3e-3 * b.double().norm()


@pytest.mark.parametrize("T,L", [(1024, 21), (4160, 24)])
def test_more_lambda_levels_than_the_tensor_core_kernels_hold(T, L):
    """More than twenty levels: with N = 64 every kernel is a warp-level one, so that the choice between the two generations changes no digit."""
    from hattention_b200 import _lib
    q, k, v, g, l, do = rounded_inputs(1, T, 3, 64, 64, 1, L, seed=T + L)
    o, grads = run_cuda(q, k, v, g, l, do)
    try:
        _lib.lib().llattn_testing_use_tensor_core_path(0)
        want, _ = run_cuda(q, k, v, g, l, do)
    finally:
        _lib.lib().llattn_testing_use_tensor_core_path(1)
    assert torch.equal(o, want)
    o_ref, g_ref = orc.mamba2_grads(q, k, v, g, l, do, fn=orc.mamba2_chunkwise_blocked if T > 4096 else orc.mamba2_chunkwise)
    assert_close(o, o_ref, "o")
    for got, ref, key in zip(grads, g_ref, ("dq", "dk", "dv", "dg", "dl")):
        assert_close(got, ref, key)
