"""The backward of the l2 normalisation inside the chunk-local kernel, against the pass of its own that follows a backward which recomputes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,V,L,lam", [(1, 64, 1, 64, 7, 0.0), (2, 320, 3, 128, 11, 0.0), (1, 1088, 2, 64, 13, 0.5)])
def test_normalisation_backward_matches_the_separate_pass(B, T, H, V, L, lam):
    from hattention_b200 import kernel
    dev = torch.device("cuda:0")
    gen = torch.Generator().manual_seed(T + V)
    r = lambda *s: torch.randn(*s, generator=gen)
    base = [r(B, T, H, 128) * 3, r(B, T, H, 128) * .5, r(B, T, H, V), torch.sigmoid(r(B, T, H)), -torch.rand(B, T, H, generator=gen) * .1,
            torch.rand(B, T, H, L, generator=gen)]
    base[0][0, 0] = 0                                      # a row of zeros: the epsilon under the root
    base = [x.to(dev, torch.float32 if i == 4 else torch.bfloat16) for i, x in enumerate(base)]
    do = r(B, T, H, V).bfloat16().to(dev)

    def grads(keep):
        was, kernel.KEEP_FORWARD_STATES = kernel.KEEP_FORWARD_STATES, keep
        try:
            ins = [x.clone().requires_grad_(True) for x in base]
            return torch.autograd.grad(kernel.gdn_native(*ins, 128 ** -0.5, lam), ins, do)
        finally:
            kernel.KEEP_FORWARD_STATES = was

    for a, b, name in zip(grads(True), grads(False), ("q", "k", "v", "b", "g", "l")):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.isfinite(a).all(), name
        assert (a.double() - b.double()).norm() <= 5e-3 * b.double().norm(), name
