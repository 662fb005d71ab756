"""Derivatives and transforms that the kernels do not have are refused, not dropped."""
import pytest
import torch
import torch.autograd.forward_ad as fwad

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def bf(*s):
    return torch.randn(*s, device=DEV).bfloat16()


def _kernel(v):
    from hattention_b200 import HStruct, HType, hattention_kernel
    B, T, H, _ = v.shape
    return hattention_kernel(bf(B, T, 1, 128), bf(B, T, 1, 128), v, None, -torch.rand(B, T, H, device=DEV), bf(B, T, H, 9), None, False, 2, HType.WEAK,
                             HStruct.MAMBA2)


def _gdn(v):
    from hattention_b200.gated_delta_rule_apis import chunk_h_gated_delta_rule
    B, T, H, _ = v.shape
    return chunk_h_gated_delta_rule(bf(B, T, H, 128), bf(B, T, H, 128), v, -torch.rand(B, T, H, device=DEV), bf(B, T, H, 9), bf(B, T, H).sigmoid(),
                                    use_qk_l2norm_in_kernel=True)[0]


def _layer(x):
    from hattention_b200 import HStruct, HType
    from hattention_b200.mamba_apis import hmamba_chunk_scan_combined
    B, T, H, _ = x.shape
    return hmamba_chunk_scan_combined(x, bf(B, T, H), -torch.rand(H, device=DEV), bf(B, T, 1, 128), bf(B, T, 1, 128), bf(B, T, H, 9), bf(H, 9), 64,
                                      dt_softplus=True, lambda_mode="positive", lambda_level_max=9, lambda_level_base=2, lambda_htype=HType.WEAK,
                                      lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)[0]


def _mixer(z):
    from hattention_b200 import HStruct, HType
    from hattention_b200.mamba_apis import hmamba_split_conv1d_scan_combined
    H = 2
    return hmamba_split_conv1d_scan_combined(z, bf(H * 64 + 256, 4), bf(H * 64 + 256), bf(H), -torch.rand(H, device=DEV), bf(H, 9), bf(H), 64,
                                             rmsnorm_weight=bf(H * 64), outproj_weight=bf(64, H * 64), headdim=64, ngroups=1, norm_before_gate=False,
                                             lambda_mode="positive", lambda_level_max=9, lambda_level_base=2, lambda_htype=HType.WEAK,
                                             lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)


CALLS = pytest.mark.parametrize("call,shape", [(_kernel, (1, 64, 2, 64)), (_gdn, (1, 64, 2, 64)), (_layer, (1, 64, 2, 64)), (_mixer, (1, 64, 532))])


@CALLS
def test_forward_mode_is_refused(call, shape):
    x = bf(*shape)
    call(x)
    with fwad.dual_level(), pytest.raises(NotImplementedError):
        call(fwad.make_dual(x, torch.ones_like(x)))


@CALLS
def test_function_transforms_are_refused(call, shape):
    x = bf(*shape)
    with pytest.raises(Exception):
        torch.func.grad(lambda t: call(t).float().sum())(x)
    with pytest.raises(Exception):
        torch.func.vmap(call, randomness="different")(torch.stack([x, x]))
