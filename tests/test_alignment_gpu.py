"""Operands that are contiguous views into larger tensors and start between the boundaries of the kernels' vector accesses."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def shifted(x):
    """The same values, two or four bytes behind a 16-byte boundary."""
    flat = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
    y = flat[1:].view(x.shape)
    y.copy_(x)
    assert y.is_contiguous() and y.data_ptr() % 16 == x.element_size()
    return y


def bf(*s):
    return torch.randn(*s, device=DEV).bfloat16()


def same(a, b):
    if torch.is_tensor(a):
        # gradients that are sums over tokens come from atomics in any order
        assert (a.double() - b.double()).norm() <= 2e-3 * b.double().norm() + 1e-6
    elif isinstance(a, (list, tuple)):
        for x, y in zip(a, b):
            same(x, y)


def _mamba2_kernel():
    from hattention_b200 import HStruct, HType, hattention_kernel
    B, T, H, G, N, L = 1, 192, 4, 1, 128, 12
    ins = [bf(B, T, G, N) / 11, bf(B, T, G, N) / 11, bf(B, T, H, 64), -torch.rand(B, T, H, device=DEV), bf(B, T, H, L)]
    dy = bf(B, T, H, 64)

    def run(f):
        x = [f(t).requires_grad_(True) for t in ins]
        o = hattention_kernel(*x[:3], None, *x[3:], None, False, 2, HType.WEAK, HStruct.MAMBA2)
        return [o.detach(), *torch.autograd.grad(o, x, f(dy))]
    return run


def _layer(prompt):
    def make():
        from hattention_b200 import HStruct, HType
        from hattention_b200.mamba_apis import hmamba_chunk_scan_combined
        B, T, H, G, N, L = 2, 128 + 7 * prompt, 8, 2, 64, 12
        ins = [bf(B, T, H, 64), bf(B, T, H), -torch.rand(H, device=DEV), bf(B, T, G, N) / 8, bf(B, T, G, N) / 8, bf(B, T, H, L), bf(H, L), bf(H), bf(H)]
        dy = bf(B, T, H, 64)
        kw = dict(dt_softplus=True, lambda_mode="positive", lambda_level_max=L, lambda_level_base=2, lambda_htype=HType.WEAK,
                  lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True, return_final_states=bool(prompt))

        def run(f):
            x = [f(t).requires_grad_(not prompt) for t in ins]
            y, s = hmamba_chunk_scan_combined(*x[:7], 64, D=x[7], dt_bias=x[8], **kw)
            return [y, s.states] if prompt else [y.detach(), *torch.autograd.grad(y, x, f(dy))]
        return run
    return make


def _mixer():
    from hattention_b200 import HStruct, HType
    from hattention_b200.mamba_apis import hmamba_split_conv1d_scan_combined
    B, T, H, G, N, L = 1, 128, 8, 1, 128, 12
    dim = H * 64
    ch = dim + 2 * G * N
    ins = [bf(B, T, 2 * dim + 2 * G * N + H + H * L), bf(ch, 4) * 0.3, bf(ch), bf(H), -torch.rand(H, device=DEV), bf(H, L), bf(H), bf(dim), bf(64, dim) / 20]
    dy = bf(B, T, 64)

    def run(f):
        # (the weight of the output projection as it is: torch's product with a shifted one rounds differently)
        x = [f(t).requires_grad_(True) for t in ins[:-1]] + [ins[-1].clone().requires_grad_(True)]
        y = hmamba_split_conv1d_scan_combined(*x[:7], 64, rmsnorm_weight=x[7], outproj_weight=x[8], headdim=64, ngroups=G, norm_before_gate=False,
                                              lambda_mode="positive", lambda_level_max=L, lambda_level_base=2, lambda_htype=HType.WEAK,
                                              lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)
        return [y.detach(), *torch.autograd.grad(y, x, f(dy))]
    return run


def _gdn(prompt):
    def make():
        from hattention_b200.gated_delta_rule_apis import chunk_h_gated_delta_rule
        B, T, H, D, L = 2, 128 + 5 * prompt, 4, 128, 10
        ins = [bf(B, T, H, D), bf(B, T, H, D), bf(B, T, H, D), -torch.rand(B, T, H, device=DEV), bf(B, T, H, L).abs(), torch.rand(B, T, H, device=DEV).bfloat16()]
        dy = bf(B, T, H, D)

        def run(f):
            x = [f(t).requires_grad_(not prompt) for t in ins]
            o, s = chunk_h_gated_delta_rule(*x, use_qk_l2norm_in_kernel=True, output_final_state=bool(prompt))
            return [o, s.states] if prompt else [o.detach(), *torch.autograd.grad(o, x, f(dy))]
        return run
    return make


def _step(struct, shift_states):
    def make():
        from hattention_b200 import HState, HStruct, HType
        from hattention_b200.kernel import hattention_step
        gdn = struct == "GDELTA"
        B, H, K, V, L = 2, 4, 128, 64, 10
        states = torch.randn(B, H, L, K, V, device=DEV)
        states[:, :, 9] = 0                          # 256 tokens fill the levels below
        args = [bf(B, H, K), bf(B, H, K), bf(B, H, V), torch.rand(B, H, device=DEV).bfloat16() if gdn else None, -torch.rand(B, H, device=DEV), bf(B, H, L)]

        def run(f):
            s = HState.holding((f(states) if shift_states else states.clone()).permute(0, 1, 3, 4, 2), 2, HType.WEAK, HStruct[struct])
            s.set_counts_after(256)
            x = [f(t) if t is not None else None for t in args]
            with torch.no_grad():
                o, s = hattention_step(s, *x, K ** -0.5 if gdn else None, 2, HType.WEAK, HStruct[struct], gdn)
            return [o, s.states]
        return run
    return make


@pytest.mark.parametrize("make", [_mamba2_kernel, _layer(0), _layer(1), _mixer, _gdn(0), _gdn(1), _step("MAMBA2", 0), _step("MAMBA2", 1),
                                  _step("GDELTA", 0), _step("GDELTA", 1)],
                         ids=["mamba2 kernel", "layer", "layer prompt", "mixer", "gdn", "gdn prompt", "mamba2 step", "mamba2 states", "gdn step", "gdn states"])
def test_misaligned_operands_give_the_same(make):
    torch.manual_seed(0)
    run = make()
    same(run(shifted), run(lambda x: x.clone()))
