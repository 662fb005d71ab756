"""The fused mixer passes (convolution + preparation, D residual + gated norm, and their backward) against the same call made of
torch operators around the kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


# rows of the projection that are a multiple of 16 bytes / of 4 bytes only; two groups; runs of tokens that end inside and at the
# end of a sequence; heads below and above one CTA of the norm
@pytest.mark.parametrize("B,T,H,G,N,L", [(2, 192, 2, 1, 128, 10), (1, 448, 4, 2, 64, 11), (2, 128, 5, 1, 64, 8), (1, 64, 80, 1, 128, 7),
                                         (1, 2112, 6, 1, 128, 14)])
@pytest.mark.parametrize("mode,params,bias", [("positive", torch.bfloat16, True), ("bounded", torch.float32, True), (None, torch.bfloat16, False)])
def test_mixer_matches_torch_operators(B, T, H, G, N, L, mode, params, bias):
    from hattention_b200 import mamba_apis
    from hattention_b200.base import HStruct, HType
    gen = torch.Generator(device=DEV).manual_seed(T + H)
    rn = lambda *s, scale=1.0, dtype=params: (torch.randn(s, generator=gen, device=DEV) * scale).to(dtype)
    dim, ch = H * 64, H * 64 + 2 * G * N
    base = dict(zx=rn(B, T, 2 * dim + 2 * G * N + H + H * L, dtype=torch.bfloat16), cw=rn(ch, 4, scale=0.3),
                cb=rn(ch, scale=0.1) if bias else None, dtb=rn(H, scale=0.1) - 2, A=-torch.rand(H, generator=gen, device=DEV) * 4 - 0.1,
                Lp=(rn(H, L, scale=0.2) + 1), D=rn(H), nw=rn(dim, scale=0.2) + 1, ow=rn(96, dim, scale=dim ** -0.5))
    dout = rn(B, T, 96, dtype=torch.bfloat16)

    def run(fused):
        mamba_apis.FUSED_PREP = fused
        try:
            t = {k: v if v is None else v.clone().requires_grad_(True) for k, v in base.items()}
            y = mamba_apis.hmamba_split_conv1d_scan_combined(
                t["zx"], t["cw"], t["cb"], t["dtb"], t["A"], t["Lp"], t["D"], 64, rmsnorm_weight=t["nw"], outproj_weight=t["ow"],
                headdim=64, ngroups=G, norm_before_gate=False, lambda_mode=mode, lambda_level_max=L, lambda_level_base=2,
                lambda_htype=HType.WEAK, lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)
            names = [k for k in t if t[k] is not None]
            return y.detach(), dict(zip(names, torch.autograd.grad(y, [t[k] for k in names], dout)))
        finally:
            mamba_apis.FUSED_PREP = True

    y1, g1 = run(True)
    y0, g0 = run(False)
    rel = lambda a, b: ((a.float() - b.float()).norm() / b.float().norm()).item()
    assert y1.dtype == y0.dtype and rel(y1, y0) < 1e-2
    for k in g0:
        assert g1[k].shape == g0[k].shape and g1[k].dtype == g0[k].dtype, k
        # the gradients of A and dt_bias are sums over B T tokens of signed terms that nearly cancel in the short cases: what the scan rounds differently
        # is a tenth of them there (test_pass_gradients_gpu.py compares these sums alone, with fp64)
        assert rel(g1[k], g0[k]) < (0.25 if k in ("A", "dtb") else 3e-2 if k in ("Lp", "D") else 1.5e-2), (k, rel(g1[k], g0[k]))
