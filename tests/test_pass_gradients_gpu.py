"""The backward passes around the scan, each alone: from given upstream tensors, so that its sums over tokens are compared with an fp64 evaluation of
the same operators and not with what the scan's rounding leaves of them.  The upstream values have random signs: the parameter sums do not
cancel, and a run of tokens, a head or a column that is left out shows."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
I, F, P, Lg = ctypes.c_int, ctypes.c_float, ctypes.c_void_p, ctypes.c_long


def call(name, *args):
    from hattention_b200 import _lib
    fn = getattr(_lib.lib(), name)
    old, fn.argtypes = fn.argtypes, None
    try:
        rc = fn(*[P(a.data_ptr()) if torch.is_tensor(a) else P(0) if a is None else a for a in args],
                P(torch.cuda.current_stream().cuda_stream))
    finally:
        fn.argtypes = old
    assert rc == 0, (name, rc)


def close(got, want, name, bound):
    got, want = got.double(), want.double()
    err = ((got - want).norm() / want.norm()).item()
    assert got.shape == want.shape and err < bound, (name, err)


def lam_of(mode, lp, d):
    sp = torch.nn.functional.softplus
    return sp(lp * d) if mode == 0 else torch.exp(-torch.exp(lp) * sp(d)) if mode == 1 else lp * d


def leaf(x):
    return x.double().requires_grad_(True)


class Draws:
    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def __call__(self, *s, dtype=torch.bfloat16, scale=1.0, shift=0.0):
        return (torch.randn(s, generator=self.gen, device=DEV) * scale + shift).to(dtype)


# fp32 results: sums of up to B T 64 exact products in fp32, and the fast exponential (1e-6); bf16 results: one rounding (2e-3)
FP32, BF16 = 1e-4, 4e-3


# runs of tokens that end inside a sequence; heads that do not fill a CTA, or take several; lambda columns that come in eights or not
@pytest.mark.parametrize("rows,H,L", [(1, 2, 9), (65, 3, 7), (1000, 8, 15), (2113, 6, 14), (333, 48, 15)])
@pytest.mark.parametrize("mode,params", [(0, torch.float32), (1, torch.bfloat16), (2, torch.bfloat16)])
def test_layer_prep_bwd(rows, H, L, mode, params):
    d = Draws(rows + H)
    x, dv, dy = d(rows, H, 64), d(rows, H, 64), d(rows, H, 64)
    dt, dl = d(rows, H, shift=-1.0), d(rows, H, L)
    dg, dlam = d(rows, H, dtype=torch.float32), d(rows, H, L, dtype=torch.float32)
    A = -torch.exp(d(H, dtype=torch.float32))
    bias, Lp, D = d(H, dtype=params, scale=0.3), d(H, L, dtype=params, scale=0.3, shift=1.0), d(H, dtype=params)
    f32 = I(params == torch.float32)
    dx, ddt, ddl = torch.empty_like(x), torch.empty_like(dt), torch.empty_like(dl)
    dA, db, dD, dL = (torch.zeros(n, device=DEV) for n in (H, H, H, H * L))
    call("llattn_mamba2_layer_prep_bwd", x, dt, bias, f32, A, dl, Lp, f32, D, f32, dv, dg, dlam, dy, dx, ddt, ddl, dA, db, dL, dD, Lg(rows * H), I(H), I(64),
         I(L), I(mode))
    t = [leaf(v) for v in (x, dt, A, dl, bias, Lp, D)]
    step = torch.nn.functional.softplus(t[1] + t[4])
    loss = (t[0] * step[..., None] * dv.double()).sum() + (t[2] * step * dg.double()).sum() + (lam_of(mode, t[5], t[3]) * dlam.double()).sum() \
        + (t[0] * t[6][:, None] * dy.double()).sum()
    want = torch.autograd.grad(loss, t)
    for got, w, name, bound in zip((dx, ddt, dA, ddl, db, dL.view(H, L), dD), want, ("dx", "ddt", "dA", "ddl", "dbias", "dL", "dD"),
                                   (BF16, BF16, FP32, BF16, FP32, FP32, FP32)):
        close(got, w, name, bound)


@pytest.mark.parametrize("B,T,H,G,N,L", [(1, 64, 2, 1, 128, 9), (2, 100, 5, 1, 64, 8), (1, 1000, 8, 2, 64, 15), (2, 2113, 6, 1, 128, 14), (1, 333, 48, 1, 128, 15)])
@pytest.mark.parametrize("mode,params,cbias", [(0, torch.float32, True), (1, torch.bfloat16, False)])
def test_mixer_prep_bwd(B, T, H, G, N, L, mode, params, cbias):
    d = Draws(T + H)
    dim, gn = H * 64, G * N
    ch, W = dim + 2 * gn, 2 * dim + 2 * gn + H + H * L
    zx = d(B, T, W)
    cw, cb, bias = d(ch, 4, dtype=torch.bfloat16, scale=0.3).to(params), d(ch, dtype=torch.bfloat16, scale=0.1).to(params), d(H, dtype=params, shift=-1.0)
    A, Lp, D = -torch.exp(d(H, dtype=torch.float32)), d(H, L, dtype=params, scale=0.3, shift=1.0), d(H, dtype=params)
    dv, dy, dq, dk = d(B, T, dim), d(B, T, dim), d(B, T, gn), d(B, T, gn)
    dg, dlam = d(B, T, H, dtype=torch.float32), d(B, T, H, L, dtype=torch.float32)
    f32 = I(params == torch.float32)
    dzx = torch.zeros_like(zx)
    dcw, dcb, dA, db, dL = (torch.zeros(n, device=DEV) for n in (ch * 4, ch, H, H, H * L))
    call("llattn_mixer_prep_bwd", zx, cw, f32, cb if cbias else None, f32, bias, f32, A, Lp, f32, D, f32, dv, dy, dq, dk, dg, dlam, dzx, dcw, dcb if cbias else None,
         dA, db, dL, I(B), I(T), I(H), I(G), I(N), I(L), I(mode))
    t = [leaf(v) for v in (zx, cw, cb, bias, A, Lp, D)]
    z, xbc, dt, dl = torch.split(t[0], [dim, ch, H, H * L], dim=-1)
    y = torch.nn.functional.conv1d(xbc.transpose(1, 2), t[1].unsqueeze(1), t[2] if cbias else None, padding=3, groups=ch)[..., :T].transpose(1, 2)
    x, k, q = torch.split(torch.nn.functional.silu(y), [dim, gn, gn], dim=-1)
    step = torch.nn.functional.softplus(dt + t[3])
    xh = x.reshape(B, T, H, 64)
    loss = (xh * step[..., None] * dv.double().view_as(xh)).sum() + (xh * t[6][:, None] * dy.double().view_as(xh)).sum() + (k * dk.double()).sum() \
        + (q * dq.double()).sum() + (t[4] * step * dg.double()).sum() + (lam_of(mode, t[5], dl.reshape(B, T, H, L)) * dlam.double()).sum()
    used = [i for i in range(6) if cbias or i != 2]
    want = dict(zip(used, torch.autograd.grad(loss, [t[i] for i in used])))
    # the pass rounds the convolution's output to bf16 before the activation, as the forward does: 2^-9 of each term, at random
    close(dzx[..., dim:], want[0][..., dim:], "dzx", 2 * BF16)
    close(dcw.view(ch, 4), want[1], "dconv_w", 1e-2)
    if cbias:
        close(dcb, want[2], "dconv_b", 1e-2)
    close(db, want[3], "dbias", 1e-2)
    close(dA, want[4], "dA", FP32)
    close(dL.view(H, L), want[5], "dL", FP32)


# tokens below and above the persistent CTAs; heads of one CTA, of 4096 columns and beyond
@pytest.mark.parametrize("rows,H", [(1, 2), (100, 5), (1000, 16), (2113, 48), (333, 64), (129, 80)])
@pytest.mark.parametrize("params", [torch.float32, torch.bfloat16])
def test_mixer_norm_bwd(rows, H, params):
    d = Draws(rows + H)
    dim, W = H * 64, H * 64 + 24
    o, x, dn, zx = d(rows, dim), d(rows, dim), d(rows, dim), d(rows, W)
    D, w = d(H, dtype=params), d(dim, dtype=params, scale=0.3, shift=1.0)
    f32 = I(params == torch.float32)
    eps = 1e-6
    out, rstd, dy, dzx = torch.empty_like(o), torch.empty(rows, device=DEV), torch.empty_like(o), torch.zeros_like(zx)
    dw, dD = torch.zeros(dim, device=DEV), torch.zeros(H, device=DEV)
    call("llattn_mixer_norm_fwd", o, x, D, f32, zx, I(W), w, f32, out, rstd, Lg(rows), I(H), F(eps))
    call("llattn_mixer_norm_bwd", o, x, D, f32, zx, I(W), w, f32, dn, rstd, dy, dzx, dw, dD, Lg(rows), I(H))
    t = [leaf(v) for v in (o, x, D, zx, w)]
    y = t[0] + (t[1].view(rows, H, 64) * t[2][:, None]).reshape(rows, dim)
    s = y * torch.nn.functional.silu(t[3][:, :dim])
    r = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + eps) * t[4]
    want = torch.autograd.grad((r * dn.double()).sum(), t)
    # with a bf16 D the sum o + D x is rounded to bf16
    close(out, r, "out", 2 * BF16)
    close(dy, want[0], "dy", 2 * BF16)
    close(dzx[:, :dim], want[3][:, :dim], "dz", 2 * BF16)
    close(dw, want[4], "dw", 2 * BF16)
    close(dD, want[2], "dD", 2 * BF16)


@pytest.mark.parametrize("T,N", [(192, 128), (256, 128), (576, 64), (1088, 128), (1024, 64)])
def test_layer_gradients_match_oracle(T, N):
    """The layer's own gradients, at odd and even chunk counts and both state widths, against fp64 autograd through the oracle.  d A and d dt_bias are sums of
    dg dt that nearly cancel: bounded by 2^-8, the rounding of a bf16 operand, of the sum of their absolute terms."""
    from hattention_b200 import HStruct, HType
    from hattention_b200.mamba_apis import hmamba_chunk_scan_combined
    from oracle import loglinear_oracle as orc
    H, L = 2, 13
    d = Draws(T)
    x, dt, Bm, Cm, dl = d(1, T, H, 64), d(1, T, H, shift=-2.0), d(1, T, 1, N, scale=N ** -0.5), d(1, T, 1, N, scale=N ** -0.5), d(1, T, H, L)
    A, Lp, D, bias, do = -torch.exp(d(H, dtype=torch.float32)), d(H, L, scale=0.2, shift=1.0), d(H), d(H, scale=0.1), d(1, T, H, 64)
    ins = [t.detach().requires_grad_(True) for t in (x, dt, A, Bm, Cm, dl, Lp, D, bias)]
    y, _ = hmamba_chunk_scan_combined(*ins[:7], 64, D=ins[7], dt_bias=ins[8], dt_softplus=True, lambda_mode="positive", lambda_level_max=L, lambda_level_base=2,
                                      lambda_htype=HType.WEAK, lambda_hstruct=HStruct.MAMBA2, lambda_level_fixed=True)
    got = torch.autograd.grad(y, ins, do)
    t = [v.detach().double().cpu().requires_grad_(True) for v in ins]
    step = torch.nn.functional.softplus(t[1] + t[8])
    g = t[2] * step
    o = orc.mamba2_chunkwise(t[4], t[3], t[0] * step[..., None], g, torch.nn.functional.softplus(t[6] * t[5]))
    yr = o + t[0] * t[7][:, None]
    want = torch.autograd.grad((yr * do.double().cpu()).sum(), t + [g])
    close(y.detach().cpu(), yr, "y", 1e-2)
    for i, name in ((0, "dx"), (1, "ddt"), (3, "dB"), (4, "dC"), (5, "ddl"), (6, "dL"), (7, "dD")):
        close(got[i].cpu(), want[i], name, 2e-2 if name == "ddt" else 1e-2)
    terms = {"dA": (want[-1] * step).abs().sum((0, 1)), "dbias": want[1].abs().sum((0, 1))}
    for i, name in ((2, "dA"), (8, "dbias")):
        err = (got[i].double().cpu() - want[i]).abs()
        assert (err <= 2 ** -8 * terms[name] + 2 ** -8 * want[i].abs()).all(), (name, (err / terms[name]).max().item())
