"""Performance cases of log-linear attention: the calls that a program makes of this package, at the sizes at which
it makes them.  Each case is a dict of plain values; `prepare` makes what such a program has in hand before the
call, `run` is one pass through the public entry points.

Sizes: the configurations of BASELINE.json (forward B=8 T=4096 H=24; forward + backward B=2 T=16384 H=32; Gated
DeltaNet B=4 T=8192 H=16, 128 x 128 heads; one GPU's share of the 65536-token configuration), the head counts of the
models that reach these kernels (48 heads of 64 x 128 for Mamba-2, 6 heads for Gated DeltaNet), and the state widths,
group counts, ragged lengths and wide value heads of the test-suite."""
import math
import os
import sys

import torch

# the package's folder in the repository that is the working folder
sys.path.insert(0, os.path.join(os.getcwd(), "log-linear-attention_b200"))

from hattention_b200 import HState, HStruct, HType, hattention_kernel  # noqa: E402
from hattention_b200.gated_delta_rule_apis import chunk_h_gated_delta_rule  # noqa: E402
from hattention_b200.mamba_apis import (  # noqa: E402
    hmamba_chunk_scan_combined, hmamba_split_conv1d_scan_combined, hselective_state_update)

P = 64          # width of a Mamba-2 head
CHUNK = 64


def listed():
    return [
        # generation of one sequence, one layer and token at a time: the smallest call, launches and host work count
        {"name": "mamba2 decode B1", "kind": "mamba2_decode", "B": 1, "H": 48, "N": 128, "G": 1, "L": 15, "position": 3000,
         "params": "bfloat16"},
        # generation for a batch of sequences: the level states go through memory once per token
        {"name": "mamba2 decode B64", "kind": "mamba2_decode", "B": 64, "H": 32, "N": 128, "G": 1, "L": 15, "position": 3000,
         "params": "bfloat16"},
        # a prompt before generation; its length is whatever the text has
        {"name": "mamba2 prompt T1000", "kind": "mamba2_prompt", "B": 1, "T": 1000, "H": 48, "N": 128, "G": 1, "L": 15,
         "params": "bfloat16"},
        # scoring / evaluation: forward without gradients (the forward configuration)
        {"name": "mamba2 forward T4096", "kind": "mamba2_forward", "B": 8, "T": 4096, "H": 24, "N": 128, "G": 1, "L": 13,
         "params": "bfloat16"},
        # training step of the layer's scan with fp32 master parameters (the headline configuration)
        {"name": "mamba2 train T16384", "kind": "mamba2_train", "B": 2, "T": 16384, "H": 32, "N": 128, "G": 1, "L": 15,
         "params": "float32"},
        # short fine-tuning sequences: an odd number of chunks, the narrow state, two groups of B / C
        {"name": "mamba2 train odd N64", "kind": "mamba2_train", "B": 2, "T": 1984, "H": 8, "N": 64, "G": 2, "L": 12,
         "params": "bfloat16"},
        # long context: one GPU's share of the 65536-token configuration, through the kernel-level entry point
        {"name": "mamba2 kernel T65536", "kind": "mamba2_kernel", "B": 1, "T": 65536, "H": 32, "N": 128, "G": 1, "L": 17},
        # training step of the whole mixer: convolution, scan, gated norm, output projection
        {"name": "mamba2 block T8192", "kind": "mamba2_block", "B": 1, "T": 8192, "H": 48, "N": 128, "G": 1, "L": 15,
         "params": "bfloat16"},
        # generation with Gated DeltaNet heads
        {"name": "gdn decode B16", "kind": "gdn_decode", "B": 16, "H": 16, "Dk": 128, "Dv": 128, "L": 15, "position": 3000},
        # a prompt for Gated DeltaNet
        {"name": "gdn prompt T777", "kind": "gdn_prompt", "B": 1, "T": 777, "H": 16, "Dk": 128, "Dv": 128, "L": 15},
        # training step of the Gated DeltaNet configuration
        {"name": "gdn train T8192", "kind": "gdn_train", "B": 4, "T": 8192, "H": 16, "Dk": 128, "Dv": 128, "L": 14},
        # few heads with values twice as wide as the keys, an odd number of chunks
        {"name": "gdn train wide T2112", "kind": "gdn_train", "B": 1, "T": 2112, "H": 6, "Dk": 128, "Dv": 256, "L": 14},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _levels(T):
    """Levels that a sequence of T tokens needs (whole chunks), as the drivers count them."""
    return 7 + (-(-T // CHUNK) - 1).bit_length()


def draw(rng):
    kind = rng.choice(["mamba2_decode", "mamba2_prompt", "mamba2_forward", "mamba2_train", "mamba2_kernel", "mamba2_block",
                       "gdn_decode", "gdn_prompt", "gdn_train"])
    c = {"kind": kind}
    mamba2 = kind.startswith("mamba2")
    H = c["H"] = rng.choice([4, 8, 16, 24, 32, 48]) if mamba2 else rng.choice([2, 4, 6, 12, 16])
    if mamba2:
        c["N"] = rng.choice([64, 128, 128, 128])
        c["G"] = rng.choice([1, 1, 2])
        if kind != "mamba2_kernel":
            c["params"] = rng.choice(["float32", "bfloat16"])
    else:
        c["Dk"] = rng.choice([64, 128, 128])
        c["Dv"] = rng.choice([64, 128, 128, 192, 256])
    if kind.endswith("decode"):
        c["B"] = _log_int(rng, 1, 64)
        c["L"] = 15
        c["position"] = _log_int(rng, 10, 8000)
        return c
    if kind.endswith("prompt"):
        c["B"] = rng.choice([1, 1, 2, 4])
        c["T"] = _log_int(rng, 16, 8000)
        c["L"] = 15
        return c
    # (batch x tokens x heads) of one pass, bounded by the largest listed case of the same kind
    most = {"mamba2_forward": 8 * 4096 * 24, "mamba2_train": 2 * 16384 * 32, "mamba2_kernel": 65536 * 32,
            "mamba2_block": 8192 * 48, "gdn_train": 4 * 8192 * 16 * 128 // max(128, c.get("Dv", 0))}[kind]
    longest = 256 if not mamba2 else 1024 if kind == "mamba2_kernel" else 256
    c["B"] = rng.choice([1, 2, 4, 8])
    chunks = _log_int(rng, 2, longest)
    c["T"] = CHUNK * max(1, min(chunks, most // (c["B"] * H * CHUNK)))
    c["L"] = _levels(c["T"]) + rng.choice([0, 1, 2])
    return c


def _softplus(x):
    return torch.nn.functional.softplus(x)


class _Draws:
    """Tensors from one seed, made on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda")
        self.gen = torch.Generator(device=self.dev).manual_seed(seed)

    def randn(self, *shape, dtype=torch.bfloat16, scale=1.0, shift=0.0):
        return (torch.randn(shape, generator=self.gen, device=self.dev) * scale + shift).to(dtype)

    def rand(self, *shape):
        return torch.rand(shape, generator=self.gen, device=self.dev)


def _level_state(d, case, hstruct, K, V):
    """Level states after `position` tokens: every level that holds tokens is filled, the others are zero."""
    s = HState(base=2, htype=HType.WEAK, hstruct=hstruct, shape=(case["B"], case["H"], K, V, case["L"]), dtype=torch.float32,
               device=d.dev)
    s.set_counts_after(case["position"])
    for level, count in enumerate(s.counts):
        if count:
            s.states[..., level] = d.randn(case["B"], case["H"], K, V, dtype=torch.float32, scale=0.05)
    return s


def _mamba2_parameters(d, case):
    """A (fp32, as -exp of its logarithm is), and the per-head parameters in the dtype the model keeps them in."""
    H, L = case["H"], case["L"]
    dt = getattr(torch, case["params"])
    return {"A": -torch.exp(d.rand(H) * math.log(16.0)), "L": (d.rand(H, L) + 0.5).to(dt), "D": d.randn(H, dtype=dt),
            "dt_bias": d.randn(H, dtype=dt, scale=0.1)}


_MAMBA2 = dict(lambda_mode="positive", lambda_level_base=2, lambda_htype=HType.WEAK, lambda_hstruct=HStruct.MAMBA2,
               lambda_level_fixed=True)


def prepare(case, seed):
    d = _Draws(seed)
    kind = case["kind"]
    B, H, L = case["B"], case["H"], case["L"]
    T = case.get("T", 1)
    st = {"case": case}
    if kind.startswith("mamba2"):
        N, G = case["N"], case["G"]
        bc = 1.0 / math.sqrt(N)
        if kind == "mamba2_kernel":
            step = _softplus(d.randn(B, T, H, dtype=torch.float32, shift=-2.0))
            A = -torch.exp(d.rand(H) * math.log(16.0))
            v = (d.randn(B, T, H, P, dtype=torch.float32) * step[..., None]).bfloat16()
            ins = [d.randn(B, T, G, N, scale=bc), d.randn(B, T, G, N, scale=bc), v, A * step,
                   _softplus(d.randn(B, T, H, L, dtype=torch.float32)).bfloat16()]
            st["ins"] = [x.requires_grad_(True) for x in ins]
            st["dy"] = d.randn(B, T, H, P)
            return st
        st["kw"] = dict(_MAMBA2, lambda_level_max=L)
        par = st["par"] = _mamba2_parameters(d, case)
        if kind == "mamba2_decode":
            st["state"] = _level_state(d, case, HStruct.MAMBA2, N, P)
            st["x"] = d.randn(B, H, P)
            st["dt"] = d.randn(B, H, shift=-2.0)
            st["Bm"], st["Cm"] = d.randn(B, G, N, scale=bc), d.randn(B, G, N, scale=bc)
            st["dl"] = d.randn(B, H, L)
            return st
        if kind == "mamba2_block":
            dim, hidden, width = H * P, H * P // 2, 4
            conv = dim + 2 * G * N
            dt = getattr(torch, case["params"])
            st["zx"] = d.randn(B, T, 2 * dim + 2 * G * N + H + H * L)
            par["dt_bias"] = d.randn(H, dtype=dt, scale=0.1, shift=-2.0)
            st["conv_w"], st["conv_b"] = d.randn(conv, width, dtype=dt, scale=0.3), d.randn(conv, dtype=dt, scale=0.1)
            st["norm_w"] = (d.rand(dim) + 0.5).to(dt)
            st["out_w"] = d.randn(hidden, dim, dtype=dt, scale=dim ** -0.5)
            st["grads_of"] = [st["zx"], st["conv_w"], st["conv_b"], par["dt_bias"], par["A"], par["L"], par["D"], st["norm_w"],
                              st["out_w"]]
            for x in st["grads_of"]:
                x.requires_grad_(True)
            st["dy"] = d.randn(B, T, hidden)
            return st
        st["x"] = d.randn(B, T, H, P)
        st["dt"] = d.randn(B, T, H, shift=-2.0)
        st["Bm"], st["Cm"] = d.randn(B, T, G, N, scale=bc), d.randn(B, T, G, N, scale=bc)
        st["dl"] = d.randn(B, T, H, L)
        if kind == "mamba2_train":
            st["grads_of"] = [st["x"], st["dt"], par["A"], st["Bm"], st["Cm"], st["dl"], par["L"], par["D"], par["dt_bias"]]
            for x in st["grads_of"]:
                x.requires_grad_(True)
            st["dy"] = d.randn(B, T, H, P, dtype=getattr(torch, case["params"]))
        return st
    Dk, Dv = case["Dk"], case["Dv"]
    ins = {"q": d.randn(B, T, H, Dk), "k": d.randn(B, T, H, Dk), "v": d.randn(B, T, H, Dv),
           "g": torch.nn.functional.logsigmoid(d.randn(B, T, H, dtype=torch.float32, shift=3.0)),
           "l": _softplus(d.randn(B, T, H, L, dtype=torch.float32)).bfloat16(),
           "beta": torch.sigmoid(d.randn(B, T, H, dtype=torch.float32)).bfloat16()}
    st["ins"] = ins
    if kind == "gdn_decode":
        st["state"] = _level_state(d, case, HStruct.GDELTA, Dk, Dv)
    if kind == "gdn_train":
        for x in ins.values():
            x.requires_grad_(True)
        st["dy"] = d.randn(B, T, H, Dv)
    return st


def _next_token(state):
    """A state whose levels are full belongs to a sequence that has ended: the next one starts from empty levels."""
    if sum(state.counts) >= 1 << (state.max_num_levels - 1):
        state.reset_states()
    return state


def _scan(st, **more):
    par = st["par"]
    return hmamba_chunk_scan_combined(st["x"], st["dt"], par["A"], st["Bm"], st["Cm"], st["dl"], par["L"], CHUNK, D=par["D"],
                                      dt_bias=par["dt_bias"], dt_softplus=True, **st["kw"], **more)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "mamba2_decode":
        par = st["par"]
        with torch.no_grad():
            y, state = hselective_state_update(_next_token(st["state"]), st["x"], st["dt"], par["A"], st["Bm"], st["Cm"], st["dl"],
                                               par["L"], D=par["D"], dt_bias=par["dt_bias"], dt_softplus=True, **st["kw"])
        return [y, state.states, state.counts]
    if kind == "mamba2_prompt":
        with torch.no_grad():
            y, state = _scan(st, return_final_states=True)
        return [y, state.states, state.counts]
    if kind == "mamba2_forward":
        with torch.no_grad():
            return _scan(st)[0]
    if kind == "mamba2_train":
        y, _ = _scan(st)
        return [y.detach(), *torch.autograd.grad(y, st["grads_of"], st["dy"])]
    if kind == "mamba2_kernel":
        q, k, v, g, l = st["ins"]
        o = hattention_kernel(q, k, v, None, g, l, None, False, 2, HType.WEAK, HStruct.MAMBA2)
        return [o.detach(), *torch.autograd.grad(o, st["ins"], st["dy"])]
    if kind == "mamba2_block":
        par = st["par"]
        y = hmamba_split_conv1d_scan_combined(
            st["zx"], st["conv_w"], st["conv_b"], par["dt_bias"], par["A"], par["L"], par["D"], CHUNK, rmsnorm_weight=st["norm_w"],
            outproj_weight=st["out_w"], headdim=P, ngroups=case["G"], norm_before_gate=False, **st["kw"])
        return [y.detach(), *torch.autograd.grad(y, st["grads_of"], st["dy"])]
    if kind == "gdn_decode":
        with torch.no_grad():
            o, state = chunk_h_gated_delta_rule(**st["ins"], initial_state=_next_token(st["state"]), output_final_state=True,
                                                use_qk_l2norm_in_kernel=True)
        return [o, state.states, state.counts]
    if kind == "gdn_prompt":
        with torch.no_grad():
            o, state = chunk_h_gated_delta_rule(**st["ins"], output_final_state=True, use_qk_l2norm_in_kernel=True)
        return [o, state.states, state.counts]
    ins = st["ins"]
    o, _ = chunk_h_gated_delta_rule(**ins, use_qk_l2norm_in_kernel=True)
    return [o.detach(), *torch.autograd.grad(o, list(ins.values()), st["dy"])]


def work(case):
    """Inputs read once, outputs written once; operations of the chunkwise algorithm on dense 64 x 64 tiles."""
    kind = case["kind"]
    B, H, L, T = case["B"], case["H"], case["L"], case.get("T", 1)
    rows = B * T * H
    NT = T / CHUNK
    Lc = max(0, (-(-T // CHUNK) - 1).bit_length())
    C = CHUNK
    if kind.startswith("mamba2"):
        N, G = case["N"], case["G"]
        K, V = N, P
        qk = 2 * B * T * G * N * 2
    else:
        K, V = case["Dk"], case["Dv"]
        qk = 2 * rows * K * 2
    pb = 4 if case.get("params") == "float32" else 2                 # fp32 parameters promote the output
    io = qk + rows * V * 2 + rows * (L * 2 + 4)                      # q, k, v (x), levels, decay / step
    if kind.endswith("decode"):
        # levels that hold tokens, over the positions that follow: half of those that have been reached
        live = max(1.0, case["position"].bit_length() / 2)
        return {"bytes": io + rows * V * 2 + 2 * 4 * B * H * K * V * live, "flops": (4 if kind.startswith("mamba2") else 8) * B * H * K * V * live}
    CK, CV, S = 2 * C * C * K, 2 * C * C * V, 2 * C * K * V
    per = B * H * NT
    if kind.startswith("mamba2"):
        fwd, bwd = CK + CV + (1 + Lc / 2) * S, 3 * CK + 2 * CV + (3 + Lc) * S
    else:
        # q k^T, k k^T, the two transforms of k and v, P v; kd^T u, w h, q h per level
        fwd, bwd = 3 * CK + 2 * CV + (2 + Lc) * S, 6 * CK + 4 * CV + (4 + 2 * Lc) * S
    if kind.endswith("prompt"):
        return {"bytes": io + rows * V * 2 + 4 * B * H * K * V * L, "flops": (fwd + S) * per}
    if kind == "mamba2_forward":
        return {"bytes": io + rows * V * 2, "flops": fwd * per}
    grads = io + rows * V * 2                                        # inputs again, their gradients, the upstream gradient
    if kind == "mamba2_block":
        dim = H * P
        width = 2 * dim + 2 * G * N + H + H * L
        proj = dim * dim // 2
        return {"bytes": B * T * (3 * width + 2 * dim // 2) * 2 + 3 * proj * pb, "flops": (fwd + bwd) * per + 3 * 2 * B * T * proj}
    return {"bytes": io + rows * V * pb + grads + io, "flops": (fwd + bwd) * per}


def tolerance(case):
    # bf16 operands and outputs, fp32 accumulation
    return {"rel": 1e-2}
