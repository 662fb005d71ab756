"""CPU-side checks of the C ABI: the library loads, exports every symbol that include/llattn.h
declares, and rejects bad arguments before touching a device."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as ge
    ge.build()
    from hattention_b200 import _lib
    return _lib.lib()


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "llattn.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(llattn_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported(lib):
    names = declared_symbols()
    assert "llattn_mamba2_fwd" in names and "llattn_mamba2_bwd" in names
    for n in names:
        assert hasattr(lib, n), n


def test_version_and_chunk(lib):
    assert lib.llattn_version() >= 2
    assert lib.llattn_chunk() == 64
    assert lib.llattn_kernel_launches() >= 0


def test_static_scratch_capacity_stated_in_the_header(lib):
    """include/llattn.h and INTEGRATION.md say: 1.125 MiB per (batch, head) at T = 4096, K = 128, V = 64, so the
    16 MiB array serves B*H <= 14 there."""
    cap = lib.llattn_static_scratch_bytes()
    assert cap == 16 << 20
    need = lambda bh: lib.llattn_mamba2_fwd_workspace_bytes(1, 4096, bh, 1, 128, 64, 13)
    assert abs((need(2) - need(1)) / 2 ** 20 - 1.125) < 1e-3
    assert need(14) <= cap < need(15)
    null = ctypes.c_void_p(0)
    # a size beyond the array is refused before anything touches a device or a pointer; so is a missing pointer
    dummy = ctypes.c_void_p(256)
    assert lib.llattn_mamba2_fwd_static(*([dummy] * 7), 1, 4096, 15, 1, 128, 64, 13, null) == -7
    assert lib.llattn_mamba2_fwd_static(*([null] * 7), 1, 4096, 14, 1, 128, 64, 13, null) == -6


def test_longest_supported_sequence(lib):
    """The scans over segments hold ten segment levels: T = 512 * 1024 is the longest sequence; longer ones are
    refused instead of reading levels that were never written."""
    assert lib.llattn_mamba2_fwd_workspace_bytes(1, 524288, 1, 1, 128, 64, 20) > 0
    assert lib.llattn_mamba2_fwd_workspace_bytes(1, 524288 + 512, 1, 1, 128, 64, 21) == 0
    null = ctypes.c_void_p(0)
    assert lib.llattn_mamba2_fwd(*([null] * 8), 0, 1, 1048576, 1, 1, 128, 64, 21, null) == -1


def test_bf16_only(lib):
    """fp32 q / k / v never reach a kernel: the Python driver refuses them (no fp32 mode; no CPU path either)."""
    import torch
    from hattention_b200.base import HType
    from hattention_b200.chunkwise import _check
    q = torch.zeros(1, 64, 1, 128)
    v = torch.zeros(1, 64, 2, 64)
    g = torch.zeros(1, 64, 2)
    l = torch.zeros(1, 64, 2, 7)
    with pytest.raises((NotImplementedError, RuntimeError)):
        _check(q, q, v, g, l, False, 2, HType.WEAK, 64)


def test_workspace_sizes(lib):
    # one segment (T <= 512): only the 256-byte status word
    assert lib.llattn_mamba2_fwd_workspace_bytes(1, 512, 2, 1, 128, 64, 10) == 256
    small = lib.llattn_mamba2_fwd_workspace_bytes(1, 1024, 2, 1, 128, 64, 11)
    big = lib.llattn_mamba2_fwd_workspace_bytes(2, 16384, 32, 1, 128, 64, 15)
    assert 0 < small < big
    assert lib.llattn_mamba2_bwd_workspace_bytes(2, 16384, 32, 1, 128, 64, 15) > big
    # rejected shapes size to zero
    assert lib.llattn_mamba2_fwd_workspace_bytes(1, 100, 2, 1, 128, 64, 10) == 0


@pytest.mark.parametrize("T,K", [(512, 128), (576, 64), (576, 128), (4096, 64), (4096, 128)])
def test_backward_workspace_has_tiles_for_the_tensor_core_kernels_only(lib, T, K):
    """Calls that take the warp-level kernels (more than twenty lambda levels; layers of an odd number of chunks or with K = 64) read neither the level states
    inside a single segment nor the gradients of the pairs' summaries: their workspace does without those tiles."""
    B, H = 2, 3
    need = lambda L: lib.llattn_mamba2_bwd_workspace_bytes(B, T, H, 1, K, 64, L)
    layer = lambda L: lib.llattn_mamba2_bwd_layer_workspace_bytes(B, T, H, 1, K, 64, L)
    tiles = (2 if T <= 512 else 1) * B * H * -(-T // 128) * K * 64 * 2
    assert need(20) - need(21) == tiles
    assert need(21) == need(32) == layer(21)
    assert layer(20) == (need(21) if K == 64 or (T // 64) % 2 else need(20))


@pytest.mark.parametrize("shape,code", [
    ((1, 100, 2, 1, 128, 64, 10), -2),     # T % 64
    ((1, 1024, 3, 2, 128, 64, 12), -4),    # H % G
    ((1, 1024, 2, 1, 96, 64, 12), -1),     # K
    ((1, 1024, 2, 1, 128, 32, 12), -1),    # V
    ((1, 1024, 2, 1, 128, 64, 10), -3),    # L < 7 + log2(16)
    ((1, 1024, 2, 1, 128, 64, 40), -1),    # L > 32
])
def test_bad_arguments_are_rejected_without_a_device(lib, shape, code):
    null = ctypes.c_void_p(0)
    rc = lib.llattn_mamba2_fwd(null, null, null, null, null, null, null, null, 0, *shape, null)
    assert rc == code
    rc = lib.llattn_mamba2_bwd(*([null] * 11), null, 0, *shape, null)
    assert rc == code


def test_null_pointers_are_rejected(lib):
    null = ctypes.c_void_p(0)
    assert lib.llattn_mamba2_fwd(null, null, null, null, null, null, null, null, 0, 1, 512, 2, 1, 128, 64, 10, null) == -6


def test_python_wrappers_refuse_cpu_tensors():
    import torch
    from hattention_b200 import HStruct, HType, hattention_kernel
    q = torch.zeros(1, 64, 1, 64, dtype=torch.bfloat16)
    v = torch.zeros(1, 64, 2, 64, dtype=torch.bfloat16)
    g = torch.zeros(1, 64, 2)
    l = torch.zeros(1, 64, 2, 7, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        hattention_kernel(q, q, v, None, g, l, None, False, 2, HType.WEAK, HStruct.MAMBA2)
    with pytest.raises(NotImplementedError):
        hattention_kernel(q, q, v, None, g, l, None, True, 2, HType.WEAK, HStruct.MAMBA2)
    with pytest.raises(ValueError):
        hattention_kernel(q, q, v, g, g, l, None, False, 2, HType.WEAK, HStruct.MAMBA2)


def test_gdn_entry_points_reject_bad_arguments(lib):
    null = ctypes.c_void_p(0)
    # K must be 128, V 64 or 128, at most eight inter-chunk levels
    assert lib.llattn_gdn_fwd_workspace_bytes(1, 1024, 2, 96, 64, 12) == 0
    assert lib.llattn_gdn_fwd_workspace_bytes(1, 1024, 2, 128, 256, 12) == 0
    assert lib.llattn_gdn_fwd_workspace_bytes(1, 32768, 2, 128, 64, 16) == 0
    fwd = lib.llattn_gdn_fwd_workspace_bytes(1, 1024, 2, 128, 128, 11)
    lev = lib.llattn_gdn_bwd_levels_workspace_bytes(1, 1024, 2, 128, 128, 11)
    bwd = lib.llattn_gdn_bwd_workspace_bytes(1, 1024, 2, 128, 128, 11)
    assert 0 < fwd < lev < bwd
    assert lib.llattn_gdn_fwd(*([null] * 10), null, 0, 1, 1000, 2, 128, 64, 11, null) == -2
    assert lib.llattn_gdn_fwd(*([null] * 10), null, 0, 1, 1024, 2, 128, 64, 10, null) == -3
    assert lib.llattn_gdn_fwd(*([null] * 10), null, 0, 1, 1024, 2, 128, 64, 11, null) == -6
    assert lib.llattn_gdn_bwd(*([null] * 15), null, 0, 1, 1024, 2, 64, 64, 11, null) == -1
    assert lib.llattn_gdn_bwd(*([null] * 15), null, 0, 1, 1024, 2, 128, 64, 11, null) == -6
    assert lib.llattn_gdn_bwd_levels(*([null] * 15), null, 0, 1, 1024, 2, 128, 64, 11, null) == -6
    # forward that keeps its intermediates / backward that reads them
    keep = lib.llattn_gdn_fwd_keep_workspace_bytes(1, 1024, 2, 128, 128, 11)
    bkept = lib.llattn_gdn_bwd_kept_workspace_bytes(1, 1024, 2, 128, 128, 11)
    assert keep > fwd and 0 < bkept < bwd and keep + bkept >= bwd
    assert lib.llattn_gdn_fwd_keep_workspace_bytes(1, 1024, 2, 96, 64, 12) == 0
    assert lib.llattn_gdn_fwd_keep(*([null] * 10), null, 0, 1, 1024, 2, 128, 64, 11, null) == -6
    assert lib.llattn_gdn_bwd_kept(*([null] * 15), null, 0, null, 0, 1, 1024, 2, 128, 64, 11, null) == -6
    assert lib.llattn_gdn_bwd_kept_bf16dv(*([null] * 15), null, 0, null, 0, 1, 1024, 2, 128, 64, 11, null) == -6


def test_elementwise_entry_points_reject_bad_arguments(lib):
    null = ctypes.c_void_p(0)
    assert lib.llattn_l2norm_fwd(null, null, 10, 128, 1.0, null) == -6
    assert lib.llattn_l2norm_fwd(null, null, 10, 100, 1.0, null) == -1          # D % 8
    assert lib.llattn_l2norm_bwd(null, null, null, 10, 512, 1.0, null) == -1     # D > 256
    assert lib.llattn_mamba2_prep_fwd(*([null] * 9), 64, 2, 64, 12, 7, null) == -1     # lambda mode
    assert lib.llattn_mamba2_prep_fwd(*([null] * 9), 63, 2, 64, 12, 0, null) == -1     # rows % H
    assert lib.llattn_mamba2_prep_fwd(*([null] * 9), 64, 2, 64, 12, 0, null) == -6
    assert lib.llattn_mamba2_prep_bwd(*([null] * 18), 64, 2, 60, 12, 0, null) == -1    # P % 8
    assert lib.llattn_mamba2_residual(null, null, null, null, 0, 64, 2, 64, null) == -6


def test_prefill_and_step_entry_points_reject_bad_arguments(lib):
    null = ctypes.c_void_p(0)
    assert lib.llattn_mamba2_final_state(null, null, null, null, 1, 1000, 2, 1, 128, 64, 8, null) == -3    # 1000 tokens need 11 levels
    assert lib.llattn_mamba2_final_state(null, null, null, null, 1, 1000, 2, 1, 128, 64, 11, null) == -6
    assert lib.llattn_mamba2_final_state(null, null, null, null, 1, 1000, 3, 2, 128, 64, 11, null) == -1
    assert lib.llattn_mamba2_step(*([null] * 7), 1, 2, 1, 128, 64, 11, 11, null) == -3                    # carry level out of range
    assert lib.llattn_mamba2_step(*([null] * 7), 1, 2, 1, 128, 48, 11, 0, null) == -1                     # 256 % V
    assert lib.llattn_mamba2_step(*([null] * 7), 1, 2, 1, 128, 64, 11, 0, null) == -6


def test_decode_state_counts_follow_the_cascade():
    """Host-side token counts of the decode state: after T tokens they are the binary decomposition of
    T - 1 plus the newest token, whether reached by stepping the cascade or set directly."""
    import torch
    from hattention_b200 import HState, HStruct, HType
    for T in (1, 2, 3, 64, 65, 200, 255, 256, 1000):
        hs = HState(2, HType.WEAK, HStruct.MAMBA2, (1, 1, 1, 1, 12), torch.float32, torch.device("cpu"))
        for _ in range(T):
            hs.cascade_counts()
            hs.counts[0] += 1
        ref = HState(2, HType.WEAK, HStruct.MAMBA2, (1, 1, 1, 1, 12), torch.float32, torch.device("cpu"))
        ref.set_counts_after(T)
        assert hs.counts == ref.counts, T
        assert sum(hs.counts) == T


def test_misaligned_pointers_are_refused(lib):
    """Pointers between the boundaries of the vector accesses come back as an error code before anything touches a device."""
    P, I, F, Z = ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_size_t
    ok, odd, null = P(4096), P(4098), P(0)

    def call(name, *args):
        fn = getattr(lib, name)
        old = fn.argtypes
        fn.argtypes = None
        try:
            return fn(*args)
        finally:
            fn.argtypes = old

    step = [I(x) for x in (1, 2, 1, 128, 64, 9)]
    assert call("llattn_mamba2_layer_step", odd, ok, ok, ok, null, ok, ok, null, I(0), null, I(0), null, I(0), null, ok, *step, ctypes.c_uint(1), I(0), I(2), I(0),
                I(0), null) == -9
    assert call("llattn_gdn_layer_step", ok, ok, ok, odd, ok, ok, ok, ok, *step, ctypes.c_uint(1), I(0), I(1), F(1), F(0), I(0), null) == -9
    rows = [ctypes.c_long(64), I(2), I(64), I(9), I(0), null]
    assert call("llattn_mamba2_layer_prep_fwd", odd, ok, ok, I(0), ok, ok, ok, I(0), ok, ok, ok, *rows) == -9
    assert call("llattn_mamba2_layer_prep_bwd", ok, ok, ok, I(0), ok, ok, ok, I(0), null, I(0), ok, ok, ok, null, odd, ok, ok, ok, ok, ok, null, *rows) == -9
    mixer = [I(x) for x in (1, 64, 2, 1, 128, 9, 0)] + [null]
    assert call("llattn_mixer_prep_fwd", odd, ok, I(0), ok, I(0), ok, I(0), ok, ok, I(0), *[ok] * 6, *mixer) == -9
    assert call("llattn_mixer_prep_bwd", ok, ok, I(0), ok, I(0), ok, I(0), ok, ok, I(0), null, I(0), ok, null, ok, ok, ok, ok, odd, *[ok] * 5, *mixer) == -9
    norm = [ctypes.c_long(64), I(2)]
    assert call("llattn_mixer_norm_fwd", ok, ok, null, I(0), odd, I(400), ok, I(0), ok, ok, *norm, F(1e-6), null) == -9
    assert call("llattn_mixer_norm_bwd", ok, ok, null, I(0), ok, I(400), ok, I(0), odd, ok, ok, ok, ok, null, *norm, null) == -9
    assert call("llattn_mamba2_prompt_prep", odd, ok, null, I(0), ok, ok, ok, I(0), ok, ok, ok, ok, ok, null, null, *[I(x) for x in (1, 64, 3, 2, 1, 128, 64, 9, 0)],
                null) == -9
    assert call("llattn_mamba2_prompt_tail", odd, ok, ok, ok, ok, null, null, I(0), ok, ok, I(9), ok, *[I(x) for x in (1, 64, 3, 2, 1, 128, 64, 9)], null) == -9
    assert call("llattn_gdn_prompt_prep", ok, odd, ok, ok, ok, ok, ok, ok, null, null, null, null, *[I(x) for x in (1, 64, 3, 2, 2, 128, 128, 128, 1, 9)], F(1), F(0),
                null) == -9
    assert call("llattn_gdn_grad_out", odd, ok, ok, ok, ok, ok, null, ok, ok, ok, ok, null, ctypes.c_long(64), *[I(x) for x in (1, 128, 128, 9)], F(1), F(0), null) == -9
    assert call("llattn_l2norm_fwd", odd, ok, ctypes.c_long(64), I(128), F(1), null) == -9
    shape = [I(x) for x in (1, 64, 2, 1, 128, 64, 9)]
    assert call("llattn_mamba2_fwd", odd, ok, ok, ok, ok, ok, ok, ok, Z(1 << 30), *shape, null) == -9
    assert call("llattn_mamba2_bwd_saved", ok, ok, ok, ok, ok, odd, *[ok] * 6, Z(1 << 30), null, Z(0), *shape, null) == -9


def test_static_scratch_serves_narrow_states_and_odd_chunk_counts(lib):
    """The state part of the scratch goes with the state width: 0.8 MiB per (batch, head) at T = 4096, K = 64, so 19 of them fit; and 97 of 9 chunks at
    K = 128 do without the half pair of partial outputs.  Beyond that the call is refused before a device is touched."""
    need = lambda K, T, bh: lib.llattn_mamba2_fwd_workspace_bytes(1, T, bh, 1, K, 64, 13)
    # states: NS summaries in fp32 and NS LH level states in bf16; partial outputs: bf16 rows
    per = lambda K, T: (lambda NS, LH: NS * K * 64 * 4 + NS * LH * K * 64 * 2 + NS * 4)(-(-T // 512), max(0, (-(-T // 512) - 1).bit_length())) + T * 128
    for K in (64, 128):
        assert abs(need(K, 4096, 8) - 8 * per(K, 4096)) < 2048
    assert need(64, 4096, 19) <= lib.llattn_static_scratch_bytes() < need(64, 4096, 20)
    null, dummy = ctypes.c_void_p(0), ctypes.c_void_p(4096)
    static = lambda K, T, bh: lib.llattn_mamba2_fwd_static(*([null] + [dummy] * 6), 1, T, bh, 1, K, 64, 13, null)
    import torch
    if torch.cuda.is_available():
        return                                        # a call that is not refused would launch
    run = lambda K, T, bh: lib.llattn_mamba2_fwd_static(*([dummy] * 7), 1, T, bh, 1, K, 64, 13, null)
    assert static(64, 4096, 19) == -6
    assert run(64, 4096, 20) == -7 and run(128, 576, 98) == -7
    assert run(64, 4096, 19) > 0 and run(128, 576, 97) > 0      # no device here: a CUDA error code, not a refusal
