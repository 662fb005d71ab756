"""Decode-time level states, with the interface of the reference's `hattention/recurrent.py`
(`HState` :9-131).  The token recurrence itself (`step_state` / `step_output` :134-166) runs in one CUDA
kernel behind `hattention_b200.kernel.hattention_step`."""
import torch

from .base import HStruct, HType


def is_level_major(states: torch.Tensor) -> bool:
    """Whether a (B,H,K,V,L) tensor is stored (B,H,L,K,V): one contiguous K x V block per level of a head, at the 16-byte boundary that
    the kernels for that layout need."""
    B, H, K, V, L = states.shape
    return states.stride() == (H * L * K * V, L * K * V, V, 1, K * V) and (not states.is_cuda or states.data_ptr() % 16 == 0)


def level_major_states(shape, device, dtype=torch.float32, zero=False) -> torch.Tensor:
    """An (uninitialised) (B,H,K,V,L) tensor stored (B,H,L,K,V)."""
    B, H, K, V, L = shape
    make = torch.zeros if zero else torch.empty
    return make((B, H, L, K, V), dtype=dtype, device=device).permute(0, 1, 3, 4, 2)


def _zero_states(shape, dtype, device) -> torch.Tensor:
    # level-major where the decode kernels for that layout take the value width: they move only the levels that hold tokens
    if len(shape) == 5 and shape[3] % 16 == 0 and torch.device(device).type == "cuda":
        return level_major_states(shape, device, dtype, zero=True)
    return torch.zeros(shape, dtype=dtype, device=device)


class HState:
    """Level states of one layer for decoding, with the fields of the reference's `HState`
    (hattention/recurrent.py:9-131): `states` (B,H,K,V,L) in `dtype` and one token count per level.
    The counts are identical for every sequence and are kept on the host, so that the cascade
    (recurrent.py:42-54) costs no device synchronisation."""

    def __init__(self, base: int, htype: HType, hstruct: HStruct, shape, dtype: torch.dtype, device) -> None:
        if base != 2 or htype != HType.WEAK:
            raise NotImplementedError
        self.base, self.htype, self.hstruct = base, htype, hstruct
        self.shape, self.dtype, self.device = tuple(shape), dtype, device
        self.max_num_levels = self.shape[-1]
        self.states = _zero_states(self.shape, dtype, device)
        self.counts = [0] * self.max_num_levels

    @classmethod
    def holding(cls, states: torch.Tensor, base: int, htype: HType, hstruct: HStruct) -> "HState":
        """A state around an existing tensor (B,H,K,V,L), which is adopted as it is; the counts start at zero."""
        self = cls.__new__(cls)
        self.base, self.htype, self.hstruct = base, htype, hstruct
        self.shape, self.dtype, self.device = tuple(states.shape), states.dtype, states.device
        self.max_num_levels = self.shape[-1]
        self.states = states
        self.counts = [0] * self.max_num_levels
        return self

    def live_levels(self) -> int:
        """Bit l is set when level l holds tokens."""
        live = 0
        for level, count in enumerate(self.counts):
            if count:
                live |= 1 << level
        return live

    def cascade_counts(self) -> int:
        """Runs the cascade on the counts; returns the level that receives the merged levels."""
        for level in range(self.max_num_levels):
            cap = 1 << level
            if self.counts[level] == cap:
                if level + 1 >= self.max_num_levels:
                    raise ValueError("more tokens than the levels can hold")
                self.counts[level + 1] += self.counts[level]
                self.counts[level] = 0
            elif self.counts[level] < cap:
                return level
            else:
                raise ValueError
        return self.max_num_levels - 1

    def set_counts_after(self, T: int) -> None:
        """Counts after T tokens: level 0 holds the last token, level j+1 holds 2^j tokens for each set
        bit j of T-1 (the bookkeeping at the end of kernel.py:452-463)."""
        self.counts = [0] * self.max_num_levels
        if T <= 0:
            return
        self.counts[0] = 1
        m = T - 1
        for j in range(m.bit_length()):
            if (m >> j) & 1:
                if j + 1 >= self.max_num_levels:
                    raise ValueError("more tokens than the levels can hold")
                self.counts[j + 1] = 1 << j

    def set_counts_before(self, t: int) -> None:
        """Counts as the cascade leaves them just before token t (0-based) is inserted: level 0 empty, level j+1
        holds 2^j tokens for each set bit j of t."""
        self.counts = [0] * self.max_num_levels
        for j in range(max(t, 0).bit_length()):
            if (t >> j) & 1:
                if j + 1 >= self.max_num_levels:
                    raise ValueError("more tokens than the levels can hold")
                self.counts[j + 1] = 1 << j

    def reset_states(self) -> None:
        """recurrent.py:102-103; the token counts restart with the states."""
        self.states = _zero_states(self.shape, self.dtype, self.device)
        self.counts = [0] * self.max_num_levels

    def replace(self, other: "HState") -> None:
        """Adopt another state of the same shape (recurrent.py:105-115), token counts included: the cascade
        of the next decode step depends on them."""
        if not (tuple(self.shape) == tuple(other.shape) and self.base == other.base and self.htype == other.htype
                and self.dtype == other.dtype and torch.device(self.device) == torch.device(other.device)):
            raise ValueError("Shape, dtype or device mismatch")
        self.states = other.states
        self.counts = list(other.counts)

    def to(self, dtype=None, device=None) -> "HState":
        """recurrent.py:117-131.  The states stay fp32 (the decode kernel reads fp32 states and casts its
        output), so only fp32 / the same device is a no-op copy; other targets are not supported."""
        if (dtype is not None and dtype != self.dtype) or (device is not None and torch.device(device) != torch.device(self.device)):
            raise NotImplementedError("level states are kept in fp32 on their device")
        new = HState(self.base, self.htype, self.hstruct, self.shape, self.dtype, self.device)
        new.states = self.states
        new.counts = list(self.counts)
        return new
