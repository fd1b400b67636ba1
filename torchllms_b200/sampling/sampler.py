"""Choosing next tokens for a batch of requests: greedy, temperature, optional top-k.

Reference: ``sample`` (torchllms/inference/utils.py:36-48): temperature 0 is argmax; otherwise
logits / max(T, 1e-5), optional top-k cut, softmax, and ``argmax(probs / Exp(1))``
(:18-33).  The reference draws its noise from PyTorch's global generator, so a request's sample
depends on what else is in the batch.  Here the noise of a row is a pure function of
(seed, request, index of the generated token), computed inside the kernel, so a request samples
the same tokens alone or batched, whole or in portions, before or after a pre-emption.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import List, Optional, Sequence

import numpy as np
import torch

from ..kernels.streams import current_stream

MASK64 = (1 << 64) - 1
GOLDEN = 0x9E3779B97F4A7C15


def mix64(z: int) -> int:
    """The 64-bit finaliser the sampling kernel uses (same constants, same shifts)."""
    z &= MASK64
    z ^= z >> 30
    z = (z * 0xBF58476D1CE4E5B9) & MASK64
    z ^= z >> 27
    z = (z * 0x94D049BB133111EB) & MASK64
    z ^= z >> 31
    return z


def row_key(seed: int, request: int, token_index: int) -> int:
    """Key of the noise for the ``token_index``-th generated token of ``request``."""
    return mix64((seed & MASK64) ^ mix64((request & MASK64) ^ mix64((token_index + GOLDEN) & MASK64)))


@dataclass
class SamplingParams:
    temperature: float = 0.0
    top_k: Optional[int] = None
    seed: int = 0


class PendingTokens:
    """Sampled tokens on their way to the host."""

    __slots__ = ("host", "done", "room")

    def __init__(self, host, done, room: Optional[torch.Tensor] = None):
        self.host, self.done, self.room = host, done, room      # room: the pinned buffer that ``host`` is the start of


class Sampler:
    ROOMS = 4

    def __init__(self, ops, device):
        self.ops = ops
        self.device = torch.device(device)
        # pinned buffers that are free again, with their events (allocating the two takes as long as the copy): at most
        # ROOMS, as many as steps in flight want
        self._rooms: List[tuple] = []

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], requests: Sequence[int],
               token_indices: Sequence[int]) -> List[int]:
        """One token per row of ``logits`` ``[n, vocab]`` (float32, on the device)."""
        return self.finish(self.launch(logits, params, requests, token_indices))

    def launch(self, logits: torch.Tensor, params: Sequence[SamplingParams], requests: Sequence[int],
               token_indices: Sequence[int]) -> torch.Tensor:
        """Start sampling and return the tokens as a device tensor without waiting for them:
        the caller may do host work before :meth:`finish` reads them back."""
        n = logits.shape[0]
        assert n == len(params) == len(requests) == len(token_indices)
        if all(not p.temperature > 0 for p in params):
            return self.ops.sample(logits)
        packed = np.zeros((n, 4), dtype=np.int32)  # temperature bits | top_k | key low | key high
        packed[:, 0] = np.asarray([p.temperature for p in params], dtype=np.float32).view(np.int32)
        packed[:, 1] = [int(p.top_k or 0) for p in params]
        keys = np.asarray([row_key(p.seed, r, t) for p, r, t in zip(params, requests, token_indices)], dtype=np.uint64)
        packed[:, 2:4] = keys.view(np.int32).reshape(n, 2)
        host = torch.from_numpy(packed)
        if self.device.type == "cuda":
            host = host.pin_memory()        # a copy from pageable memory would wait for the device
        dev = host.to(self.device, non_blocking=True)
        temperature = dev[:, 0].contiguous().view(torch.float32)
        # without a rank filter in the batch the kernel library may spread a row over many CTAs
        top_k = dev[:, 1].contiguous() if any((p.top_k or 0) > 0 for p in params) else None
        row_keys = dev[:, 2:4].contiguous().view(torch.int64).reshape(n)
        return self.ops.sample(logits, temperature, top_k, row_keys)

    def read_back(self, tokens: torch.Tensor) -> "PendingTokens":
        """Start copying the tokens of :meth:`launch` to the host.  Work queued on the device after
        this call does not delay :meth:`finish`, which waits for this copy alone."""
        if tokens.device.type != "cuda":
            return PendingTokens(tokens, None)
        n = tokens.numel()
        try:
            room, done = self._rooms.pop()
        except IndexError:
            room = None
        if room is None or room.numel() < n or room.dtype != tokens.dtype or tokens.dim() != 1:
            room, done = torch.empty(max(n, 64), dtype=tokens.dtype, pin_memory=True), torch.cuda.Event()
        host = room[:n].view(tokens.shape)
        host.copy_(tokens, non_blocking=True)
        done.record(current_stream())
        return PendingTokens(host, done, room)

    def finish(self, tokens) -> List[int]:
        """The tokens of :meth:`launch` (or of :meth:`read_back`) on the host; this waits for them."""
        if isinstance(tokens, PendingTokens):
            if isinstance(tokens.host, torch.Tensor):
                if tokens.done is not None:
                    tokens.done.synchronize()
                room, tokens.host = tokens.room, tokens.host.tolist()
                if room is not None and len(self._rooms) < self.ROOMS:
                    self._rooms.append((room, tokens.done))         # (read: nothing is on its way into it any more)
                tokens.room = tokens.done = None
            return self._checked(list(tokens.host))
        return self._checked(tokens.tolist())

    def _checked(self, tokens: List[int]) -> List[int]:
        # the device has finished everything up to the read-back: a kernel that gave up a wait has said so by now
        check = getattr(self.ops, "check_status", None)
        if check is not None:
            check()
        return tokens
