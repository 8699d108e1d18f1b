"""Sampling of next tokens on the device.

Greedy (temperature <= 0): argmax with ties to the lowest id.  Otherwise
temperature and nucleus (top-p) sampling as LockStep defines it
(engine/sampler/philox.py:71-98): softmax(logits / T), rank by (-p, id), keep
the shortest head whose mass reaches top_p, inverse CDF over the head with the
Philox draw for (seed, uid, position).
"""

from __future__ import annotations

import functools
from dataclasses import dataclass

import torch

from .. import kernels as K
from . import philox


@dataclass
class SamplingParams:
    uid: str
    seed: int = 0
    temperature: float = 0.0
    top_p: float = 1.0
    position: int = 0        # position of the last context token


class Sampler:
    def __init__(self, device):
        self.device = torch.device(device)
        self._probs = None
        self._host = None                     # pinned: one row of parameters a request, copied in one go
        self._copied = None                   # the last copy out of it

    def sample(self, logits: torch.Tensor, params: list[SamplingParams]) -> list[int]:
        """One token per row of ``logits`` [rows, vocab] (float32, on the device)."""
        if logits.shape[0] == 0:
            return []
        return self.sample_device(logits, params).tolist()

    def sample_device(self, logits: torch.Tensor, params: list[SamplingParams]) -> torch.Tensor:
        """As ``sample``, but the tokens stay on the device (int32 [rows])."""
        rows, vocab = logits.shape
        if rows != len(params):
            raise ValueError("one SamplingParams per row of logits")
        out = torch.empty(rows, dtype=torch.int32, device=self.device)
        if rows == 0:
            return out
        temperatures = [p.temperature for p in params]
        if all(t <= 0 for t in temperatures):
            K.argmax(logits, out)
            return out
        top_ps = [p.top_p for p in params]
        for p, t, top in zip(params, temperatures, top_ps):
            if t > 0 and not 0 < top <= 1:
                raise ValueError(f"{p.uid}: top_p must lie in (0, 1], got {top}")
        # keys, positions, temperatures and nucleus sizes in one pinned buffer and one copy
        if self._host is None or self._host.numel() < 6 * rows:
            self._host = torch.empty(6 * max(rows, 64), dtype=torch.int32).pin_memory()
            self._copied = torch.cuda.Event()
        else:
            self._copied.synchronize()        # the copy before this one has read the buffer
        host = self._host[:6 * rows]
        words = host.numpy()
        pairs, reals = words[:4 * rows].view("uint64"), words.view("float32")      # low word first
        pairs[:rows] = [_key(p.seed, p.uid) for p in params]
        pairs[rows:] = [p.position & 0xFFFFFFFFFFFFFFFF for p in params]
        reals[4 * rows:5 * rows] = [max(0.0, t) for t in temperatures]
        reals[5 * rows:] = top_ps
        dev = host.to(self.device, non_blocking=True)
        self._copied.record()
        keys, positions = dev[:2 * rows].view(rows, 2), dev[2 * rows:4 * rows].view(rows, 2)
        temperature, top_p = dev[4 * rows:5 * rows].view(torch.float32), dev[5 * rows:].view(torch.float32)
        need = K.sample_scratch_floats(rows, vocab)
        if need and (self._probs is None or self._probs.numel() < need):
            self._probs = torch.empty(need, dtype=torch.float32, device=self.device)
        K.sample(logits, self._probs if need else None, temperature, top_p, keys, positions, out)
        return out


@functools.lru_cache(maxsize=4096)
def _key(seed: int, uid: str) -> int:
    low, high = philox.key_words(seed, uid)
    return low | high << 32
