"""Token selection for the rows of one step.

Same knobs and meanings as the reference's ``GenerationParams`` and ``StochasticSampler``
(pulsar-core/inc/pulsar/runtime/sampler.hpp:21-40; pulsar-core/src/runtime/sampler.cpp:12-57):
temperature <= 0 is exact greedy on the raw logits and leaves the generator untouched;
otherwise softmax(logits / temperature), top_k > 0 keeps the k most probable, top_p in
(0, 1) keeps a token while the mass before it is <= top_p, both give the intersection;
seed >= 0 makes a request reproducible, seed < 0 draws a fresh seed.

The reference samples one row at a time with a device-to-host read each.  Here a few
kernels handle all rows of the step (many blocks per row) and the chosen ids stay on the
device for the next step or come back in one copy; the uniform number of each stochastic
row comes from that request's own host generator, so a request's tokens do not depend on
what else is in the batch.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import List, Optional, Sequence

import torch

from .. import ops

_MAX_TOP_K = 2 ** 31 - 1           # the kernels count in 32 bits


@dataclass
class GenerationParams:
    temperature: float = 0.0
    top_p: float = 1.0
    top_k: int = 0
    seed: int = -1

    def validate(self) -> None:
        if not (0.0 < self.top_p <= 1.0):
            raise ValueError(f"top_p must lie in (0, 1], found {self.top_p}")
        if self.top_k < 0:
            raise ValueError(f"top_k must be >= 0, found {self.top_k}")
        if not self.greedy and not self.top_k <= _MAX_TOP_K:
            raise ValueError(f"top_k must be at most {_MAX_TOP_K}, found {self.top_k}")

    @property
    def greedy(self) -> bool:
        return not (self.temperature > 0.0)

    def device_top_k(self) -> int:
        """``top_k`` as the kernels take it (a greedy row has no use for its own)."""
        k = int(self.top_k) if self.temperature > 0.0 else 0
        if not -_MAX_TOP_K - 1 <= k <= _MAX_TOP_K:
            raise ValueError(f"top_k must be at most {_MAX_TOP_K}, found {self.top_k}")
        return k


def make_generator(seed: int) -> torch.Generator:
    """Per-request generator: seed >= 0 reproducible, seed < 0 nondeterministic
    (pulsar-core/src/runtime/sampler.cpp:48-57)."""
    g = torch.Generator(device="cpu")
    if seed >= 0:
        g.manual_seed(int(seed))
    else:
        g.seed()
    return g


def draw_uniform(generator: torch.Generator) -> float:
    return torch.rand(1, generator=generator).item()


class Sampler:
    HEAD = 8

    def __init__(self, device):
        self.device = torch.device(device)
        # [HEAD words for whoever reads the ids back | the ids]: one copy brings both
        self._report = torch.zeros(self.HEAD + 64, dtype=torch.int32, device=self.device)
        self.last_ids: Optional[torch.Tensor] = None      # what the last call returned
        # The rows' parameters travel in one copy from pinned memory, one buffer for each of the last calls: (the memory, the same
        # as C floats and as C ints).
        self._staging: List[Optional[tuple]] = [None] * 4
        self._staging_next = 0

    def report(self, rows: int) -> torch.Tensor:
        """The head words and the ids of the last call's ``rows`` rows, on the device."""
        return self._report[:self.HEAD + rows]

    @property
    def head(self) -> torch.Tensor:
        return self._report[:self.HEAD]

    def _on_device(self, params: Sequence[GenerationParams], uniform: List[float]) -> torch.Tensor:
        """float32 [4, rows] on the device: temperatures, top_p, uniform numbers, and the bits of the int32 top_k."""
        rows, i = len(params), self._staging_next
        self._staging_next = (i + 1) % len(self._staging)
        slot = self._staging[i]
        if slot is not None:
            slot[0].wait()                        # the copy out of this buffer, some calls ago
        if slot is None or slot[0].host.numel() < 4 * rows:
            buf = ops.Pinned(4 * max(rows, 64), torch.float32)
            at, n = buf.host.data_ptr(), buf.host.numel()
            slot = self._staging[i] = (buf, (ctypes.c_float * n).from_address(at), (ctypes.c_int * n).from_address(at))
        buf, floats, ints = slot
        floats[:3 * rows] = [p.temperature for p in params] + [p.top_p for p in params] + uniform
        ints[3 * rows:4 * rows] = [p.device_top_k() for p in params]
        out = torch.empty((4, rows), dtype=torch.float32, device=self.device)
        buf.to_device(out, 4 * rows)
        return out

    def sample_on_device(self, logits: torch.Tensor, params: Sequence[GenerationParams],
                         generators: Sequence[Optional[torch.Generator]], uniform: Optional[List[float]] = None) -> torch.Tensor:
        """One token id per row of ``logits`` (float32 [R, V] on the device), left on the device:
        an int32 tensor that stays valid until the next call.  ``uniform``: the rows' uniform numbers (0.0 for greedy rows), where
        the caller has drawn them already."""
        rows = logits.shape[0]
        assert len(params) == rows and (len(generators) == rows if uniform is None else len(uniform) == rows)
        if self._report.numel() < self.HEAD + rows:
            self._report = torch.zeros(self.HEAD + rows, dtype=torch.int32, device=self.device)
        out = self._report[self.HEAD:self.HEAD + rows]
        self.last_ids = out
        if rows == 0:
            return out
        if all(p.greedy for p in params):
            ops.sample(logits, out)
        else:
            if uniform is None:
                uniform = [0.0 if p.greedy else draw_uniform(g) for p, g in zip(params, generators)]
            temperature, top_p, drawn, top_k = self._on_device(params, uniform).unbind(0)
            ops.sample(logits, out, temperature, top_k.view(torch.int32), top_p, drawn, any_greedy=any(p.greedy for p in params))
        return out

    def sample(self, logits: torch.Tensor, params: Sequence[GenerationParams],
               generators: Sequence[Optional[torch.Generator]]) -> List[int]:
        """One token id per row of ``logits``, read back to the host."""
        if logits.shape[0] == 0:
            return []
        return self.sample_on_device(logits, params, generators).tolist()
