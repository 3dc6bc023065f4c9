"""Token selection on the device.

A batch whose rows are all greedy takes the argmax kernel (ties to the lowest
index, as ``logits.argmax`` in ``src/einf/executors/torch/sampler.py:31-32``);
otherwise one kernel filters and draws every row from its own parameters and a
uniform number keyed by ``(seed, sample_index)``, so a request's tokens do not
depend on the batch it shares (``sampler.py:93-94`` seeds a generator per row
for the same reason).
"""
from __future__ import annotations

from typing import Sequence

import numpy as np
import torch

from .. import ops
from ..cache.control import pack_sampling


class Sampler:
    def __init__(self, device: torch.device | str, max_rows: int) -> None:
        self.device = torch.device(device)
        self.max_rows = max_rows
        self.tokens = torch.zeros(max_rows, dtype=torch.int32, device=self.device)
        pin = self.device.type == "cuda"
        # A row's parameters lie in one buffer, so that a step copies once: [seed, sample_index] as int64,
        # [temperature, top_p, min_p] as float32, [top_k] as int32.
        # The copy to the device is asynchronous and a caller may sample several steps before it
        # waits for the device, so the pinned staging is a ring: a slot is written again only after
        # the copy that read it last has run (its event).
        self._ring = 8
        self._turn = 0
        self._events = [None] * self._ring
        staging = torch.zeros((self._ring, 32 * max_rows), dtype=torch.uint8, pin_memory=pin)
        self._host, self._staging = staging.unbind(0), staging.numpy()
        self._dev = torch.zeros(32 * max_rows, dtype=torch.uint8, device=self.device)
        n = max_rows
        wide, real = self._dev[:16 * n].view(torch.int64), self._dev[16 * n:28 * n].view(torch.float32)
        self._columns = (real[:n], self._dev[28 * n:].view(torch.int32), real[n:2 * n], real[2 * n:], wide[:n], wide[n:])

    def sample(self, logits: torch.Tensor, params: Sequence, sample_indices: Sequence[int]) -> torch.Tensor:
        """One token per row of ``logits`` (float32 ``[rows, vocab]``); returns an
        int32 device tensor of ``rows`` tokens (a view of an internal buffer)."""
        rows = logits.shape[0]
        if rows != len(params) or rows != len(sample_indices):
            raise ValueError("one set of sampling parameters per logits row is needed")
        if rows > self.max_rows:
            raise ValueError(f"{rows} rows exceed the sampler's {self.max_rows}")
        if rows == 0:
            return self.tokens[:0]
        if all(p.temperature == 0 for p in params):
            ops.argmax(logits, self.tokens)
            return self.tokens[:rows]
        turn = self._turn
        self._turn = (turn + 1) % self._ring
        if self._events[turn] is not None:
            self._events[turn].synchronize()
        staging = self._host[turn]
        try:
            pack_sampling(params, sample_indices, staging.data_ptr(), self.max_rows)
        except TypeError:               # other objects with the same attributes, other collections than sequences
            self._pack(turn, params, sample_indices)
        self._dev.copy_(staging, non_blocking=True)
        if self.device.type == "cuda":
            if self._events[turn] is None:
                self._events[turn] = torch.cuda.Event()
            self._events[turn].record(ops.current_stream())
        ops.sample(logits, self.tokens, *self._columns)
        return self.tokens[:rows]

    def _pack(self, turn: int, params: Sequence, sample_indices: Sequence[int]) -> None:
        """What ``pack_sampling`` does, for any objects with the attributes of sampling parameters in any collections."""
        n, host = self.max_rows, self._staging[turn]
        wide, real = host[:16 * n].view(np.int64).reshape(2, n), host[16 * n:28 * n].view(np.float32).reshape(3, n)
        whole = host[28 * n:].view(np.int32)
        for r, (p, index) in enumerate(zip(params, sample_indices)):
            wide[0, r], wide[1, r] = np.int64(p.seed), index
            real[0, r], real[1, r], real[2, r] = p.temperature, p.top_p, p.min_p
            whole[r] = p.top_k or 0
