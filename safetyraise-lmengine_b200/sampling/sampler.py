"""Batch sampler over the logits a step returned: one kernel for all rows.

The random draw of a request's i-th generated token is a function of (seed, i)
alone, so the same seed gives the same tokens however the requests were batched,
cut or preempted.  The reference draws from ``rand::StdRng`` seeded per request
(src/frontend/sampling.rs:72-80); its bit stream is not reproduced, its
distribution and order of operations are.
"""
from __future__ import annotations

import os
from array import array
from itertools import chain
from typing import List, Sequence

import numpy as np
import torch

from ..cache.manager import runtime
from ..kernels import ops
from ..parts.base import FAULT_LOGITS, FAULT_TOKEN, STATUS_WORDS
from .params import SamplingParams

_MASK = (1 << 64) - 1
_LISTS = frozenset((list, tuple))


def _splitmix64(x: int) -> int:
    x = (x + 0x9E3779B97F4A7C15) & _MASK
    z = x
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _MASK
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _MASK
    return z ^ (z >> 31)


def uniform_for(seed: int, index: int) -> float:
    """A float32 in [0, 1) for the index-th draw of a request with this seed."""
    bits = _splitmix64(_splitmix64(seed & _MASK) ^ ((index + 1) * 0xD1B54A32D192ED03 & _MASK))
    return float(np.float32((bits >> 40) * (1.0 / (1 << 24))))


def fill_uniforms(seeds: Sequence[int], indices: Sequence[int], out: np.ndarray) -> None:
    """out[i] = uniform_for(seeds[i], indices[i]) (float32, contiguous) in one native call: two microseconds a pair in Python."""
    n = len(out)
    if len(seeds) != n or len(indices) != n:
        raise ValueError(f"{n} rows, {len(seeds)} seeds and {len(indices)} indices")
    try:
        pairs = array("Q", chain(seeds, indices))
    except OverflowError:                                     # negative, or more than 64 bits
        pairs = array("Q", [x & _MASK for x in chain(seeds, indices)])
    at = pairs.buffer_info()[0]
    runtime().srlm_sampling_uniforms(n, at, at + 8 * n, out.ctypes.data)


def fresh_seed() -> int:
    return int.from_bytes(os.urandom(8), "little")


class Sampler:
    """``status``: an engine's status buffer (int32: STATUS_WORDS fault words, then room for one token per
    request).  With it the sampled tokens are written behind the fault words and one read-back
    fetches both; a non-finite logit raises the word FAULT_LOGITS (src/frontend/sampling.rs:97-99).
    Without it the sampler keeps words of its own."""

    def __init__(self, device, vocab_size: int, max_rows: int = 64, status: torch.Tensor = None):
        self.device, self.vocab = device, vocab_size
        self._shared = status is not None
        self._status = status
        if status is None:
            self._status = torch.zeros(STATUS_WORDS + max_rows, dtype=torch.int32, device=device)
        self._words = STATUS_WORDS
        self.bad = self._status[FAULT_LOGITS:FAULT_LOGITS + 1]
        self.last_words = [0] * STATUS_WORDS      # the fault words as the last collect() read them
        self._cap = 0
        self._hosts, self._host_turn, self._dev = [], 0, None
        self._grow(max_rows)

    def _grow(self, rows: int):
        if rows <= self._cap:
            return
        if self._words + rows > self._status.numel():
            if self._shared:
                raise ValueError(f"{rows} rows to sample exceed the engine's {self._status.numel() - self._words}")
            old = self._status
            self._status = torch.zeros(self._words + rows, dtype=torch.int32, device=self.device)
            self._status[:self._words].copy_(old[:self._words])
            self.bad = self._status[FAULT_LOGITS:FAULT_LOGITS + 1]
        self._cap = rows
        self._out = self._status[self._words:self._words + rows]
        self._scratch = None               # [rows, vocab] float32, made when a row is first sampled

    def _buffer(self, words: int):
        """A pinned buffer of at least ``words`` 32-bit words, one of three taken in turn (a launch may be queued while the
        copy of the launch before it has not run yet), once the event behind its last copy has passed."""
        if not self._hosts or self._hosts[0][0].numel() < words:
            cap = max(words, 4096, 2 * self._hosts[0][0].numel() if self._hosts else 0)
            self._hosts = [[torch.empty(cap, dtype=torch.int32, pin_memory=True), torch.cuda.Event(), False] for _ in range(3)]
            self._dev = torch.empty(cap, dtype=torch.int32, device=self.device)
        self._host_turn = (self._host_turn + 1) % len(self._hosts)
        turn = self._hosts[self._host_turn]
        if turn[2]:
            turn[1].synchronize()
        return turn

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               indices: Sequence[int], histories: Sequence[Sequence[int]]) -> List[int]:
        """logits [n, V] float32 on the device; one token id per row, as Python ints."""
        return self.collect(self.launch(logits, params, seeds, indices, histories))

    def collect(self, n) -> List[int]:
        """The tokens of the last launch(): waits for the device and reads them back, the fault words
        with them (``last_words``; the caller decides what a raised word means).  ``n``: the number of
        rows that launch() returned, or what snapshot() returned for them."""
        if isinstance(n, tuple):
            host, event, rows = n
            event.synchronize()
            got = host[:self._words + rows].tolist()
        else:
            got = self._status[:self._words + n].tolist()
        self.last_words = got[:self._words]
        return got[self._words:]

    def snapshot(self, n: int):
        """Copies the fault words and the ``n`` tokens of the last launch() to pinned host memory behind
        what the stream holds so far, so that collect() of the returned handle waits for that copy alone
        and further work may be queued behind it meanwhile (it may overwrite the words and the tokens).
        At most two handles are alive at a time."""
        ring = self.__dict__.setdefault("_snapshots", [])
        need = self._words + self._cap
        if not ring or ring[0].numel() < need:
            ring[:] = [torch.empty(need, dtype=torch.int32, pin_memory=True) for _ in range(3)]
        self._snapshot_turn = (getattr(self, "_snapshot_turn", 0) + 1) % len(ring)
        host = ring[self._snapshot_turn]
        host[:self._words + n].copy_(self._status[:self._words + n], non_blocking=True)
        event = torch.cuda.Event()
        event.record()
        return host, event, n

    def clear_words(self) -> None:
        self._status[:self._words].zero_()
        self.last_words = [0] * self._words

    def launch(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               indices: Sequence[int], histories: Sequence[Sequence[int]], pending=None) -> int:
        """Starts the sampling kernel for the rows of ``logits``; returns the number of rows.  The host
        does not wait: collect() does.

        pending: per row, None or the row of the launch before this one whose token (still on the device,
        behind the fault words) is the last of this row's history: a repetition penalty counts it, the
        device puts it in place."""
        n = logits.shape[0]
        if n == 0:
            return 0
        self._grow(n)
        if all(p.is_greedy for p in params):
            ops.argmax(logits, self._out[:n], self.bad)
            return n
        # All that the rows bring goes through one pinned buffer and one asynchronous copy (a pageable copy would make the host
        # wait for the forward that is still running on the device), as 32-bit words: five parameters a row, each n words;
        # with a penalty the rows' offsets and ids, and the pairs of patch_words behind them.
        temperatures, penalties = [p.temperature for p in params], [p.repetition_penalty for p in params]
        penalised = [x != 1.0 for x in penalties]
        words, late, total = 5 * n, [], 0
        if any(penalised):
            late = [on and pending is not None and pending[i] is not None for i, on in enumerate(penalised)]
            lens = [len(ids) + behind if on else 0 for on, ids, behind in zip(penalised, histories, late)]
            total = sum(lens)
            words += n + 1 + max(total, 1) + 2 * sum(late)
        turn = self._buffer(words)
        host = turn[0].numpy()
        h = host[:4 * n].view(np.float32)
        h[:3 * n] = temperatures + [p.top_p for p in params] + penalties
        uniforms = h[3 * n:]
        if min(temperatures) > 0 and len(seeds) == n == len(indices):
            fill_uniforms(seeds, indices, uniforms)
        else:                                                 # the seeds of rows without a temperature are not read
            drawn = [i for i, t in enumerate(temperatures) if t > 0]
            of_drawn = np.empty(len(drawn), dtype=np.float32)
            fill_uniforms([seeds[i] for i in drawn], [indices[i] for i in drawn], of_drawn)
            uniforms[:] = 0.0
            uniforms[drawn] = of_drawn
        host[4 * n:5 * n] = [p.top_k for p in params]
        pairs = []
        if late:
            offsets, at = host[5 * n:6 * n + 1], 6 * n + 1
            offsets[0] = 0
            np.cumsum(lens, out=offsets[1:])
            # lists in one run over all ids; an array's or a tensor's ids are copied as one piece (80,000 of them 33 us, one by
            # one 9 ms)
            if True not in late and _LISTS.issuperset(map(type, histories)):
                host[at:at + total] = np.fromiter(chain.from_iterable(ids for on, ids in zip(penalised, histories) if on),
                                                  np.int32, total)
            else:
                for i, (ln, ids) in enumerate(zip(lens, histories)):
                    if ln:
                        host[at:at + ln - late[i]] = ids
                        if late[i]:
                            host[at + ln - 1] = -1                # an id the kernel skips, until it is put in place
                            pairs += [at + ln - 1 - 5 * n, int(pending[i])]
                        at += ln
            if total == 0:
                host[6 * n + 1] = 0
            ids_end = 6 * n + 1 + max(total, 1)
            host[ids_end:ids_end + len(pairs)] = pairs
        dev = self._dev[:words]
        dev.copy_(turn[0][:words], non_blocking=True)
        turn[1].record()
        turn[2] = True
        if pairs:
            ops.patch_words(dev[5 * n:], dev[ids_end:ids_end + len(pairs)], self._status[self._words:], len(pairs) // 2,
                            self._status[FAULT_TOKEN:FAULT_TOKEN + 1])
        if self._scratch is None or self._scratch.shape[0] < self._cap:
            self._scratch = torch.empty(self._cap, self.vocab, dtype=torch.float32, device=self.device)
        ops.sample_packed(logits, dev, max(total, 1) if late else 0, self._out[:n], self.bad, self._scratch)
        return n
