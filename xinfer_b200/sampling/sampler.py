"""Device-side sampling for a batch of logits rows: one launch for penalties, one for the draw
(greedy, temperature, top-k, top-p, top-k then top-p; src/utils/logits_processor.rs:258-344)."""
from __future__ import annotations

import struct
from typing import Optional, Sequence

import numpy as np
import torch

from .. import kernels, tracing
from .params import SamplingParams

# tokens that the penalties count: the most recent ones of the request, as many as the reference
# tracks (src/core/runner.rs:1887-1912)
PENALTY_HISTORY = 128

_RECORD = struct.Struct("<fifIIIffii")      # a row of kernels.SAMPLE_PARAMS, 40 bytes


def _uint32_halves(values, n: int) -> np.ndarray:
    """The low 64 bits of n whole numbers, as uint32 [low, high, low, high, ...]."""
    try:
        return np.array(values[:n] if isinstance(values, (list, tuple)) else [int(values[r]) for r in range(n)], dtype=np.int64).view(np.uint32)
    except OverflowError:
        return np.array([int(values[r]) & 0xFFFFFFFFFFFFFFFF for r in range(n)], dtype=np.uint64).view(np.uint32)


def fill_records(records: np.ndarray, params: Sequence[SamplingParams], seeds, draws, histories, history: np.ndarray) -> int:
    """The rows' options into ``records`` (a row each, in the order of its fields) and the tokens that penalties count into
    ``history``, one row's behind another's; returns how many tokens those are.  A row is packed as a whole, and options are
    read once for neighbouring rows that share them; many rows that all share one object are filled column by column.  64 rows:
    18 us where they share one object, 56 us where each has its own, 325 us field by field through numpy."""
    n, off, last = len(params), 0, None
    view, at, pack = memoryview(records).cast("B"), 0, _RECORD.pack_into
    columns = n >= 16 and not (params[0].has_penalties and histories is not None) and all(p is params[0] for p in params)
    for r, p in enumerate(params[:1] if columns else params):
        if p is not last:
            k = p.top_k
            last, penalised, t = p, p.has_penalties and histories is not None, 0.0 if p.greedy else float(p.temperature)
            k, top_p = int(k) if k and k > 0 else 0, float(p.top_p) if p.top_p is not None else 1.0
            frequency, presence = float(p.frequency_penalty or 0.0), float(p.presence_penalty or 0.0)
        m = 0
        if penalised:
            h = list(histories[r])[-PENALTY_HISTORY:]
            m = len(h)
            history[off:off + m] = h
        s = int(seeds[r])
        row = (t, k, top_p, s & 0xFFFFFFFF, (s >> 32) & 0xFFFFFFFF, int(draws[r]) & 0xFFFFFFFF, frequency, presence, off, m)
        try:
            pack(view, at, *row)
        except (struct.error, OverflowError):
            records[r] = row            # a float beyond float32 is an infinity, a whole number beyond its field an OverflowError
        at += 40
        off += m
    if columns:
        records[1:n] = records[0]
        s = _uint32_halves(seeds, n)
        records["seed_lo"][:n], records["seed_hi"][:n], records["draw"][:n] = s[0::2], s[1::2], _uint32_halves(draws, n)[0::2]
    return off


class _PinnedSets:
    """Where calls' records and counted tokens lie on the host until they have been copied, for calls that nobody may have waited
    for: sets used in turn.  Half of them are taken again only after the copies that read them have been made: one event per
    half, since recording and asking one for every call took a tenth of its time.  A call that a CUDA graph captures neither waits
    nor records (its copies have not been made, and an event of the graph cannot be waited for): the graph copies from the set of
    that call whenever it is replayed."""

    def __init__(self, max_rows: int, record_bytes: int, half: int = 8):
        self.params = torch.zeros((2 * half, max_rows * record_bytes), dtype=torch.uint8, pin_memory=True)
        self.max_rows, self.hist = max_rows, None
        self.sets = [None] * (2 * half)         # (bytes, the same as records, counted tokens, the same as an array), made when needed
        self.copied = [torch.cuda.Event(), torch.cuda.Event()]
        self.half, self.at = half, 0

    def take(self, counts_tokens: bool):
        """A set that no copy reads any more: (bytes, the same as records, counted tokens, the same as an array; None without)."""
        if self.at % self.half == 0 and not torch.cuda.is_current_stream_capturing():
            self.copied[self.at // self.half].synchronize()
        mine = self.sets[self.at]
        if mine is None or (counts_tokens and mine[2] is None):
            if counts_tokens and self.hist is None:
                self.hist = torch.zeros((2 * self.half, self.max_rows * PENALTY_HISTORY), dtype=torch.int32, pin_memory=True)
            params, hist = self.params[self.at], self.hist[self.at] if self.hist is not None else None
            mine = self.sets[self.at] = (params, params.numpy().view(kernels.SAMPLE_PARAMS), hist, hist.numpy() if hist is not None else None)
        return mine

    def sent(self) -> None:
        """The set last taken has been handed to its copies."""
        self.at += 1
        if self.at % self.half == 0:
            if not torch.cuda.is_current_stream_capturing():
                self.copied[self.at // self.half - 1].record()
            self.at %= 2 * self.half


class Sampler:
    def __init__(self, device, max_rows: int, out_dev: Optional[torch.Tensor] = None,
                 err_word: Optional[torch.Tensor] = None):
        """``out_dev``: int32 device buffer of max_rows + 1 that receives the ids (default: one of
        its own).  ``err_word``: a device int32 whose value is copied behind the ids, so that the
        step's tokens and its error word reach the host in one copy (``finish_copy`` returns both)."""
        self.device = device
        self.max_rows = max_rows
        self.err_word = err_word
        rec = kernels.SAMPLE_PARAMS.itemsize
        self._pinned = _PinnedSets(max_rows, rec)
        self._params_dev = torch.zeros(max_rows * rec, dtype=torch.uint8, device=device)
        self._hist_dev = torch.zeros(max_rows * PENALTY_HISTORY, dtype=torch.int32, device=device)
        self._out_dev = out_dev if out_dev is not None else torch.zeros(max_rows + 1, dtype=torch.int32, device=device)
        if self._out_dev.numel() < max_rows + 1 or self._out_dev.dtype != torch.int32:
            raise ValueError("the sampler's output buffer must hold max_rows + 1 int32")
        self._out_host = torch.zeros(max_rows + 1, dtype=torch.int32, pin_memory=True)
        self._scratch = torch.zeros(kernels.sample_scratch_bytes(max_rows), dtype=torch.uint8, device=device)

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               draws: Sequence[int], histories: Optional[Sequence[Sequence[int]]] = None) -> torch.Tensor:
        """One token per logits row, as an int32 device tensor (a view of a reused buffer).
        ``seeds[r]`` / ``draws[r]``: the request's seed and how many tokens it has drawn before.
        ``histories[r]``: the request's recent tokens, used when it has penalties."""
        R = logits.shape[0]
        if R > self.max_rows:
            raise ValueError(f"{R} rows exceed the sampler's capacity {self.max_rows}")
        params_host, records, hist_host, hist = self._pinned.take(histories is not None)
        off = fill_records(records, params[:R], seeds, draws, histories, hist)
        any_pen = off > 0
        nb = R * kernels.SAMPLE_PARAMS.itemsize
        self._params_dev[:nb].copy_(params_host[:nb], non_blocking=True)
        if any_pen:
            self._hist_dev[:off].copy_(hist_host[:off], non_blocking=True)
        self._pinned.sent()
        if tracing.ENABLED:
            tracing.push("sample")
        kernels.sample(self._out_dev, logits, self._params_dev, self._hist_dev, any_pen, self._scratch, self.err_word,
                       capacity=self.max_rows)
        if tracing.ENABLED:
            tracing.pop()
        return self._out_dev[:R]

    def reset(self) -> None:
        """After a failed step: the scratch is zeroed again (a kernel that did not finish may have
        left counters behind) and a queued copy is forgotten."""
        self._scratch.zero_()
        self._copied = 0
        self._copy_done = None

    def to_host(self, tokens_dev: torch.Tensor) -> np.ndarray:
        """Copy sampled ids to the host (synchronises the stream)."""
        self.start_copy(tokens_dev)
        return self.finish_copy()[0]

    def start_copy(self, tokens_dev: torch.Tensor) -> None:
        """Queue the copy of the sampled ids (and the error word behind them) to the host;
        ``finish_copy`` waits for it alone, so work queued after it keeps running."""
        n = tokens_dev.shape[0]
        self._out_host[:n + 1].copy_(self._out_dev[:n + 1], non_blocking=True)
        self._copied = n
        self._copy_done = torch.cuda.Event()
        self._copy_done.record()

    def finish_copy(self):
        """(ids, error word); the word is 0 when the sampler was given none."""
        self._copy_done.synchronize()
        n = self._copied
        return self._out_host[:n].numpy().copy(), (int(self._out_host[n]) if self.err_word is not None else 0)
