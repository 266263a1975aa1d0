"""Choosing the next token of every row of a logits matrix, on the device.

Order of operations as in the reference (src/qwen25vl_lite/sampling.py:44-106;
src/qwen25vl_lite/engine.py:813-821): penalties on the logits, then for temperature > 0
``scores = logits / T``, top-k, min-p, top-p, softmax and one draw; temperature 0 is argmax.

Everything runs in the engine's own kernels (``csrc/sampling.cu``), all rows of a step in one
launch: greedy and plain temperature rows in one that scans the logits, and steps in which a row
asks for penalties, top-k, min-p or top-p in one that holds a row in a cluster's shared memory.
Only rows of a vocabulary too large for that (above 400,000 tokens) are narrowed row by row with
device-side sort and scan primitives.  The draw is keyed by ``(seed, index of the token being drawn)`` like the
reference's ``seed + len(outputs)`` generator (engine.py:823-829); a request without a seed
gets a fresh random one.
"""

from __future__ import annotations

import secrets
from array import array
from collections import Counter
from typing import List, Optional, Sequence

import numpy as np
import torch

from ..ops import kernels
from ..ops.host import host_ints
from .params import SamplingParams


def new_seed() -> int:
    return secrets.randbits(63)


def filter_scores(scores: torch.Tensor, top_k: int, min_p: float, top_p: float) -> torch.Tensor:
    """One row of scaled logits -> the same row with dropped tokens at -inf
    (sampling.py:74-101: top-k keeps ties with the k-th value; min-p compares with
    ``min_p * max probability``; top-p keeps the smallest sorted prefix whose cumulative
    probability reaches top_p, the crossing token included)."""
    neg_inf = torch.full_like(scores, float("-inf"))
    if top_k and top_k > 0:
        k = min(int(top_k), scores.numel())
        kth = torch.topk(scores, k).values[-1]
        scores = torch.where(scores < kth, neg_inf, scores)
    if min_p > 0:
        probs = torch.softmax(scores, dim=-1)
        scores = torch.where(probs < min_p * probs.max(), neg_inf, scores)
    if top_p < 1.0:
        sorted_scores, order = torch.sort(scores, descending=True, stable=True)
        cumulative = torch.cumsum(torch.softmax(sorted_scores, dim=-1), dim=-1)
        # keep everything up to and including the first position whose cumulative >= top_p
        keep = torch.ones_like(cumulative, dtype=torch.bool)
        keep[1:] = cumulative[:-1] < top_p
        filtered = torch.where(keep, sorted_scores, torch.full_like(sorted_scores, float("-inf")))
        scores = torch.empty_like(scores).scatter_(0, order, filtered)
    return scores


class Sampler:
    def __init__(self, device):
        self.device = torch.device(device)
        self._host = None                     # pinned buffer the sampled ids are copied to

    def _upload(self, values, dtype) -> torch.Tensor:
        return torch.tensor(values, dtype=dtype).to(self.device, non_blocking=True)

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               token_indices: Sequence[int], previous: Optional[Sequence[Sequence[int]]] = None) -> List[int]:
        """``logits`` [rows, vocab] float32 on the device; one token id per row.

        ``seeds[r]`` and ``token_indices[r]`` key the draw of row r; ``previous[r]`` are the
        tokens generated so far (only read for rows with penalties)."""
        return self.collect(self.sample_async(logits, params, seeds, token_indices, previous))

    def collect(self, pending) -> List[int]:
        """Waits for the draw that ``sample_async`` started and returns its token ids."""
        if pending is None:
            return []
        host, event, rows = pending[:3]
        if event is None:
            return host
        event.synchronize()
        return host[:rows].tolist()

    @staticmethod
    def device_ids(pending):
        """The ids a pending draw leaves on the device (int32 [rows]), for a next step that is fed
        from there before the ids have reached the host; None when there are none."""
        return pending[3] if isinstance(pending, tuple) and len(pending) > 3 else None

    def sample_async(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
                     token_indices: Sequence[int], previous: Optional[Sequence[Sequence[int]]] = None):
        """Starts the draw and the copy of its result to pinned host memory; the host is free until
        ``collect``.  Returns (pinned ids, event of the copy, rows, ids on the device)."""
        rows = logits.shape[0]
        if rows == 0:
            return None
        if any(p.has_penalties or p.has_filters for p in params) and kernels.sample_filtered_supports(logits):
            out = torch.empty(rows, dtype=torch.int32, device=self.device)
            kernels.sample_filtered(logits, self._asks(params, seeds, token_indices, previous, rows), out)
            return self._copy_back(out, rows)
        if any(p.has_penalties for p in params):
            logits = logits.clone()
            ids: List[int] = []
            counts: List[int] = []
            offsets = [0]
            for p, prev in zip(params, previous or [[]] * rows):
                if p.has_penalties and prev:
                    c = Counter(int(t) for t in prev)
                    ids += list(c.keys())
                    counts += list(c.values())
                offsets.append(len(ids))
            if ids:
                kernels.apply_penalties(
                    logits, self._upload(ids, torch.int32), self._upload(counts, torch.int32),
                    self._upload(offsets, torch.int32),
                    self._upload([p.repetition_penalty for p in params], torch.float32),
                    self._upload([p.presence_penalty for p in params], torch.float32),
                    self._upload([p.frequency_penalty for p in params], torch.float32))
        temps = [float(p.temperature) for p in params]
        if any(p.has_filters for p in params):
            logits = logits.clone() if not any(p.has_penalties for p in params) else logits
            for r, p in enumerate(params):
                if p.has_filters:
                    logits[r] = filter_scores(logits[r] / p.temperature, p.top_k, p.min_p, p.top_p)
                    temps[r] = 1.0
        out = torch.empty(rows, dtype=torch.int32, device=self.device)
        if all(t <= 0 for t in temps):
            kernels.sample_rows(logits, None, None, None, out)
        else:
            seed_arr = np.asarray([int(s) & ((1 << 64) - 1) for s in seeds], dtype=np.uint64).view(np.int64)
            kernels.sample_rows(logits, self._upload(temps, torch.float32),
                                torch.from_numpy(seed_arr).to(self.device, non_blocking=True),
                                self._upload([int(t) for t in token_indices], torch.int32), out)
        return self._copy_back(out, rows)

    def _asks(self, params, seeds, token_indices, previous, rows: Optional[int] = None) -> torch.Tensor:
        """What every row asks for, as the kernel reads it (``SampleRow``), and behind it the earlier tokens of the rows
        with penalties as they came: the kernel counts them.  One copy from pinned memory.  Seeds and places of the draw are
        read only where a row is drawn."""
        rows = len(params) if rows is None else rows
        if len(params) < rows:
            raise ValueError(f"{rows} rows of logits and what {len(params)} of them ask for")
        params = params[:rows]
        spans, lists, n = [], [], 0
        for p, prev in zip(params, previous or [()] * rows):
            begin = n
            if p.has_penalties and prev:
                if type(prev) is not list:
                    prev = self._ints(prev)
                n += len(prev)
                lists.append((begin, n, prev))
            spans.append((begin, n))
        spans += [(n, n)] * (rows - len(spans))
        words = rows * kernels.SAMPLE_ASK_WORDS
        staged = torch.empty(words + max(n, 1), dtype=torch.int32, pin_memory=True)
        host = staged.numpy()
        asks = host[:words].reshape(rows, kernels.SAMPLE_ASK_WORDS)
        floats = asks.view(np.float32)
        floats[:, (0, 2, 3, 7, 8, 9)] = [
            (p.temperature, p.min_p, p.top_p, p.repetition_penalty, p.presence_penalty, p.frequency_penalty) if p.has_filters else
            (p.temperature, 0.0, 1.0, p.repetition_penalty, p.presence_penalty, p.frequency_penalty) for p in params]
        asks[:, 1] = [max(0, min(int(p.top_k or 0), 1 << 30)) if p.has_filters else 0 for p in params]
        if any(p.temperature > 0 for p in params):
            seed = np.array([int(s) & ((1 << 64) - 1) for s in list(seeds)[:rows]], dtype=np.uint64)
            asks[:, 4] = seed.astype(np.uint32).view(np.int32)
            asks[:, 5] = (seed >> np.uint64(32)).astype(np.uint32).view(np.int32)
            asks[:, 6] = [int(t) for t in list(token_indices)[:rows]]
        else:
            asks[:, 4:7] = 0
        asks[:, 10:12] = spans
        if n == 0:
            host[words] = 0
        for begin, end, prev in lists:
            if type(prev) is not list or not host_ints(prev, end - begin, staged.data_ptr() + 4 * (words + begin)):
                host[words + begin:words + end] = np.frombuffer(self._ints(prev), dtype=np.int32)
        return staged.to(self.device, non_blocking=True)

    @staticmethod
    def _ints(numbers) -> array:
        out = array("i")
        try:
            out.extend(numbers)
        except TypeError:                      # numbers that are no ints, or an array of other ints
            out = array("i", [int(t) for t in numbers])
        return out

    def _copy_back(self, out: torch.Tensor, rows: int):
        if self.device.type != "cuda":
            return out.tolist(), None, rows, out
        if self._host is None or self._host.numel() < rows:
            self._host = torch.empty(max(rows, 64), dtype=torch.int32, pin_memory=True)
        self._host[:rows].copy_(out, non_blocking=True)
        event = torch.cuda.Event()
        event.record()
        return self._host, event, rows, out
