"""Batched sampling on the device: one call for rows with mixed settings.

Order as in tinyserve's ``sample`` (serve.py:1501-1588): repetition penalty on the
logits, then argmax for greedy rows, else temperature, top-k, top-p and Gumbel-max.
Unlike there, the noise of a row depends only on (engine seed, the request's stream,
how many tokens the request has generated), not on the batch around it."""
from __future__ import annotations

import zlib

import numpy as np
import torch

from ..kernels import ops


_TORCH = {np.float32: torch.float32, np.int32: torch.int32, np.int64: torch.int64}


def stream_of(request_id, params) -> int:
    """The request's noise stream: its ``seed`` if given, else a hash of its id."""
    if params.seed is not None:
        return int(params.seed) & (2 ** 63 - 1)
    return zlib.crc32(str(request_id).encode()) | (1 << 40)


def recent_tokens(params, token_ids) -> list:
    """Distinct tokens the repetition penalty applies to (serve.py:1469-1476)."""
    if params.repetition_penalty == 1.0 or params.repeat_last_n == 0:
        return []
    window = token_ids if params.repeat_last_n < 0 else token_ids[-params.repeat_last_n:]
    return sorted(set(window))


class Sampler:
    def __init__(self, seed: int, device, max_rows: int = 0):
        self.seed = int(seed)
        self.device = device
        self._zeros: dict = {}
        self._staging = None
        self._rows = max_rows
        self._flip = 0

    def _stage(self, *columns):
        """Columns of 32-bit (or, as int64, 64-bit) values as device tensors, through one pinned staging
        buffer and one copy (two buffers take turns: the copy of the step before may still be pending; an
        event per buffer keeps a host that runs further ahead from overwriting one)."""
        sizes = [c.nbytes // 4 for c in columns]
        offsets, words = [], 0
        for size in sizes:
            offsets.append(words)
            words += (size + 3) // 4 * 4
        if self._staging is None or words > self._staging[0].numel():
            room = max(words, 6 * max(self._rows, 8), 2 * self._staging[0].numel() if self._staging else 0)
            pin = torch.device(self.device).type == "cuda"
            self._staging = [(torch.zeros(room, dtype=torch.int32).pin_memory() if pin
                              else torch.zeros(room, dtype=torch.int32)) for _ in range(2)]
            self._device_words = torch.zeros(room, dtype=torch.int32, device=self.device)
            self._copied = [None, None]
        at_buffer, self._flip = self._flip, self._flip ^ 1
        host, copied = self._staging[at_buffer], self._copied[at_buffer]
        if copied is not None:
            copied.synchronize()
        h = host.numpy()
        for column, at, size in zip(columns, offsets, sizes):
            h[at:at + size] = column.reshape(-1).view(np.int32)
        self._device_words[:words].copy_(host[:words], non_blocking=True)
        if self._device_words.is_cuda:
            self._copied[at_buffer] = copied or torch.cuda.Event()
            self._copied[at_buffer].record()
        return [self._device_words[at:at + size].view(_TORCH[column.dtype.type]).view(column.shape)
                for column, at, size in zip(columns, offsets, sizes)]

    def _greedy_args(self, n):
        """Device tensors for an all-greedy batch (temperature 0 ignores the noise arguments)."""
        if n not in self._zeros:
            self._zeros[n] = (torch.zeros(n, dtype=torch.float32, device=self.device),
                              torch.zeros(n, dtype=torch.int64, device=self.device),
                              torch.zeros(n, dtype=torch.int32, device=self.device))
        return self._zeros[n]

    def __call__(self, logits, requests, slot_tokens=None, slots=None):
        """logits float32 [B, V] (modified in place by the penalty); ``requests``: objects with
        request_id, params, token_ids, prompt_len.  Returns int32 [B] on the device.  With
        ``slot_tokens`` and ``slots`` (int32 [B], device) every token is also left at its request's
        state slot for the next step."""
        B = logits.shape[0]
        feedback = dict(slot_tokens=slot_tokens, slots=slots)
        if all(r.params.temperature == 0 and (r.params.repetition_penalty == 1.0 or r.params.repeat_last_n == 0)
               for r in requests):
            temps, streams, steps = self._greedy_args(B)
            return ops.sample(logits, temps, streams, steps, self.seed, **feedback)
        temps, ks, ps, streams, steps = [], [], [], [], []
        pen_rows, pen_ids, pen_vals = [], [], []
        for i, r in enumerate(requests):
            p = r.params
            temps.append(float(p.temperature))
            ks.append(int(p.top_k) if p.top_k and p.top_k > 0 else 0)
            ps.append(float(p.top_p))
            streams.append(stream_of(r.request_id, p))
            steps.append(len(r.token_ids) - r.prompt_len)
            ids = recent_tokens(p, r.token_ids)
            if ids:
                pen_rows.append(i)
                pen_ids.append(ids)
                pen_vals.append(float(p.repetition_penalty))
        need_k = any(k > 0 for k, t in zip(ks, temps) if t > 0)
        need_p = any(p < 1.0 for p, t in zip(ps, temps) if t > 0)
        columns = [np.array(temps, np.float32), np.array(ps, np.float32), np.array(ks, np.int32), np.array(steps, np.int32),
                   np.array(streams, np.int64)]
        if pen_rows:
            table = np.full((len(pen_rows), max(len(x) for x in pen_ids)), -1, np.int32)
            for row, ids in zip(table, pen_ids):
                row[:len(ids)] = ids
            columns += [np.array(pen_rows, np.int32), table, np.array(pen_vals, np.float32)]
        d_temps, d_ps, d_ks, d_steps, d_streams, *penalty = self._stage(*columns)
        if penalty:
            ops.apply_repetition_penalty(logits, *penalty)
        return ops.sample(logits, d_temps, d_streams, d_steps, self.seed, top_k=d_ks if need_k else None,
                          top_p=d_ps if need_p else None, **feedback)
