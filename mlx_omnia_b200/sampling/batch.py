"""One call of the sampling kernel for the rows of a step."""

from __future__ import annotations

import numpy as np
import torch

from mlx_omnia_b200.kernels import ops
from mlx_omnia_b200.sampling.options import SamplingParams


def sample_rows(logits: torch.Tensor, params: list[SamplingParams], seeds: list[int], draws: list[int],
                histories: list[list[int]]) -> torch.Tensor:
    """Choose one token per row of float32 `logits` [rows, vocab]. `seeds[i]` and
    `draws[i]` (how many tokens row i's request has drawn so far) fix the random stream;
    `histories[i]` are the request's latest tokens for the repetition penalty.
    -> int32 [rows] on the device."""
    if all(p.greedy and p.repetition_penalty == 1.0 for p in params):
        return ops.argmax(logits)
    rows = len(params)
    penalised = any(p.repetition_penalty != 1.0 for p in params)
    width = max(p.penalty_context for p in params) if penalised else 0
    # All rows' parameters in one buffer and one copy (`ops.sample` takes them one tensor each).
    words = np.empty((9 if penalised else 8) * rows + rows * width, dtype=np.int32)
    wide, real = words[: 4 * rows].view(np.int64), words.view(np.float32)
    wide[:rows] = [s & 0x7FFFFFFFFFFFFFFF for s in seeds]
    wide[rows:] = draws
    real[4 * rows: 5 * rows] = [p.temperature for p in params]
    words[5 * rows: 6 * rows] = [p.top_k for p in params]
    real[6 * rows: 7 * rows] = [p.top_p for p in params]
    real[7 * rows: 8 * rows] = [p.min_p for p in params]
    if penalised:
        real[8 * rows: 9 * rows] = [p.repetition_penalty for p in params]
        table = words[9 * rows:].reshape(rows, width)
        table.fill(-1)
        for i, (p, h) in enumerate(zip(params, histories)):
            recent = h[-p.penalty_context:] if p.repetition_penalty != 1.0 else []
            table[i, : len(recent)] = recent
    packed = torch.from_numpy(words).to(logits.device, non_blocking=True)
    whole, real = packed[: 4 * rows].view(torch.int64), packed.view(torch.float32)
    part = lambda t, i: t[i * rows: (i + 1) * rows]  # noqa: E731
    return ops.sample(logits, part(real, 4), part(packed, 5), part(real, 6), part(real, 7), part(whole, 0), part(whole, 1),
                      part(real, 8) if penalised else None, packed[9 * rows:].view(rows, width) if penalised else None)
