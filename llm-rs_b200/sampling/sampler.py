"""Chooses the next token of each request from its row of logits, on the device."""
from __future__ import annotations

from typing import List, Sequence

import numpy as np
import torch

from .. import ops
from .params import SamplingParams


class Sampler:
    """``sample(logits, rows)``: ``logits`` is float32 [n, vocab] on the device, ``rows`` gives per
    row ``(params, request_id, index of the token to generate, token history)``. Returns
    int32 tokens on the device. Rows that are plainly greedy take the argmax kernel; any
    other row sends the batch through the sampling kernel, whose result for a row
    depends on that row's logits, parameters, request id and index only."""

    def __init__(self, device):
        self.device = torch.device(device)

    def sample(self, logits: torch.Tensor, rows: Sequence[tuple]) -> torch.Tensor:
        n = logits.size(0)
        if n != len(rows):
            raise ValueError(f"{n} rows of logits for {len(rows)} requests")
        if all(p.plain for p, _, _, _ in rows):
            return ops.argmax(logits)
        need_hist = any(p.repetition_penalty != 1.0 for p, _, _, _ in rows)
        # One array, one copy to the device: seeds and ids (64-bit words first), temperatures, top_p, penalties, top_k, indices,
        # the histories' bounds and the histories. (Five pageable copies and two numpy integers a row held a step of 32 rows
        # up for 100 us.)
        hist: List[int] = []
        offsets = [0]
        if need_hist:
            for p, _, _, history in rows:
                if p.repetition_penalty != 1.0:
                    hist.extend(set(map(int, history)))      # distinct: the kernel touches a token's logit once
                offsets.append(len(hist))
        words = np.empty(9 * n + len(offsets) + len(hist), np.int32)
        whole = words[: 4 * n].view(np.uint64)
        whole[:n] = np.array([p.seed & (2**64 - 1) for p, _, _, _ in rows], np.uint64)
        whole[n:] = np.array([rid & (2**64 - 1) for _, rid, _, _ in rows], np.uint64)
        words[4 * n: 7 * n].view(np.float32)[:] = np.array(
            [[p.temperature for p, _, _, _ in rows], [p.top_p for p, _, _, _ in rows],
             [p.repetition_penalty for p, _, _, _ in rows]], np.float32).ravel()
        words[7 * n: 8 * n] = np.array([p.top_k for p, _, _, _ in rows], np.int32)
        words[8 * n: 9 * n] = np.array([index for _, _, index, _ in rows], np.int32)
        words[9 * n: 9 * n + len(offsets)] = offsets
        words[9 * n + len(offsets):] = np.array(hist, np.int32)
        d = torch.from_numpy(words).to(self.device, non_blocking=True)
        whole, numbers = d[: 4 * n].view(torch.int64), d[4 * n: 7 * n].view(torch.float32)
        return ops.sample(logits, numbers[:n], d[7 * n: 8 * n], numbers[n: 2 * n], numbers[2 * n:] if need_hist else None,
                          d[9 * n + len(offsets):] if need_hist else None, d[9 * n: 9 * n + len(offsets)] if need_hist else None,
                          whole[:n], whole[n:], d[8 * n: 9 * n])
