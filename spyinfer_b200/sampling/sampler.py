"""Chooses the next token of every row of a step's logits, on the device.

One kernel launch for the whole batch; only the token ids cross to the host.  A row's token
depends on its logits, its request's seed and the number of tokens the request has drawn so
far, not on the batch: a request preempted and recomputed draws the same tokens again.
"""
from __future__ import annotations

from typing import Sequence

import numpy as np
import torch

from .. import kernels
from .params import SamplingParams


class Sampler:
    def __init__(self, device):
        self.device = device

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], draws: Sequence[int]) -> torch.Tensor:
        """``logits [R, V]`` float32 on the device; ``draws[r]`` is how many tokens row r's
        request has generated before this one.  Returns int32 ``[R]`` on the device."""
        R = logits.shape[0]
        tokens = torch.empty(R, dtype=torch.int32, device=logits.device)
        if all(p.temperature == 0.0 for p in params):
            return kernels.sample(logits, tokens)
        draws = list(draws)
        if not len(params) == len(draws) == R:                 # a single number would be spread over all rows
            raise kernels.KernelError("sample: temperature, seed and draw need one entry per row")
        use_k = any(p.top_k > 0 and p.temperature > 0.0 for p in params)
        if use_k and max(p.top_k for p in params) > np.iinfo(np.int32).max:     # where no row uses it its size does not matter
            raise kernels.KernelError("sample: top_k does not fit 32 bits")
        host = np.zeros((4, R), np.int64)                      # one transfer: seeds, draws, temperatures, top_k
        try:
            host[0], host[1] = [p.seed for p in params], draws
        except OverflowError:
            raise ValueError("sample: seeds and draws must fit 64 bits") from None
        host[2].view(np.float32)[:R] = [p.temperature for p in params]
        if use_k:
            host[3].view(np.int32)[:R] = [p.top_k for p in params]
        dev = torch.from_numpy(host).to(logits.device, non_blocking=True)
        s, d, t = dev[0], dev[1], dev[2].view(torch.float32)[:R]
        return kernels.sample(logits, tokens, t, s, d, dev[3].view(torch.int32)[:R] if use_k else None)
