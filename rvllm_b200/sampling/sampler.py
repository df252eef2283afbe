"""Sampling of one token per logits row on the device.

`Sampler.sample` gathers the rows' parameters into small tensors, launches the sampling
kernel and returns the token ids; only these ids leave the GPU
(as in the reference, v3/crates/rvllm-runtime/src/bring_up.rs:1443-1454).
"""
from __future__ import annotations

import struct
from typing import List, Optional, Sequence

import numpy as np
import torch

from ..errors import SamplingError
from .params import SamplingParams


def request_seed(engine_seed: int, request_number: int) -> int:
    """Seed of a request that brought none: a fixed mix of the engine's seed and the request's
    arrival number (splitmix64 finaliser), so that runs repeat."""
    z = (engine_seed * 0x9E3779B97F4A7C15 + request_number + 1) & 0xFFFFFFFFFFFFFFFF
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & 0xFFFFFFFFFFFFFFFF
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & 0xFFFFFFFFFFFFFFFF
    return (z ^ (z >> 31)) & 0x7FFFFFFFFFFFFFFF


class Sampler:
    def __init__(self, kernels=None, device="cuda:0"):
        if kernels is None:
            from ..kernels import get_library
            kernels = get_library(device)
        self.kernels = kernels

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               draw_index: Sequence[int]) -> torch.Tensor:
        """logits float32 [R, V]; one parameter set, seed and output index per row.
        Returns int32 token ids [R] on the device."""
        R = logits.shape[0]
        if not (len(params) == len(seeds) == len(draw_index) == R):
            raise SamplingError(f"{R} logits rows but {len(params)} parameter sets, {len(seeds)} seeds, "
                                f"{len(draw_index)} draw indices")
        if all(p.is_greedy for p in params):
            return self.kernels.sample(logits)
        top_ps, top_ks = [p.top_p for p in params], [p.top_k for p in params]
        temperatures = [p.temperature for p in params]
        try:      # with the launch itself: seeds and draw indices (64 bits), then temperatures, top-p and top-k (32 bits)
            packed = struct.pack(f"={2 * R}q{2 * R}f{R}i", *seeds, *draw_index, *temperatures, *top_ps, *top_ks)
        except (struct.error, OverflowError, TypeError):
            packed = None
        if packed is not None and hasattr(self.kernels, "sample_rows"):
            ids = self.kernels.sample_rows(logits, packed)
            if ids is not None:
                return ids
        # more rows than a launch carries: one buffer and one copy; the parameters' tensors are views of it on the device
        host = np.empty((7 * R,), dtype=np.int32)
        wide, real = host[:4 * R].view(np.int64), host[4 * R:6 * R].view(np.float32)
        wide[:R] = seeds
        wide[R:] = draw_index
        real[:R] = temperatures
        real[R:] = top_ps
        host[6 * R:] = top_ks
        flat = torch.from_numpy(host).to(logits.device, non_blocking=True)
        wide, real = flat[:4 * R].view(torch.int64), flat[4 * R:6 * R].view(torch.float32)
        return self.kernels.sample(logits, real[:R], flat[6 * R:] if max(top_ks) > 0 else None,
                                   real[R:] if min(top_ps) < 1.0 else None, wide[:R], wide[R:])
