"""Sampler: logits -> token ids, one kernel launch for the whole batch.

liteinfer/sampling/sampler.py:19-63 takes greedy rows together in one arg-max
and loops over the stochastic rows (temperature, top-k, softmax, top-p,
multinomial with a per-request generator).  Here both kinds are one launch: a
batch of only greedy rows runs the arg-max kernel, any other batch the
sampling kernel, which treats a row with temperature 0 or top_k 1 as arg-max.

Random numbers come from the host: every request owns a `random.Random` stream
(seeded by `SamplingParams.seed` alone, or for unseeded requests by the engine's
seed and a key the caller gives), and each sampled token consumes one uniform number from it.  What a
request draws therefore does not depend on which other requests share its
batch.
"""

from __future__ import annotations

import random

import numpy as np
import torch

from liteinfer_b200 import ops
from liteinfer_b200.sampling.params import SamplingParams


class Sampler:
    def __init__(self, seed: int = 42) -> None:
        self.seed = seed
        self._streams: dict[tuple[int, str | None], random.Random] = {}

    def _new_stream(self, params: SamplingParams, key: str | None) -> random.Random:
        if params.seed is not None:
            # Every request with this seed draws the same numbers: the same prompt gives the same tokens.
            stream = random.Random(params.seed)
        else:
            stream = random.Random(f"{self.seed}/{params.id}" if key is None else f"{self.seed}/{params.id}/{key}")
        self._streams[params._serial, key] = stream
        return stream

    def forget(self, params: SamplingParams, key: str | None = None) -> None:
        """Drop the random stream of a finished request."""
        self._streams.pop((params._serial, key), None)

    def __call__(self, logits: torch.Tensor, params: list[SamplingParams],
                 keys: list[str | None] | None = None) -> torch.Tensor:
        """One token id per row of `logits` [batch, vocab]; int32 on the logits' device.

        `keys` tells apart requests that share one SamplingParams object (a list of
        prompts generated with the same parameters): each key gets its own stream.
        """
        if logits.ndim != 2:
            raise ValueError(f"expected 2D logits, got shape {tuple(logits.shape)}")
        if len(params) != logits.shape[0]:
            raise ValueError(f"params length {len(params)} != batch size {logits.shape[0]}")
        rows = logits.shape[0]
        out = torch.empty(rows, dtype=torch.int32, device=logits.device)
        if rows == 0:
            return out
        if all(p.greedy for p in params):
            return ops.argmax(logits, out)
        # A loop of plain lookups: 48 rows held a call up for 67 us by comprehensions over properties and a
        # pinned copy, and are now done before the kernel is (55 us).
        temperatures, top_ks, top_ps, uniforms = [], [], [], []
        streams = self._streams
        for p, key in zip(params, keys or [None] * rows):
            temperature, top_k = p.temperature, p.top_k
            top_ps.append(p.top_p)
            top_ks.append(top_k if top_k > 0 else 0)
            if temperature == 0.0 or top_k == 1:            # greedy: no number is drawn for it
                temperatures.append(0.0)
                uniforms.append(0.0)
                continue
            temperatures.append(temperature)
            stream = streams.get((p._serial, key)) or self._new_stream(p, key)
            uniforms.append(stream.random())
        if len(uniforms) != rows:
            raise ValueError(f"keys length {len(uniforms)} != batch size {rows}")
        # Temperature, top_p, uniform (float32) and top_k (the bits of int32).
        along = logits.is_cuda and rows <= ops.SAMPLE_FROM_HOST
        host = torch.empty((4, rows), dtype=torch.float32, pin_memory=logits.is_cuda and not along)
        staged = host.numpy()
        staged[0], staged[1], staged[2] = temperatures, top_ps, uniforms
        staged[3].view(np.int32)[:] = top_ks
        if along:
            return ops.sample_from_host(logits, host, out)
        dev = host.to(logits.device, non_blocking=True)
        return ops.sample(logits, dev[0], dev[3].view(torch.int32), dev[1], dev[2], out)
