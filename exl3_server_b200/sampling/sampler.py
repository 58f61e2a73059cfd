"""Choosing how a batch of logit rows is sampled.

Rows that are all greedy take the argmax kernel.  Everything else that the
device sampler covers (temperature with top-k up to its cap, top-p, min-p and
the penalties over the context) is sampled on the device by the reference's
algorithm (``csrc/sampling_filtered.cu``): only the options, the uniform numbers
and the chosen ids cross between host and device.  ``host.sample_token`` is the
same algorithm on the host (src/model.cpp:667-757), for logits that are not on
the device and for ``top_k`` above the cap; the tests hold the two against
each other.
"""
from __future__ import annotations

import struct
from itertools import chain
from operator import attrgetter
from typing import List, Optional, Sequence

import numpy as np
import torch

from .host import sample_token
from .options import SampleOptions, SplitMix64


class RowSampler:
    """Sampling state of one request: its options, generator and context."""

    def __init__(self, opt: SampleOptions, request_index: int, prompt: Sequence[int]):
        self.opt = opt
        self.rng = SplitMix64(opt.seed + request_index)
        self.context: List[int] = list(prompt)
        self._counts: Optional[torch.Tensor] = None      # int32 [vocab] on the device: how often each token occurs
        self._counted = 0                                # tokens of the context that the counts hold

    def device_counts(self, vocab: int, device) -> torch.Tensor:
        """The context's token counts on the device, for the penalties: made from the whole context when first
        asked for, then kept up by the sampler's own kernel (``counted``) or from the context's new tokens."""
        if self._counts is None:
            self._counts = torch.zeros(vocab, dtype=torch.int32, device=device)
        if self._counted < len(self.context):
            new = torch.tensor([t for t in self.context[self._counted:] if 0 <= t < vocab], dtype=torch.int64)
            if new.numel():
                self._counts.index_add_(0, new.to(device), torch.ones(new.numel(), dtype=torch.int32, device=device))
            self._counted = len(self.context)
        return self._counts

    def counted(self, n: int = 1) -> None:
        """The device has added the next ``n`` tokens of the context to the counts itself."""
        self._counted += n


def on_device(logits: torch.Tensor, rows: Sequence[RowSampler]) -> bool:
    """Whether ``launch_on_device`` takes this batch."""
    if not logits.is_cuda:
        return False
    from ..ops import kernels as K
    cap = K.sample_filtered_cap()
    return all(r.opt.top_k <= cap for r in rows)


def launch_on_device(logits: torch.Tensor, rows: Sequence[RowSampler]) -> torch.Tensor:
    """Starts the sampling of one token per row on the device and returns the ids (int32 on the device)
    without waiting for them.  The generators advance now; the tokens join the rows' contexts when the caller
    has read them (``record``).  The penalties' token counts are kept up on the device."""
    return _launch(logits, rows, None)


# a row's options in the order in which the kernels take them
_OPTIONS = attrgetter("temperature", "top_k", "top_p", "min_p", "repetition_penalty", "presence_penalty", "frequency_penalty")


def _launch(logits: torch.Tensor, rows: Sequence[RowSampler], host_out: Optional[torch.Tensor]) -> torch.Tensor:
    """``launch_on_device``; ``host_out`` as in ``kernels.sample_batch``, for at most ``sample_direct_rows()`` rows."""
    from ..engine.decode import TRANSFERRED
    from ..ops import kernels as K
    if not logits.is_contiguous():
        if any(r.opt.has_penalties for r in rows):
            logits = logits.clone()                      # a slice of padded rows, or one row for all, becomes dense
        K._contig(logits, "logits")                      # before any generator has moved on
    R, V = logits.shape
    opts = [_OPTIONS(r.opt) for r in rows]
    # a greedy row draws no number from its generator, as on the host
    states = [0 if o[0] <= 0.0 else r.rng.step() for r, o in zip(rows, opts)]
    counts, penalised = [], []
    for r, o in zip(rows, opts):
        if o[4] != 1.0 or o[5] != 0.0 or o[6] != 0.0:
            counts.append(r.device_counts(V, logits.device).data_ptr())
            penalised.append(r)
        else:
            counts.append(0)
    if R <= K.sample_direct_rows():
        # the options travel with the launch.  The kernel reads the logits with their penalties (the step's own buffer stays
        # as the model left it), and the chosen tokens join the counts without a trip to the host
        packed = struct.pack(f"<{7 * R}d{2 * R}Q", *chain.from_iterable(opts), *states, *counts)
        kept = [c for c in counts if c]
        ids = K.sample_batch(logits, packed, len(set(kept)) < len(kept), host_out)
        n_bytes = len(packed)
    elif not penalised:
        host = np.array([(*o[:4], SplitMix64.uniform_of(z)) for o, z in zip(opts, states)], dtype=np.float64)
        ids = K.sample_filtered(logits, torch.from_numpy(host).to(logits.device))
        n_bytes = host.nbytes
    else:
        # options, the counts' addresses and the penalties as one buffer: one copy to the device
        host = np.empty(R * (40 + 8 + 12), dtype=np.uint8)
        host[:R * 40].view(np.float64).reshape(R, 5)[:] = [(*o[:4], SplitMix64.uniform_of(z)) for o, z in zip(opts, states)]
        host[R * 40:R * 48].view(np.int64)[:] = counts
        host[R * 48:].view(np.float32).reshape(R, 3)[:] = [o[4:] if c else (1.0, 0.0, 0.0) for o, c in zip(opts, counts)]
        dev = torch.from_numpy(host).to(logits.device)
        ids = K.sample_rows(logits, dev[:R * 40].view(torch.float64).view(R, 5), dev[R * 40:R * 48].view(torch.int64),
                            dev[R * 48:].view(torch.float32).view(R, 3))
        n_bytes = host.nbytes
    for r in penalised:
        r.counted()
    TRANSFERRED["h2d"] += n_bytes
    return ids


def record(rows: Sequence[RowSampler], picked: Sequence[int]) -> None:
    """The rows' sampled tokens, read by the host, join their contexts."""
    for r, t in zip(rows, picked):
        r.context.append(int(t))


def sample_rows(logits: torch.Tensor, rows: Sequence[RowSampler],
                device_argmax: Optional[torch.Tensor] = None) -> List[int]:
    """One token per row of ``logits`` ``[len(rows), vocab]`` (float32).
    ``device_argmax`` is the argmax of each row when the step already
    computed it on the device."""
    if logits.shape[0] != len(rows):
        raise ValueError(f"{logits.shape[0]} logit rows for {len(rows)} requests")
    picked: Optional[List[int]] = None
    if logits.is_cuda:
        from ..ops import kernels as K
        if all(r.opt.greedy and not r.opt.has_penalties for r in rows):
            ids = device_argmax if device_argmax is not None else K.argmax(logits)
            picked = ids.cpu().tolist()
            from ..engine.decode import TRANSFERRED
            TRANSFERRED["d2h"] += ids.numel() * 4
        elif on_device(logits, rows):
            if len(rows) <= K.sample_direct_rows():
                # the kernel writes the ids to page-locked memory itself
                host = torch.empty(len(rows), dtype=torch.int32, pin_memory=True)
                _launch(logits.to(torch.float32), rows, host)
                torch.cuda.current_stream().synchronize()
                picked = host.tolist()
            else:
                picked = launch_on_device(logits.to(torch.float32), rows).cpu().tolist()
            from ..engine.decode import TRANSFERRED
            TRANSFERRED["d2h"] += len(rows) * 4
    if picked is None:
        host = logits.detach().to(torch.float32).cpu().numpy()
        picked = [sample_token(host[i], r.opt, r.context, r.rng) for i, r in enumerate(rows)]
    record(rows, picked)
    return picked
