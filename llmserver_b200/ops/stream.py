"""Two small types with which a step of few rows does without stand-alone residual-add + RMSNorm kernels.

A product whose result belongs on the residual stream adds it there in its own epilogue (``StreamSink``) and leaves,
for the RMSNorm that follows, the stream times the norm's weight (bfloat16) and partial sums of squares of the
updated rows (``RowScaled``).  The product that consumes the norm's output multiplies its 32-bit accumulators row by
row with 1 / rms: W (s w x) = s W (w x) for one scalar s per row.  Statistics, scale and the residual sum stay 32-bit;
only the place where bfloat16 rounding happens moves (before the division instead of after it).
"""
from __future__ import annotations

import os
from typing import Optional

import torch

# Up to this many rows a step always runs this way (LLMSERVER_B200_STREAM_ROWS changes it, up to the kernel's 128 rows);
# LLMSERVER_B200_STREAM_EPILOGUES=0 switches it off: the stand-alone add + norm kernel then runs at every row count.
STREAM_ROWS = (min(max(int(os.environ.get("LLMSERVER_B200_STREAM_ROWS", "16")), 0), 128)
               if os.environ.get("LLMSERVER_B200_STREAM_EPILOGUES", "1") != "0" else 0)
# The most rows that may run this way at all; ``stream_rows`` says how many do.
STREAM_MANY_ROWS = STREAM_ROWS if "LLMSERVER_B200_STREAM_ROWS" in os.environ else 128 if STREAM_ROWS else 0
STREAM_DEVICE_ROWS, STREAM_LAUNCH_WIDTH = 64, 4096


def stream_rows(width: int, decode: bool) -> int:
    """Up to how many rows a step over a stream of ``width`` columns runs this way where the environment does not say; ``decode``: it
    is a step of single tokens, which graphs replay.

    Up to 64 rows every step: the products are level with the library's and four launches a layer fall away.  Beyond, a token tile is
    as large as a weight tile and the library's products were faster on the device when these bounds were drawn, which decides wherever
    launches are replayed or the matrices are wide; only steps that the host's launches bound gain.  (This package's product kernel has
    since become 7 to 18 % faster there; replayed steps beyond 64 rows were not measured again.)  Stand-alone kernels from 17 rows on / none, ms:
    replayed decode steps, contexts of 301 to 2000: width 2048 2.33 / 2.24 at 24 rows, 2.94 / 2.95 at 64, 3.93 / 4.07 at 96, 4.72 / 4.98
    at 128; 8B shape 4.75 / 4.70 at 24, 5.55 / 5.43 at 48, 5.63 / 5.40 at 61, 7.04 / 7.23 at 96, 8.09 / 8.51 at 128; 14B shape (5120) 6.68 /
    6.42 at 24, 7.91 / 7.94 at 64, 9.90 / 9.76 at 96, 11.19 / 11.43 at 128; 32B shape (5120) 15.66 / 15.50 at 64.  Prompts: width 2048 4.33 /
    3.16 at 128 tokens; 8B 5.38 / 3.92 at 20, 6.18 / 4.38 at 64, 5.39 / 4.11 at 100, 5.34 / 4.21 at 128; 14B 6.02 / 5.61 at 20, 6.52 / 6.31
    at 64, 6.93 / 6.38 at 70, 6.88 / 6.82 at 100, 7.01 / 7.08 at 128; 32B 13.6 / 13.1 at 40, 14.4 / 14.1 at 64, 15.2 / 16.0 at 100, 15.8 / 16.9 at 128
    (the 8B prompts of 100 and 128 tokens and the 14B ones from 70 on with blocks that have an SM to themselves, the others beyond 64 rows before)."""
    if STREAM_MANY_ROWS <= STREAM_ROWS:
        return STREAM_MANY_ROWS
    return STREAM_DEVICE_ROWS if decode or width > STREAM_LAUNCH_WIDTH else STREAM_MANY_ROWS


NO_SCALE = (0, 0, 0, 0.0)


class RowScaled:
    """``x`` [N, H] bfloat16 = stream * norm weight; ``parts`` float32 [n_parts, >= N]: the sum over i of parts[i, n] is
    the sum of squares of stream row n.  Stands for x[n] / sqrt(sum / H + eps)."""

    __slots__ = ("x", "parts", "eps")

    def __init__(self, x: torch.Tensor, parts: torch.Tensor, eps: float):
        self.x, self.parts, self.eps = x, parts, float(eps)

    @property
    def shape(self):
        return self.x.shape

    @property
    def dtype(self):
        return self.x.dtype

    @property
    def device(self):
        return self.x.device

    def scale_args(self) -> tuple:
        """(parts pointer, number of parts, row capacity, eps) as the launchers take them."""
        return self.parts.data_ptr(), self.parts.shape[0], self.parts.shape[1], self.eps


def scale_args_of(x) -> tuple:
    return x.scale_args() if isinstance(x, RowScaled) else NO_SCALE


def rows_of(x) -> torch.Tensor:
    return x.x if isinstance(x, RowScaled) else x


class StreamSink:
    """Where a product may add its result: the 32-bit stream ``residual`` [N, H].  With ``norm_weight`` (and ``eps``)
    the product also prepares the input of the RMSNorm that follows (``scaled``, a ``RowScaled``).  ``owner`` is
    whoever made the sink (the norm it prepares for); ``added`` says whether a product took it."""

    __slots__ = ("residual", "norm_weight", "eps", "owner", "added", "scaled")

    def __init__(self, residual: torch.Tensor, norm_weight: Optional[torch.Tensor] = None, eps: float = 0.0, owner=None):
        self.residual, self.norm_weight, self.eps, self.owner = residual, norm_weight, float(eps), owner
        self.added = False
        self.scaled: Optional[RowScaled] = None
