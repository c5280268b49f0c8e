"""What one step runs: the packed tokens of its sequences and where each token sits.

Every array is int32 on the device, filled from one pinned host buffer with a single copy:
  tokens[t]     token id                    token_seq[t]  index of its sequence in this step
  token_pos[t]  absolute position           seq_slot[s]   cache slot of sequence s
  seq_start[s]  positions cached before     seq_new[s]    tokens the step brings for s
  seq_tok0[s]   packed index of s's first token of the step
  want_rows[r]  packed token indices whose logits are asked for
"""
from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch


from ..csrc.lib import PREFILL_TILE_ROWS as Q_TILE      # query rows that one block of the prefill attention kernel takes


@dataclass
class StepBatch:
    n_tokens: int
    n_seqs: int
    n_want: int
    max_new: int
    dtype: torch.dtype
    tokens: torch.Tensor
    token_seq: torch.Tensor
    token_pos: torch.Tensor
    seq_slot: torch.Tensor
    seq_start: torch.Tensor
    seq_new: torch.Tensor
    seq_tok0: torch.Tensor
    want_rows: torch.Tensor
    slots: list
    starts: list
    n_new: list
    ctx_bucket: int = 0                # an upper bound of the longest context, a power of two (sizes key splits)
    n_q_tiles: int = 0                 # prefill only: tiles of up to Q_TILE consecutive tokens of one sequence,
    tile_tok0: torch.Tensor = None     # first packed token of each tile, longest context first
    tile_rows: torch.Tensor = None     # tokens in each tile

    @property
    def is_decode(self) -> bool:
        return self.max_new == 1


class BatchStager:
    """Builds StepBatch objects.  Index arrays go through a small ring of pinned host buffers, each
    with a device twin; a buffer is written again only after the copy that last read it has finished,
    so the host never waits for the step before last."""

    RING = 4

    def __init__(self, device):
        self.device = torch.device(device)
        self._cap = 0
        self._ring = []
        self._next = 0
        self.bytes_staged = 0          # host-to-device bytes of the latest step

    @staticmethod
    def words_needed(n_tokens: int, n_seqs: int, n_want: int) -> int:
        """int32 words a decode step (one token per sequence, no query tiles) stages."""
        return 3 * n_tokens + 4 * n_seqs + n_want

    def _reserve(self, n: int) -> None:
        if n <= self._cap:
            return
        self._cap = max(n, int(self._cap * 1.5), 4096)
        pin = self.device.type == "cuda"
        self._ring = []
        for _ in range(self.RING):
            host = torch.empty(self._cap, dtype=torch.int32, pin_memory=pin)
            dev = torch.empty(self._cap, dtype=torch.int32, device=self.device)
            self._ring.append([host, dev, None, host.numpy()])

    def stage(self, slots, starts, token_lists, wants, dtype, static_dev=None, views_of=None) -> StepBatch:
        """`static_dev`: an int32 device buffer to fill instead of the ring's (its address then stays the
        same from step to step, which a captured CUDA graph needs).  `views_of`: a batch that `stage` made over that
        buffer for a step of the same sizes; its arrays are filled again and it is returned, its host values unchanged."""
        B = len(slots)
        n_new = [len(t) for t in token_lists]
        T = sum(n_new)
        R = sum(len(w) for w in wants)
        tiles = []
        if max(n_new) > 1:
            base = 0
            for n, st in zip(n_new, starts):
                for off in range(0, n, Q_TILE):
                    rows = min(Q_TILE, n - off)
                    tiles.append((st + off + rows, base + off, rows))
                base += n
            tiles.sort(key=lambda x: -x[0])          # most keys first: the long tiles start early
        total = 3 * T + 4 * B + R + 2 * len(tiles)
        self._reserve(total)
        entry = self._ring[self._next]
        self._next = (self._next + 1) % self.RING
        h, d, ev = entry[:3]
        if static_dev is not None:
            d = static_dev
        if ev is not None:
            ev.synchronize()
        w = entry[3]                                  # the pinned buffer as a numpy array
        tok0, base = [], 0
        for n in n_new:
            tok0.append(base)
            base += n
        if max(n_new) == min(n_new) == 1:             # single tokens: a few numbers each, no query tiles
            w[:total] = ([t[0] for t in token_lists] + list(range(B)) + list(starts) + list(slots) + list(starts) + n_new + tok0
                         + [b + i for b, wt in zip(tok0, wants) for i in wt])
        else:
            for s, (toks, st, b, n) in enumerate(zip(token_lists, starts, tok0, n_new)):
                w[b:b + n] = toks
                w[T + b:T + b + n] = s
                w[2 * T + b:2 * T + b + n] = np.arange(st, st + n, dtype=np.int32)
            w[3 * T:total] = (list(slots) + list(starts) + n_new + tok0 + [b + i for b, wt in zip(tok0, wants) for i in wt]
                              + [t[1] for t in tiles] + [t[2] for t in tiles])
        d[:total].copy_(h[:total], non_blocking=True)
        self.bytes_staged = total * 4
        if self.device.type == "cuda":
            if ev is None:
                ev = entry[2] = torch.cuda.Event()
            ev.record()
        if views_of is not None:                      # the caller holds a batch of the same sizes in the same buffer
            return views_of
        o = 0

        def take(n):
            nonlocal o
            v = d[o:o + n]
            o += n
            return v

        longest = max(st + n for st, n in zip(starts, n_new))
        bucket = 256
        while bucket < longest:
            bucket *= 2
        return StepBatch(n_tokens=T, n_seqs=B, n_want=R, max_new=max(n_new), dtype=dtype, ctx_bucket=bucket,
                         tokens=take(T), token_seq=take(T), token_pos=take(T), seq_slot=take(B),
                         seq_start=take(B), seq_new=take(B), seq_tok0=take(B), want_rows=take(R),
                         slots=list(slots), starts=list(starts), n_new=n_new,
                         n_q_tiles=len(tiles), tile_tok0=take(len(tiles)), tile_rows=take(len(tiles)))
