"""Sequences that are fed with given tokens instead of sampled ones: replaying a trace, scoring texts.

They live beside the sampled requests in the scheduler's own memory: a parent row of the block table (which is also the row
of the recurrent state), pages of the shared allocator, and the worker's batch step, the one prompts run through.  A sequence
is admitted with its first tokens, may be left out of steps, and gives everything back when it ends.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Dict, Iterable, List, Sequence, Tuple

import numpy as np
import torch

from .worker import ExtendItem


@dataclass
class FedSequence:
    row: int
    length: int = 0


def _numbers(toks) -> np.ndarray:
    toks = toks.tolist() if isinstance(toks, torch.Tensor) else list(toks)
    try:
        x = None if toks and isinstance(toks[0], torch.Tensor) else np.array(toks)
    except (TypeError, ValueError):             # tensors of one element among them, on any device
        x = None
    return np.array([t.item() if isinstance(t, torch.Tensor) else t for t in toks]) if x is None else x


class TokenFeeder:
    def __init__(self, sched):
        self.s = sched
        self.live: Dict[str, FedSequence] = {}
        self.held_pages = 0

    def _open(self, rids: Sequence[str]) -> None:
        s, rows = self.s, []
        try:
            for rid in rids:
                row = s.bt.alloc_parent_row()
                if row is None:
                    raise RuntimeError(f"no free sequence row for {rid!r} ({len(self.live)} sequences are live)")
                rows.append(row)
                self.live[rid] = FedSequence(row)
        finally:
            # recurrent state of reused rows starts at zero
            if rows and (s.state_t is not None or s.state_d is not None):
                fresh = self._upload(rows)
                for pool in (s.state_t, s.state_d):
                    if pool is not None:
                        pool.clear_rows(fresh)

    def _upload(self, values) -> torch.Tensor:
        t = torch.from_numpy(np.asarray(values, dtype=np.int64))
        return t.pin_memory().to(self.s.device, non_blocking=True) if self.s.device.type == "cuda" else t

    def close(self, rid: str) -> None:
        self._close([rid])

    def _close(self, rids: Sequence[str]) -> None:
        """Rows and pages of ended sequences go back; no page of theirs has another holder."""
        s, pages = self.s, []
        try:
            for rid in rids:
                seq = self.live.pop(rid)
                if seq.length:
                    pages.append(s.bt.table[seq.row, :seq.length])
                s.bt.free_parent_row(seq.row)
                self.held_pages -= seq.length
                s.reserved_pages -= seq.length
        finally:
            if pages:
                s.alloc.free_owned(torch.cat(pages))

    def step(self, entries: Sequence[Tuple[str, List[int], List[int]]], end: Iterable[str] = ()) -> torch.Tensor:
        """``entries``: (id, next tokens, offsets among them whose logits are wanted), one batch; ``end``: ids whose rows
        and pages are given back after the step.  Returns fp32 logits [wanted, vocab] in the order of the entries."""
        s = self.s
        s._flush_pending()                          # the host changes allocator state here
        if len({rid for rid, _, _ in entries}) != len(entries):
            raise ValueError("a sequence may appear once per step")
        entries = [(rid, _numbers(toks), list(want)) for rid, toks, want in entries]
        for rid, toks, want in entries:
            have = self.live[rid].length if rid in self.live else 0
            if toks.ndim != 1:
                raise TypeError(f"{rid!r}: tokens are a flat list of numbers")
            if have + len(toks) > s.context_len:
                raise ValueError(f"{rid!r} would exceed the context length ({s.context_len})")
            if any(not 0 <= w < len(toks) for w in want):
                raise ValueError(f"{rid!r}: a wanted offset is outside its tokens")
            if not ((toks >= 0) & (toks < s.target.cfg.vocab_size)).all():
                raise ValueError(f"{rid!r}: a token is outside the vocabulary")
        need = sum(len(t) for _, t, _ in entries)
        if s.reserved_pages + need > s.alloc.size:
            raise RuntimeError(f"{need} more tokens do not fit: {s.alloc.size - s.reserved_pages} of {s.alloc.size} pages are free")
        self._open([rid for rid, _, _ in entries if rid not in self.live])
        items = [ExtendItem(self.live[rid].row, self.live[rid].length, toks.astype(np.int64), want) for rid, toks, want in entries if len(toks)]
        if items:
            pages = s.alloc.alloc(need)
            if pages is None:
                raise RuntimeError("page reservation violated")
            if len(items) > 2:                      # one indexed write for the batch
                rows = np.repeat([it.row for it in items], [len(it.input_ids) for it in items])
                cols = np.concatenate([np.arange(it.prefix, it.prefix + len(it.input_ids)) for it in items])
                at = self._upload(np.stack([rows, cols]))
                s.bt.table[at[0], at[1]] = pages
            else:
                for it, own in zip(items, pages.split([len(it.input_ids) for it in items])):
                    s.bt.table[it.row, it.prefix:it.prefix + len(it.input_ids)] = own
            for rid, toks, _ in entries:
                self.live[rid].length += len(toks)
            self.held_pages += need
            s.reserved_pages += need
        out = s.worker.extend(items) if items else torch.empty(0, s.target.cfg.vocab_size, device=s.device)
        if s.native_runner is not None:
            status = s.native_runner.check_status()
            if status:
                raise RuntimeError(f"device status {status} in a step of given tokens")
        self._close(list(end))
        return out
