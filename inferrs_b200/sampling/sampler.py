"""Choosing the next token of every row of a step, on the device.

The reference copies each row's logits to the host and samples there (inferrs/src/sampler.rs:146-357).
Here the rows of a step are sampled together by three kernels (penalties, rows with top-k, the others); what crosses
to the host is one token id per row.
"""
from __future__ import annotations

from array import array
from typing import Sequence

import numpy as np
import torch

from .. import kernels
from .params import NATIVE_ROWS, SamplingParams, host_python, uniforms_for


class Sampler:
    STAGING = 4      # pinned buffers used in turn: a step's numbers may still be on their way when the next is filled

    def __init__(self, device: torch.device, act_dtype: torch.dtype = torch.float32):
        self.device = device
        self.act_dtype = act_dtype
        self._staging = []       # [pinned int32 buffer, event of its last copy or None]
        self._turn = 0
        host_python()            # built with the sampler, not inside a step

    def _upload(self, words: np.ndarray) -> torch.Tensor:
        """The step's numbers (int32 words, floats as their bits) to the device with one copy that the host does not
        wait for: from one of a few pinned buffers, each reused only after its last copy has been made."""
        n = int(words.shape[0])
        if self.device.type != "cuda":
            return torch.from_numpy(words).to(self.device)
        if len(self._staging) < self.STAGING:
            self._staging.append([torch.empty((max(n, 4096),), dtype=torch.int32).pin_memory(), None])
            slot = self._staging[-1]
        else:
            slot = self._staging[self._turn]
            self._turn = (self._turn + 1) % self.STAGING
            if slot[1] is not None:
                slot[1].synchronize()
            if slot[0].shape[0] < n:
                slot[0] = torch.empty((2 * n,), dtype=torch.int32).pin_memory()
        slot[0].numpy()[:n] = words
        dev = torch.empty((n,), dtype=torch.int32, device=self.device)
        dev.copy_(slot[0][:n], non_blocking=True)
        if slot[1] is None:
            slot[1] = torch.cuda.Event()
        slot[1].record()
        return dev

    @staticmethod
    def _windows_natively(last, histories, pend, width: int, words: np.ndarray, counts: np.ndarray) -> bool:
        """The windows of :meth:`sample` through csrc/host_python.cpp; False where it does not take these histories."""
        native = host_python()
        n = min(len(last), len(histories), len(pend))
        if native is None or n != len(counts) or any(type(k) is not int or k > 0x7fffffff for k in last):
            return False
        lists = histories if type(histories) is list else list(histories)
        if any(type(h) is not list for h in lists):
            lists = [h if type(h) is list else [] if k <= x else h.tail(k - x) if hasattr(h, "tail") else h
                     for k, h, x in zip(last, lists, pend)]
        sizes = np.array([last[:n], pend[:n]], dtype=np.int32)
        at = sizes.__array_interface__["data"][0]
        return native.ibh_windows(lists, at, at + 4 * n, n, width, words.__array_interface__["data"][0],
                                  counts.__array_interface__["data"][0]) == 0

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], seeds: Sequence[int],
               histories: Sequence[Sequence[int]], pending: "int | Sequence[int]" = 0,
               pending_ids: "torch.Tensor | None" = None, pending_from=None) -> torch.Tensor:
        """int32 token ids [rows] (on the device) for float32 ``logits`` [rows, vocab].

        ``histories[r]`` is all tokens of row r's request so far, prompt and generated: its length is the
        step index of the random draw and its tail is the penalties' window.  It may be a list of token ids
        or an object with ``n_tokens`` and ``tail(n)`` (the scheduler's requests, which keep prompt and
        output apart).  ``logits`` is changed in place where penalties apply.  ``pending`` (0 or 1, one for all
        rows or one per row): the request has one more token that is on its way but not in its history yet; it
        counts for the step index of the draw, and ``pending_ids`` (int32 on the device, one per row; ignored
        where nothing is pending) has it for the penalties' window.  Instead of ``pending_ids``, ``pending_from`` =
        (ids, places) names a tensor of token ids on the device and, per row, the place of the row's pending token
        in it (any valid place where nothing is pending): the look-up then goes to the device with everything else.
        One options object, one seed or one history counts for every row; windows are those of the rows that have
        both an options object and a history of their own.

        Everything the kernels need per row goes to the device as one block of words in one copy that the
        host does not wait for, so a step can be prepared while the one before it still runs.
        """
        r = logits.shape[0]
        out = torch.empty((r,), dtype=torch.int32, device=self.device)
        if r == 0:
            return out
        if all(p.is_greedy and not p.has_penalty for p in params):
            kernels.argmax(logits, out, self.act_dtype)
            return out
        pend = [int(pending)] * r if isinstance(pending, int) else [int(x) for x in pending]
        if len(pend) != r or any(x not in (0, 1) for x in pend):
            raise ValueError("pending: 0 or 1, one for all rows or one per row")
        if len(params) not in (1, r):
            raise ValueError(f"options of {len(params)} rows for {r}")
        length = [(len(h) if type(h) is list else h.n_tokens if hasattr(h, "n_tokens") else len(h)) + x
                  for h, x in zip(histories, pend)]
        # rows that share an options object share its numbers (looked up within this call only): as many columns as objects
        own = list({id(p): p for p in params}.values())
        on = [p.has_penalty for p in own]
        last = [p.repeat_last_n if x else 0 for p, x in zip(own, on)]
        numbers = np.zeros((6, len(own)), dtype=np.float32)
        numbers[0] = [p.temperature for p in own]
        numbers[1] = [p.top_p for p in own]
        numbers[2] = [p.min_p for p in own]
        numbers[3] = 1.0
        if any(on):
            numbers[3] = [p.repetition_penalty if x else 1.0 for p, x in zip(own, on)]
            numbers[4] = [p.frequency_penalty if x else 0.0 for p, x in zip(own, on)]
            numbers[5] = [p.presence_penalty if x else 0.0 for p, x in zip(own, on)]
        top_k = np.array([p.top_k for p in own], dtype=np.int32)
        if len(own) == 1:
            last = last * len(params)
        elif len(own) < r:
            column = {id(p): i for i, p in enumerate(own)}
            which = [column[id(p)] for p in params]
            numbers, top_k, last = numbers[:, which], top_k[which], [last[i] for i in which]
        width = 0
        if any(on):
            if any(pend) and pending_ids is None and pending_from is None:
                raise ValueError("penalties need the whole history: the one pending token must be given on the device")
            width = max(1, max(min(k, n) for k, n in zip(last, length)))
        # the block: seven rows of floats (as their bits), two of ints, the penalties' windows, the pending tokens' places
        look_up = width > 0 and any(pend) and pending_ids is None
        words = np.empty((9 * r + r * width + (r if look_up else 0),), dtype=np.int32)
        floats = words[:7 * r].view(np.float32).reshape(7, r)
        floats[:3] = numbers[:3]
        floats[3] = uniforms_for(seeds, length)
        floats[4:] = numbers[3:]
        words[7 * r:8 * r] = top_k
        n_prev = words[8 * r:9 * r]
        n_prev[:] = 0
        if width and not (r >= NATIVE_ROWS and self._windows_natively(last, histories, pend, width, words[9 * r:9 * r + r * width], n_prev)):
            # the windows, row by row: -1 in the place of the pending token, the history's tail, -1 up to the width.  The
            # window's order does not matter: the pending token, if any, takes the first place.
            windows, counts, blank = array("i"), [], array("i", [-1]) * width
            for k, h, x in zip(last, histories, pend):
                known, n = k - x, 0
                if k:
                    if x:
                        windows.append(-1)
                    if known > 0:
                        tail = h.tail(known) if hasattr(h, "tail") else h[-known:]
                        tail = tail if isinstance(tail, list) else list(tail)
                        try:
                            windows.fromlist(tail)
                        except TypeError:               # ids held as floating-point numbers
                            windows.fromlist([int(t) for t in tail])
                        n = len(tail)
                    n += x
                counts.append(n)
                if n < width:
                    windows.extend(blank[:width - n] if n else blank)
            prev = words[9 * r:9 * r + r * width]
            prev[:len(windows)] = windows
            prev[len(windows):] = -1
            n_prev[:len(counts)] = counts
        if look_up:
            words[9 * r + r * width:] = list(pending_from[1])
        dev = self._upload(words)
        fd = dev[:7 * r].view(torch.float32).view(7, r)
        if width:
            prev_dev = dev[9 * r:9 * r + r * width].view(r, width)
            if look_up:
                pending_ids = pending_from[0].index_select(0, dev[9 * r + r * width:])
            if all(pend):
                prev_dev[:, 0].copy_(pending_ids[:r])
            elif any(pend):
                mask = self._upload(np.array(pend, dtype=np.int32)).to(torch.bool)
                prev_dev[:, 0] = torch.where(mask, pending_ids[:r].to(torch.int32), prev_dev[:, 0])
            kernels.penalties(logits, prev_dev, dev[8 * r:9 * r], fd[4], fd[5], fd[6], self.act_dtype)
        kernels.sample(logits, fd[0], dev[7 * r:8 * r], fd[1], fd[2], fd[3], out, self.act_dtype)
        return out
