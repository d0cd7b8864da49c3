"""Pinned memory through which small host arrays reach the device without the host waiting.

A copy out of ordinary memory holds the host up until the device has done everything queued
before it; a step's launches then begin on an idle device.  Out of pinned memory the copy is
queued like a kernel.  The memory must not be written again before the copy has been made,
so there is a ring of buffers, each with the event recorded behind the last copies out of it: taking
a buffer waits for that event, which bounds how far the host runs ahead and what is pinned.
(The reference copies a step's inputs from the caller's tensors, src/entry.cu:541-597.)
"""
from __future__ import annotations

import threading
from typing import List, Optional, Sequence

import torch


class Staging:
    BUFFERS = 8
    BUFFER_BYTES = 32 * 1024          # a chunk of 2,048 prompt tokens; a larger array makes its buffer grow

    def __init__(self, device: torch.device):
        self.device = torch.device(device)
        self._lock = threading.Lock()
        self._buffers: List[torch.Tensor] = []
        self._done: List[Optional[torch.cuda.Event]] = []
        self._next = 0

    def copy(self, values: torch.Tensor, parts: Sequence[torch.Tensor]) -> None:
        """Copies the flat host tensor ``values`` into ``parts`` one after the other, in the order of the current stream.
        The parts hold together as many numbers as there are values."""
        if sum(part.numel() for part in parts) != values.numel():
            raise RuntimeError(f"{values.numel()} numbers for parts of {[part.numel() for part in parts]}")
        if self.device.type != "cuda":
            at = 0
            for part in parts:
                part.copy_(values[at:at + part.numel()])
                at += part.numel()
            return
        if torch.cuda.is_current_stream_capturing():       # (a graph would read the buffer again after other copies have written it)
            raise RuntimeError("the host's numbers cannot be copied to the device while the current stream is captured")
        size = values.numel() * values.element_size()
        with self._lock:
            if not self._buffers:
                block = torch.empty(self.BUFFERS * self.BUFFER_BYTES, dtype=torch.uint8, pin_memory=True)
                self._buffers = list(block.split(self.BUFFER_BYTES))
                self._done = [None] * self.BUFFERS
            i = self._next
            self._next = (i + 1) % self.BUFFERS
            if self._done[i] is None:
                self._done[i] = torch.cuda.Event()
            else:
                self._done[i].synchronize()
            if size > self._buffers[i].numel():
                self._buffers[i] = torch.empty(1 << (size - 1).bit_length(), dtype=torch.uint8, pin_memory=True)
            host = self._buffers[i][:size].view(values.dtype)
            host.copy_(values)
            at = 0
            try:
                for part in parts:
                    part.copy_(host[at:at + part.numel()], non_blocking=True)
                    at += part.numel()
            finally:                       # also where a part has refused its numbers: those before it are on their way
                self._done[i].record(torch.cuda.current_stream(self.device))
