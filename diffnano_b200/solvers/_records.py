"""Room for curl records: the curl terms of all steps of a run, kept from its forward to
its reverse sweep in place of checkpoints and replay.

All records alive on a GPU (one per differentiated solve whose backward is still to
come, one per ``FDTDBatch2D`` that differentiates) share an eighth of its memory, and
beyond a 64th of it one takes, with the arrays of its own sweep, what the allocator has
in reserve or at most half of what is free: a program that holds many graphs, or that
fills the GPU with other tensors, gets checkpoints instead and room for them.  (To ask the
driver what is free costs the host 70 - 170 us, the allocator 9; a whole gradient of 300 x
413 cells over 600 steps takes 3 ms: small records go without.)
"""

from __future__ import annotations

import threading
import weakref

import torch

RECORD_SHARE = 1 / 8  # of the GPU's memory, for all records alive
UNASKED_SHARE = 1 / 64  # up to which nobody asks what is free

_lock = threading.RLock()
_live: weakref.WeakSet = weakref.WeakSet()


class Record:
    """What ``make()`` returned, counted until the object is dropped."""

    def __init__(self, device, nbytes: int, made):
        self.device, self.nbytes, self.made = device, nbytes, made


def is_room(device, nbytes: int) -> bool:
    """Whether the allocator has so much in reserve (memory given back to it and not to
    the GPU), or the GPU and its reserve twice as much."""
    stats = torch.cuda.memory_stats_as_nested_dict(device)
    reserve = stats["reserved_bytes"]["all"]["current"] - stats["allocated_bytes"]["all"]["current"]
    return reserve >= nbytes or torch.cuda.mem_get_info(device)[0] + reserve >= 2 * nbytes


def claim(device, nbytes: int, beside: int, make):
    """A ``Record`` of ``make()``, which allocates ``nbytes``, or None where there is no
    room; ``beside``: bytes of the other arrays that the run and its sweep still need."""
    total = torch.cuda.get_device_properties(device).total_memory
    with _lock:
        held = nbytes + sum(r.nbytes for r in _live if r.device == device)
        if held > RECORD_SHARE * total or (held > UNASKED_SHARE * total and
                                           not is_room(device, nbytes + beside)):
            return None
        try:
            record = Record(device, nbytes, make())
        except torch.OutOfMemoryError:
            return None
        _live.add(record)
        return record
