"""Many simulations stepped together (phono_batch_* of include/phono.h).

A ``Batch`` holds up to ``capacity`` device simulations of one arithmetic
scheme.  Every instance runs its own step kernels on a worker stream, so that
the instances' launches run side by side on the GPU; each instance replays
its own 12-step graph (captured when it joins) and does not wait for the
others between chunks.  Two schemes:

* ``streams=0``, the default: up to 64 workers; FP32 instances step in tiles
  the batch picks from what all of them amount to, whatever shape they were
  made with (their ``tile_j`` has to be the batch's);
* ``streams=W``: W workers; an instance made with a tile shape keeps it.

Instances keep their own step counters and budgets, so a batch can hold
simulations of different sizes at different points of their runs, and instances can join
and leave between calls.  Results are those of stepping each alone.
"""
from __future__ import annotations

import ctypes

from . import _lib
from ._lib import check


class Batch:
    def __init__(self, capacity, precision="f32k", tile_j=8, streams=0):
        L = _lib.load()
        self._L = L
        self.precision = precision
        self.tile_j = int(tile_j)
        self.streams = int(streams)
        b = ctypes.c_void_p()
        check(L.phono_batch_create(int(capacity), _lib.PRECISIONS[precision], self.tile_j, ctypes.byref(b)))
        self._b = b
        if self.streams:
            try:
                check(L.phono_batch_set_mode(b, _lib.BATCH_STREAMS, self.streams))
            except Exception:
                L.phono_batch_destroy(b)
                self._b = None
                raise
        self._members = {}  # slot -> DeviceSimulation (kept alive while in the batch)

    def add(self, sim, nsteps):
        """Attach a DeviceSimulation for nsteps more steps; returns its slot."""
        if sim.precision != self.precision:
            raise ValueError("simulation precision differs from the batch")
        rc = self._L.phono_batch_add(self._b, sim._h, int(nsteps))
        if rc < 0:
            check(rc)
        self._members[rc] = sim
        return rc

    def remove(self, slot):
        check(self._L.phono_batch_remove(self._b, int(slot)))
        return self._members.pop(slot)

    def remaining(self, slot):
        rc = self._L.phono_batch_remaining(self._b, int(slot))
        if rc < 0:
            check(rc)
        return rc

    def step(self, nsteps):
        check(self._L.phono_batch_step(self._b, int(nsteps)))

    def sync(self):
        check(self._L.phono_batch_sync(self._b))

    def last_step_ms(self):
        ms = ctypes.c_float()
        check(self._L.phono_batch_last_step_ms(self._b, ctypes.byref(ms)))
        return float(ms.value)

    @property
    def members(self):
        return dict(self._members)

    def close(self):
        if getattr(self, "_b", None):
            self._L.phono_batch_destroy(self._b)
            self._b = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.close()
