"""Whole relaxation solves as one native call (``ffx_relax_cycles``).

A ``Relaxation`` holds the plan of one grid hierarchy: V-cycles, or with a
single level weighted Jacobi sweeps. Grids that fit the SMs' shared memory
(128^3 and less) run in one cooperative launch with the iterate resident on
the chip; larger ones several sweeps per launch.
"""
import ctypes as C
import itertools
import threading

import torch

from .. import _native as N


_WORDS = 4096
_page = None
_lock = threading.Lock()
_taken = itertools.count()


class Alarm:
    """A word of host memory that a solve's launch sets when one of its bounded waits
    gives up (the GPU was held up for seconds): looking at it costs the host nothing
    and waits for nothing.

    The words are one pinned page of the process, taken in turn and never freed, so
    that a launch that outlives its solver writes into no one else's memory. Past
    4096 solvers a word has a second owner, whom an alarm then reaches as well."""

    def __init__(self):
        global _page
        with _lock:
            if _page is None:
                _page = torch.zeros(_WORDS, dtype=torch.int32, pin_memory=True)
        self.address = _page.data_ptr() + 4 * (next(_taken) % _WORDS)
        self._view = C.c_int32.from_address(self.address)

    def check(self, device, reset):
        """Raises FFX_ERR_TIMEOUT when a wait gave up since the last look; ``reset``
        then makes the workspace as new, so that later solves are right."""
        if self._view.value:
            device.synchronize()
            reset()
            device.synchronize()
            self._view.value = 0
            raise N.FfxError(N.FFX_ERR_TIMEOUT, 'a bounded wait of a pressure solve gave up: its pressure is wrong')


class Relaxation:
    def __init__(self, device, shapes, extent, omega, *, pre=1, post=1, last=1, basis=None, classes=None, sms=0):
        self.device = device
        self._keep = (basis, classes)
        plan = self.plan = N.FfxRelaxPlan()
        plan.count, plan.pre, plan.post, plan.last_sweeps, plan.omega = len(shapes), pre, post, last, omega
        plan.sms = sms
        plan.basis = basis.data_ptr() if basis is not None else None
        plan.classes = classes.data_ptr() if classes is not None else None
        for slot, shape in zip(plan.level, shapes):
            slot.grid = N.FfxRelaxGrid(N.n3(*shape), N.f3(*[n / e for n, e in zip(shape, extent)]))
        N.check(device.lib.ffx_relax_plan(C.byref(plan)))
        self.resident = plan.tail == 0 or plan.tile[0] > 0
        self.workspace = self.alarm = None
        self._levels = []
        with device.ordered():
            if plan.workspace_bytes:
                self.workspace = torch.zeros(plan.workspace_bytes, dtype=torch.uint8, device=device.device)
                plan.workspace = self.workspace.data_ptr()
                self.alarm = Alarm()
                plan.alarm = self.alarm.address
            if not self.resident:
                for slot, shape in zip(plan.level[1:], shapes[1:]):
                    fields = [device.texture(shape) for _ in range(3)]
                    slot.p, slot.q, slot.rhs = (f.data_ptr() for f in fields)
                    self._levels.append(fields)

    @property
    def allocated_bytes(self):
        fields = sum(4 * f.numel() for level in self._levels for f in level)
        return fields + (self.workspace.numel() if self.workspace is not None else 0)

    def launches(self, cycles):
        """Kernels that ``cycles`` V-cycles launch."""
        plan = self.plan
        if self.resident:
            return 1
        last = plan.count - 1
        one = int(plan.tail < plan.count)
        for slot in plan.level[:min(plan.tail, last)]:
            one += 2 + sum(-(-(n - fused.sweeps) // slot.sweep.sweeps)
                           for n, fused in ((plan.pre, slot.down), (plan.post, slot.up)))
        if plan.tail == plan.count:
            one += -(-plan.last_sweeps // plan.level[last].sweep.sweeps)
        return one * cycles

    def check(self):
        """Raises when a wait of a solve so far gave up."""
        if self.alarm is not None:
            self.alarm.check(self.device, lambda: N.check(
                self.device.lib.ffx_relax_reset(C.byref(self.plan), self.device.s)))

    def run(self, p, q, rhs, cycles, dt, from_zero):
        """Relax ``p`` (``q`` its second buffer); returns (iterate, other buffer)."""
        self.check()
        plan = self.plan
        level = plan.level[0]
        level.p, level.q, level.rhs = p.data_ptr(), q.data_ptr(), rhs.data_ptr()
        swapped = N.i32(0)
        self.device.call('ffx_relax_cycles', C.byref(plan), cycles, dt, int(from_zero), C.byref(swapped),
                         self.device.s)
        self.device.calls += self.launches(cycles) - 1
        return (q, p) if swapped.value else (p, q)

    def timeouts(self):
        """Waits of resident solves that gave up (0 unless the GPU was held up for seconds)."""
        count = N.i32(0)
        N.check(self.device.lib.ffx_relax_timeouts(C.byref(self.plan), C.byref(count), self.device.s))
        return count.value
