"""Whole relaxation solves as one native call (``ffx_relax_cycles``).

A ``Relaxation`` holds the plan of one grid hierarchy: V-cycles, or with a
single level weighted Jacobi sweeps. Grids that fit the SMs' shared memory
(128^3 and less) run in one cooperative launch with the iterate resident on
the chip; larger ones several sweeps per launch.
"""
import ctypes as C

import torch

from .. import _native as N


class Relaxation:
    def __init__(self, device, shapes, extent, omega, *, pre=1, post=1, last=1, basis=None, classes=None):
        self.device = device
        self._keep = (basis, classes)
        plan = self.plan = N.FfxRelaxPlan()
        plan.count, plan.pre, plan.post, plan.last_sweeps, plan.omega = len(shapes), pre, post, last, omega
        plan.basis = basis.data_ptr() if basis is not None else None
        plan.classes = classes.data_ptr() if classes is not None else None
        for slot, shape in zip(plan.level, shapes):
            slot.grid = N.FfxRelaxGrid(N.n3(*shape), N.f3(*[n / e for n, e in zip(shape, extent)]))
        N.check(device.lib.ffx_relax_plan(C.byref(plan)))
        self.resident = plan.tail == 0 or plan.tile[0] > 0
        self.workspace = None
        self._levels = []
        with device.ordered():
            if plan.workspace_bytes:
                self.workspace = torch.zeros(plan.workspace_bytes, dtype=torch.uint8, device=device.device)
                plan.workspace = self.workspace.data_ptr()
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

    def run(self, p, q, rhs, cycles, dt, from_zero):
        """Relax ``p`` (``q`` its second buffer); returns (iterate, other buffer)."""
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
