"""A batched plan made and run on a stream of its own while another thread keeps the
default stream busy: the plan's memory is ready before the first step, whatever the
default stream has queued."""
import threading

import pytest
import torch

from fluxfx_b200.backend.batched import BatchedSmoke, batched_scenes, build_solvers

pytestmark = pytest.mark.gpu


def run(device, steps=2):
    solvers, sources = build_solvers(batched_scenes(3, seed=3, sizes=(32, 48)), device)
    batch = BatchedSmoke(solvers, sources)
    batch.run(steps)
    stats = batch.stats()       # raises when a wait gave up
    fields = [[f.clone() for f in (d, t, *v)] for d, t, v in (batch.fields(i) for i in range(len(solvers)))]
    device.synchronize()
    batch.close()
    return fields, [s['total_cycles'] for s in stats]


def test_the_default_stream_may_be_busy():
    from fluxfx_b200.backend.device import CudaDevice
    want, cycles = run(CudaDevice())
    stop = threading.Event()

    def busy():
        for _ in range(400):        # some milliseconds each, two at most in the queue
            if stop.is_set():
                return
            torch.cuda._sleep(5_000_000)
            torch.cuda._sleep(5_000_000)
            torch.cuda.default_stream().synchronize()

    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    thread = threading.Thread(target=busy)
    thread.start()
    try:
        with torch.cuda.stream(side):
            for _ in range(5):
                got, counts = run(CudaDevice(stream=side))
                assert counts == cycles
                assert all(torch.equal(a, b) for x, y in zip(got, want) for a, b in zip(x, y))
    finally:
        stop.set()
        thread.join()
