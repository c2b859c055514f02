"""The page of alarm words is made once, however many threads ask for the first."""
import threading

import torch

from fluxfx_b200.backend import relax


def test_one_page_for_all_threads(monkeypatch):
    made = []
    start = threading.Barrier(8)
    zeros = torch.zeros

    def slow_zeros(*args, **kwargs):
        kwargs.pop('pin_memory')        # (there is no device here)
        made.append(1)
        threading.Event().wait(0.05)
        return zeros(*args, **kwargs)

    monkeypatch.setattr(relax, '_page', None)
    monkeypatch.setattr(relax.torch, 'zeros', slow_zeros)
    alarms = []

    def take():
        start.wait()
        alarms.append(relax.Alarm())

    threads = [threading.Thread(target=take) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1
    first, size = relax._page.data_ptr(), 4 * relax._WORDS
    addresses = {a.address for a in alarms}
    assert len(addresses) == 8 and all(first <= a < first + size for a in addresses)
