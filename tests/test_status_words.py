"""One status word per device, however many threads make their first call at once."""
import threading
import time

import torch

from openkimi_b200 import ops


def test_threads_share_one_word():
    class Slow(ops._DeviceStatus):
        _per_device = {}

        def __init__(self, device):
            time.sleep(0.05)  # as long as making the words in device and pinned memory may take

    got, start = [], threading.Barrier(8)

    def first_call():
        start.wait()
        got.append(Slow.get(torch.device("cuda", 0)))

    threads = [threading.Thread(target=first_call) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 8 and all(st is got[0] for st in got)
