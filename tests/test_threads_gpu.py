"""Other Python threads run while a call waits for the device: the interpreter lock is not held over launches."""
import threading
import time

import pytest
import torch

from openkimi_b200 import KimiDeltaAttention, chunk_kda, recurrent_kda_step
from tests.test_call_arguments import FUSED, _inputs

pytestmark = pytest.mark.gpu


def _call(kind):
    if kind == "step":
        x, s = _inputs(1), torch.zeros(1, 2, 128, 128, device="cuda")
        return lambda: recurrent_kda_step(**x, state=s, inplace=True, **FUSED)
    if kind == "chunk":
        x = _inputs(1, 64)
        return lambda: chunk_kda(**x, **FUSED)
    mod, x = KimiDeltaAttention(128, 1).cuda().bfloat16(), torch.zeros(1, 64, 128, device="cuda", dtype=torch.bfloat16)
    return lambda: mod(x)


@pytest.mark.parametrize("kind", ["step", "chunk", "layer"])
def test_a_waiting_call_leaves_the_interpreter_free(kind):
    """The device is kept busy for about a second; launches are issued until the queue is full and one of them waits."""
    call = _call(kind)
    with torch.no_grad():
        call()
        torch.cuda.synchronize()
        stop, gap = threading.Event(), [0.0]

        def watch():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(1e-3)
                now = time.perf_counter()
                gap[0], last = max(gap[0], now - last), now

        t = threading.Thread(target=watch)
        t.start()
        try:
            torch.cuda._sleep(2_000_000_000)
            done = torch.cuda.Event()
            done.record()
            longest = 0.0
            while longest < 0.3 and not done.query():
                begin = time.perf_counter()
                call()
                longest = max(longest, time.perf_counter() - begin)
        finally:
            stop.set()
            t.join()
            torch.cuda.synchronize()
    if longest < 0.3:
        pytest.skip("no call had to wait")
    assert gap[0] < 0.5 * longest, (gap[0], longest)


def test_threads_with_their_own_streams():
    """Calls of several threads at once give what one thread gives."""
    x = [_inputs(2, 200) for _ in range(4)]
    with torch.no_grad():
        want = [chunk_kda(**i, **FUSED)[0] for i in x]
    torch.cuda.synchronize()
    got = [None] * len(x)

    def work(n):
        s = torch.cuda.Stream()
        with torch.no_grad(), torch.cuda.stream(s):
            for _ in range(20):
                o = chunk_kda(**x[n], **FUSED)[0]
        s.synchronize()
        got[n] = o

    threads = [threading.Thread(target=work, args=(n,)) for n in range(len(x))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
