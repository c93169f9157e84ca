"""flush() on a pair of replicas in one process, engine threads running."""
import threading
import time

import pytest
import torch

import sharedtensor
from sharedtensor_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 100_001, 40_000_000])
def test_flush_waits_until_an_update_has_arrived(free_port, n):
    """One tile, a few tiles per group, several windows."""
    init = torch.randn(n, device="cuda")
    a = sharedtensor.createOrFetch("127.0.0.1", free_port, init, rejoin=False)
    b = sharedtensor.createOrFetch("127.0.0.1", free_port, torch.zeros(n, device="cuda"), rejoin=False)
    try:
        expect, out = init.clone(), torch.empty_like(init)
        for i in range(20):
            d = torch.randn(n, device="cuda") * 1e-2
            src, dst = (a, b) if i % 2 == 0 else (b, a)
            src.addFromTensor(d)
            expect += d
            assert src.flush(10.0) and dst.flush(10.0)
            dst.copyToTensor(out)
            assert ((out - expect).norm() / expect.norm()).item() < 1e-5
    finally:
        b.close()
        a.close()


def test_flush_while_another_thread_reads_all_the_time(free_port):
    """Every read asks the round kernel for its SMs, so that its launches keep leaving before they have looked at their
    tiles: flush() does not take that for silence."""
    n = 20_000_000
    init = torch.randn(n, device="cuda")
    a = sharedtensor.createOrFetch("127.0.0.1", free_port, init, rejoin=False)
    b = sharedtensor.createOrFetch("127.0.0.1", free_port, torch.zeros(n, device="cuda"), rejoin=False)
    stop = threading.Event()

    def read():
        mine = torch.empty(n, device="cuda")
        with torch.cuda.stream(torch.cuda.Stream()):
            while not stop.is_set():
                for _ in range(8):
                    a.copyToTensor(mine)
                torch.cuda.current_stream().synchronize()

    reader = threading.Thread(target=read)
    try:
        assert a.flush(10.0) and b.flush(10.0)
        reader.start()
        expect, out = init.clone(), torch.empty_like(init)
        for i in range(12):
            d = torch.randn(n, device="cuda") * 1e-2
            a.addFromTensor(d)
            expect += d
            if not a.flush(2.0):
                continue
            b.copyToTensor(out)
            assert ((out - expect).norm() / expect.norm()).item() < 1e-5, i
        stop.set()
        reader.join()
        assert a.flush(10.0) and b.flush(10.0)
        b.copyToTensor(out)
        assert ((out - expect).norm() / expect.norm()).item() < 1e-5
    finally:
        stop.set()
        b.close()
        a.close()


def test_flush_keeps_to_its_timeout(free_port):
    """Any limit can be given, infinity among them, and it covers what the caller has queued and another thread's flush."""
    n = 1000
    a = sharedtensor.createOrFetch("127.0.0.1", free_port, torch.zeros(n, device="cuda"), rejoin=False)
    b = sharedtensor.createOrFetch("127.0.0.1", free_port, torch.zeros(n, device="cuda"), rejoin=False)
    try:
        a.addFromTensor(torch.ones(n, device="cuda"))
        assert a.flush(float("inf")) and a.flush(1e12)
        assert not a.flush(0.0) and not a.flush(-1.0) and not a.flush(float("nan"))
        busy = torch.cuda.Stream()
        with torch.cuda.stream(busy):
            _native.cuda().delay(1_000_000_000, busy.cuda_stream)   # a second of queued work
            t0 = time.time()
            other = threading.Thread(target=lambda: torch.cuda.set_stream(busy) or a.flush(5.0))
            other.start()
            time.sleep(0.05)
            assert not a.flush(0.1)
            assert time.time() - t0 < 0.5
            assert a.flush(5.0)
            other.join()
    finally:
        b.close()
        a.close()
