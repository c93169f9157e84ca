"""flush() on a pair of replicas in one process, engine threads running."""
import pytest
import torch

import sharedtensor

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
