"""What flush() goes by: passes that found every frame acknowledged."""
import pytest
import torch

from sharedtensor_b200 import _native
from sharedtensor_b200.parallel.local_wiring import connect_local


def test_a_launch_that_found_open_frames_starts_the_count_anew():
    w = _native.cuda().QuietWatch()
    w.begin()
    for k, still_open in enumerate((False, True, False, False)):
        w.launched()
        w.looked(False, False, k, still_open)
        assert w.acknowledged(1) == (not still_open)
    assert w.acknowledged(2) and not w.acknowledged(3)
    assert w.quiet_launches(0, 4), "open frames are no work"


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 100_001])
def test_no_flush_before_the_neighbour_has_taken_the_frames_in(n):
    """The neighbour's rounds are made by hand: until it makes one, only the tenth of a second ends the flush."""
    cu = _native.cuda()
    a, b = cu.GpuReplica(0, n, cu.GpuConfig()), cu.GpuReplica(0, n, cu.GpuConfig())
    connect_local(a, b)
    here = torch.cuda.current_stream().cuda_stream
    delta = torch.randn(n, device="cuda") * 1e-3
    a.start_engine()
    try:
        a.add(delta.data_ptr(), here)
        assert not a.flush(here, 60)
        for _ in range(4):
            b.round()
            b.sync()
        assert a.flush(here, 5000)
    finally:
        a.stop_engine()
