"""What flush() goes by: passes that found every frame acknowledged."""
import random

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


@pytest.mark.parametrize("in_flight", [1, 2, 3, 4])
@pytest.mark.parametrize("windows", [1, 2])
def test_settled_means_a_pass_that_has_looked_and_found_nothing(windows, in_flight):
    """What a launch counts may be read along with what launches before it counted, up to the number in flight: made-up
    launches, each read at some time between its own end and the end of the last that can have been begun by then."""
    rng, settled = random.Random(10 * windows + in_flight), 0
    for _ in range(3000):
        w = _native.cuda().QuietWatch()
        w.begin()
        launches = [rng.choice(("work", "cut short", "open") + 3 * ("nothing",)) for _ in range(14)]
        seen = 0    # launches whose counts have been read
        for i in range(len(launches) - in_flight + 1):
            ended = rng.randint(max(seen, i + 1), i + in_flight)
            counted, seen = launches[seen:ended], ended
            w.launched()
            w.looked("work" in counted, "cut short" in counted, i, "open" in counted)
            if w.settled(0, windows, in_flight - 1, False):
                settled += 1
                assert launches[i + 1 - windows:i + 1] == ["nothing"] * windows
            if w.settled(0, windows, in_flight - 1, True):
                assert set(launches[i + 1 - windows:i + 1]) <= {"nothing", "open"}
    assert settled > 100


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
