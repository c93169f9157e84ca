"""What flush() goes by: launches of the engine thread that found nothing to do, and for how long."""
from sharedtensor_b200 import _native


def _watch(*looked):
    w = _native.cuda().QuietWatch()
    w.begin()
    for args in looked:
        w.launched()
        w.looked(*args)
    return w


def test_work_found_after_the_clock_was_read_is_not_a_long_quiet_time():
    w = _watch((False, False, 1000), (True, False, 5000))
    assert w.quiet_for(500, 4000) == 0, "the launch that found work was looked at after the caller took the time"
    assert w.quiet_for(6000, 4000) == 0
    assert w.quiet_for(500, 7000) == 2000
    assert w.quiet_for(6500, 7000) == 500


def test_quiet_launches_begin_after_the_caller_and_after_the_last_busy_one():
    w = _watch(*((False, False, t) for t in (1, 2, 3)))
    assert w.quiet_launches(0, 3) and not w.quiet_launches(1, 3)
    w.launched()
    w.looked(True, False, 4)
    assert not w.quiet_launches(0, 1)
    for t in (5, 6, 7):
        assert not w.quiet_launches(0, 3)
        w.launched()
        w.looked(False, False, t)
    assert w.quiet_launches(0, 3) and w.launches() == 7


def test_a_launch_that_did_not_get_to_look_does_not_count():
    """An update that wants the SMs makes groups leave before they have looked at their tiles; a wait that runs out too."""
    w = _watch(*((False, True, t) for t in (1, 2, 3)))
    assert not w.quiet_launches(0, 1) and w.quiet_for(0, 10) == 7
    w.launched()
    w.looked(False, False, 4)
    assert w.quiet_launches(0, 1) and not w.quiet_launches(0, 2)


def test_any_timeout_can_be_given():
    from sharedtensor_b200.parallel.gpu_backend import _milliseconds

    assert _milliseconds(0.25) == 250 and _milliseconds(30) == 30000
    assert _milliseconds(0.0) == _milliseconds(-1.0) == _milliseconds(float("nan")) == 0
    assert 0 < _milliseconds(float("inf")) == _milliseconds(1e300) < 2 ** 63
