"""How far the run loops send steps before they look at the control block
(fcab_steps_ahead): steps sent past the end of a run or past a pause do nothing
but cost a launch each, so no more than a chunk of them may be sent."""
import pytest

from floodca_b200.lib import core


def _simulate(max_steps, t_end, dts, dt_max, pause_every=0, chunk0=32, cap=256):
    """A run loop on a clock: steps of dts (cycled) until max_steps (0: none)
    or t_end, pausing every pause_every steps. Returns the steps taken, the
    steps sent and the polls."""
    t, step, sent, polls, chunk = 0.0, 0, 0, 0, chunk0
    while True:
        n = core().fcab_steps_ahead(max_steps, step, t, t_end, dt_max, pause_every, chunk)
        assert n >= 1
        sent += n
        for _ in range(n):
            if (max_steps and step >= max_steps) or t >= t_end:
                break
            t = min(t + dts[step % len(dts)], t_end)
            step += 1
            if pause_every and step % pause_every == 0:
                break
        polls += 1
        if (max_steps and step >= max_steps) or t >= t_end:
            return step, sent, polls
        chunk = chunk0 if pause_every and step % pause_every == 0 else min(2 * chunk, cap)


@pytest.mark.parametrize("dts", [[60.0], [7.0], [0.01, 3.0], [60.0, 1.0, 1.0]])
@pytest.mark.parametrize("max_steps,t_end", [(0, 600.0), (10**6, 600.0), (10**6, 86400.0), (142, 600.0),
                                             (400, 864000.0), (70000, 1e8)])
def test_few_steps_go_past_the_end(max_steps, t_end, dts):
    step, sent, _ = _simulate(max_steps, t_end, dts, 60.0)
    assert step <= sent < step + 256
    if max_steps and step == max_steps:
        assert sent == step


def test_fixed_counts_far_from_the_end_go_out_whole():
    assert _simulate(400, 864000.0, [5.0], 60.0) == (400, 400, 1)
    assert _simulate(14400, 864000.0, [60.0], 60.0) == (14400, 14400, 1)
    n = core().fcab_steps_ahead
    assert n(10**9, 0, 0.0, 1e300, 1e-300, 0, 32) == 65536  # bounded, whatever the clock
    assert n(10, 10, 5.0, 1.0, 60.0, 0, 32) == 1            # past both ends


@pytest.mark.parametrize("every", [1, 10, 32, 100, 1000])
@pytest.mark.parametrize("max_steps,t_end", [(400, 864000.0), (2005, 864000.0), (10**6, 3000.0), (0, 3000.0)])
def test_no_step_goes_past_a_pause(every, max_steps, t_end):
    step, sent, polls = _simulate(max_steps, t_end, [5.0], 60.0, pause_every=every)
    if max_steps and step == max_steps:
        assert (sent, polls) == (step, -(-step // every))
    else:
        assert sent < step + 256
