"""The loop of lsh_run_until (lsh_run_until.h) over a clock that fails on request: the device's record is never taken
back behind the steps that were launched."""
import ctypes

import pytest

from adj_cases import native_lib


def run(dt, t_end, max_steps=0, most=8, fail_step=0, fail_read=0, stuck=0):
    lib = native_lib("run_until_host")
    out = (ctypes.c_double * 6)()
    st = lib.rununtil(ctypes.c_double(dt), ctypes.c_double(t_end), ctypes.c_longlong(max_steps), most, fail_step, fail_read,
                      stuck, out)
    return st, dict(zip(("t", "steps", "t_end", "done", "steps_done", "launched"), out))


@pytest.mark.parametrize("t_end,max_steps,steps", [(2.5, 0, 10), (2.4, 0, 10), (100.0, 21, 21), (0.0, 0, 0), (1e9, 5, 5)])
def test_runs_to_the_end(t_end, max_steps, steps):
    st, r = run(0.25, t_end, max_steps)
    assert st == 0 and r["steps"] == r["steps_done"] == steps and r["t"] == 0.25 * steps
    assert r["launched"] == steps  # none past the end
    assert r["t_end"] == float("inf") and r["done"] == 0


def test_a_failed_launch_leaves_the_clock_with_the_state():
    # 8 steps, then 4 of the next 8
    st, r = run(0.25, 100.0, fail_step=2)
    assert st == 7 and r["steps"] == 12 and r["t"] == 3.0 and r["steps_done"] == 12
    assert r["t_end"] == float("inf") and r["done"] == 0  # steps go on


def test_a_failed_reading_leaves_the_clock_with_the_state():
    # readings: at the start, then after each 8 steps
    st, r = run(0.25, 100.0, fail_read=3)
    assert st == 7 and r["steps"] == 16 and r["t"] == 4.0 and r["steps_done"] == 16


def test_a_device_that_no_longer_answers_is_not_written():
    st, r = run(0.25, 100.0, fail_read=3, stuck=1)
    assert st == 7 and r["steps"] == 16 and r["t"] == 4.0
