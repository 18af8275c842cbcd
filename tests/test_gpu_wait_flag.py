"""Whose call reports a bounded device-side wait that ran out, with several calls in flight.  The wait is the self-test's (one thread on a barrier
of its own, limit 1 ms); the engine runs on kernels without waits (SIMT GEMMs, mma.sync attention), so that nothing gives up half-way."""
import time

import numpy as np
import pytest

from helpers import make_pair, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture
def pair(monkeypatch):
    monkeypatch.setenv("PHX_GEMM", "simt")
    monkeypatch.setenv("PHX_ATTN", "mma")
    ocfg, w, rows_fn, eng = make_pair(max_batch=4)
    eng.set_wait_limit_us(1000)
    inputs = [to_inputs(po.make_batch(ocfg, 4, seed=s, ragged=True)) for s in (3, 4)]
    yield eng, inputs, [eng.rank(i).log_probs.copy() for i in inputs]
    eng.close()


def timed_out(call, *args):
    import x_algorithm_b200 as px
    with pytest.raises(px.PhoenixError) as ei:
        call(*args)
    assert ei.value.status == 4 and "bounded device-side wait" in ei.value.message


def test_a_request_in_front_of_the_wait_is_good(pair):
    """The flag goes up behind a pipelined request's forward, before it is collected: its results are good, and whoever enqueued the wait still
    gets word of it."""
    eng, inputs, want = pair
    eng.rank_submit(inputs[0], 0)
    eng.wait_selftest_async()
    time.sleep(0.05)
    np.testing.assert_array_equal(eng.rank_collect(0).log_probs, want[0])
    timed_out(eng.sync)
    eng.sync()


def test_every_request_behind_the_wait_reports_it(pair):
    """Collecting the first one clears the flag; the second one's forward had met it all the same, and so had the device-buffer calls."""
    eng, inputs, want = pair
    eng.rank_submit(inputs[1], 1)
    eng.wait_selftest_async()
    eng.rank_submit(inputs[0], 0)
    np.testing.assert_array_equal(eng.rank_collect(1).log_probs, want[1])
    eng.rank_submit(inputs[1], 1)
    timed_out(eng.rank_collect, 0)
    timed_out(eng.rank_collect, 1)
    for slot in (0, 1):                                    # both slots work on
        eng.rank_submit(inputs[slot], slot)
    for slot in (0, 1):
        np.testing.assert_array_equal(eng.rank_collect(slot).log_probs, want[slot])
    timed_out(eng.sync)
    eng.sync()


def test_a_blocking_call_does_not_take_another_ones_report(pair):
    eng, inputs, want = pair
    eng.wait_selftest_async()
    eng.rank_submit(inputs[0], 0)
    timed_out(eng.rank, inputs[1])                         # its forward ran with the flag up
    np.testing.assert_array_equal(eng.rank(inputs[1]).log_probs, want[1])
    timed_out(eng.rank_collect, 0)
    timed_out(eng.sync)
    eng.sync()
    np.testing.assert_array_equal(eng.rank(inputs[0]).log_probs, want[0])
    eng.sync()
