"""Which form recorded steps are read back in (lists made on the device, or bitmaps that the host expands): the spikes
are the same, and neither a few words nor dense steps pay for the lists' kernels."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _backend(n):
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    pop, proj, chan = (T.uid_from_int(6600 + i) for i in range(3))
    b = GB300Backend()
    b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))])
    b.generate_projection(proj, T.NULL_UID, pop, T.GEN_ONE_TO_ONE, n, n, 256, 256, 1, 1, 1, 1)
    b.subscribe(proj, [chan])
    b.record_spikes(pop)
    b._init()
    return b, pop, chan


# One step at a time and four, around 8192 words a read and the 1024 words of a segment, a tenth of the neurons
# firing and a hundredth in turn: lists, given-up lists, bitmaps after them, and lists again.
@pytest.mark.parametrize("n", [32737, 65536, 262112, 262145, 600001])
@pytest.mark.parametrize("window", [1, 4])
def test_sparse_and_dense_windows_in_turn(n, window):
    from knp_gb300 import network as N

    b, pop, chan = _backend(n)
    rng = np.random.default_rng(n)
    rates = [0.01, 0.1, 0.1, 0.01, 0.01, 0.1, 0.01]
    trains = [np.flatnonzero(rng.random(n) < r).astype(np.uint32) for r in rates for _ in range(window)]
    offs = np.concatenate([[0], np.cumsum([t.size for t in trains])]).astype(np.int64)
    b.load_spike_schedule(N.SpikeSchedule(chan, offs, np.concatenate(trains)))
    b.step(1)
    for first in range(0, len(trains), window):
        b.step(window)
        b.synchronize()
        for t in range(first, first + window):
            np.testing.assert_array_equal(b.spikes(pop, t + 1), trains[t], err_msg=f"step {t + 1}")
    b.close()


def test_one_step_of_few_words_does_not_pay_for_lists():
    """A population one word past the size from which lists are made reads a step in about the time of one below it
    (17 us and 16; 30 with lists)."""
    times = []
    for n in (32000, 40000):
        b, pop, chan = _backend(n)
        b.generate_bernoulli_schedule(chan, n, 0.005, 0, 300, 3)
        out = np.zeros(n, np.uint32)
        took = []
        for t in range(300):
            b._step()
            b.synchronize()
            t0 = time.perf_counter()
            b.spikes_capped(pop, t, out)
            took.append(time.perf_counter() - t0)
        times.append(np.median(took[20:]))
        b.close()
    assert times[1] < 1.4 * times[0], times


def test_a_read_of_an_early_step_leaves_most_of_a_long_window_for_later():
    """600 steps of 200000 neurons (15 MB of bitmaps): the first step's read takes less than what is left then."""
    n, steps = 200000, 600
    b, pop, chan = _backend(n)
    out = np.zeros(n, np.uint32)
    first, rest = [], []
    for w in range(3):
        t = b.get_step()
        b.generate_bernoulli_schedule(chan, n, 0.005, t, steps, 3 + w)
        b.step(steps)
        b.synchronize()
        t0 = time.perf_counter()
        n_first = b.spikes_capped(pop, t + 1, out)
        t1 = time.perf_counter()
        b.spikes_capped(pop, t + steps - 1, out)
        t2 = time.perf_counter()
        first.append(t1 - t0)
        rest.append(t2 - t1)
        assert 0 < n_first < 0.01 * n
        for k in (2, 90, 99, 100, 101, 102, 103, 300, steps - 1):  # either side of what the first read brought
            assert 0 < b.spikes_capped(pop, t + k, out) < 0.01 * n
        b.discard_spikes(t + steps)
    assert min(first) < min(rest), (first, rest)
    b.close()
