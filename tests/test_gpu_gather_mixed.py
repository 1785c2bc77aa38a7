"""Two gathers into one population, one cut over blocks between delays and one in whole windows only (its spike bitmap
takes almost all of a block's shared memory): the same spikes as the scatter gives (dyadic weights)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# A bitmap of 225008 bytes: with one window's accumulators it fits a block, within 8 KB of the limit.
WHOLE_WINDOW_SOURCES = 1800000


def _trains(mode, threshold, whole_first, steps=10):
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    pop, a, b_, chan_a, chan_b = (T.uid_from_int(6300 + i) for i in range(5))
    n, n_cut = 3000, 60000
    with GB300Backend() as b:
        b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(n)),
                            N.Population(a, T.BLIFAT, T.blifat_defaults(WHOLE_WINDOW_SOURCES)),
                            N.Population(b_, T.BLIFAT, T.blifat_defaults(n_cut))])
        for k, (src, size, chan) in enumerate(((a, WHOLE_WINDOW_SOURCES, chan_a), (b_, n_cut, chan_b))):
            drive = T.uid_from_int(6310 + k)
            b.generate_projection(drive, T.NULL_UID, src, T.GEN_ONE_TO_ONE, size, size, 256, 256, 1, 1, 5, 10 + k)
            b.subscribe(drive, [chan])
        parts = [(T.uid_from_int(6320), a, WHOLE_WINDOW_SOURCES, 3), (T.uid_from_int(6321), b_, n_cut, 20)]
        for k, (uid, src, size, d_hi) in enumerate(parts if whole_first else parts[::-1]):
            b.generate_fixed_fan_in_projection(uid, src, pop, size, n, 400, -32, 32, 1, d_hi, 5, 20 + 10 * k)
            b.set_pull_threshold(uid, threshold)
        b.record_spikes(pop)
        b.set_step_mode(mode)
        b._init()
        for uid, *_ in parts if threshold >= 0 else ():
            b.set_pull_threshold(uid, threshold)  # refused for a projection without a gather form
        for chan, size in ((chan_a, WHOLE_WINDOW_SOURCES), (chan_b, n_cut)):
            b.generate_bernoulli_schedule(chan, size, 0.3, 0, steps, 9)
        b.step(steps)
        return [b.spikes(pop, t) for t in range(steps)]


@pytest.mark.parametrize("whole_first", [True, False])
def test_cut_and_whole_window_gathers_into_one_population(whole_first):
    from knp_gb300 import types as T

    ref = _trains(T.STEP_GRID, -1.0, whole_first)
    assert sum(s.size for s in ref) > 0
    for mode in (T.STEP_GRID, T.STEP_PHASES):
        got = _trains(mode, 0.0, whole_first)
        for x, y in zip(got, ref):
            np.testing.assert_array_equal(x, y)
