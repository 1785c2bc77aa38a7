"""Kernels whose dynamic shared memory differs from network to network: what is built later and
needs less takes nothing from what was built before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _network(b, n_src, n, fan_in, d_src, small_first, steps, mode, threshold, seed=3):
    """n_src driven sources -> n neurons (delays 1 .. d_src, a gather of many bitmaps), and n -> n at delay 1 (one
    bitmap), loaded in either order."""
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    src, pop, drive, wide, rec, chan = (T.uid_from_int(6100 + i) for i in range(6))
    b.load_populations([N.Population(src, T.BLIFAT, T.blifat_defaults(n_src)),
                        N.Population(pop, T.BLIFAT, T.blifat_defaults(n))])
    b.generate_projection(drive, T.NULL_UID, src, T.GEN_ONE_TO_ONE, n_src, n_src, 256, 256, 1, 1, seed, 10)
    parts = [lambda: b.generate_fixed_fan_in_projection(wide, src, pop, n_src, n, fan_in, -32, 32, 1, d_src, seed, 20),
             lambda: b.generate_fixed_fan_in_projection(rec, pop, pop, n, n, fan_in, -32, 32, 1, 1, seed, 30)]
    for part in parts[::-1] if small_first else parts:
        part()
    b.subscribe(drive, [chan])
    b.record_spikes(pop)
    for p in (wide, rec):
        b.set_pull_threshold(p, threshold)
    b.set_step_mode(mode)
    b._init()
    b.generate_bernoulli_schedule(chan, n_src, 0.3, 0, steps, seed)
    return pop


def _trains(b, pop, steps):
    b.step(steps)
    return [b.spikes(pop, t) for t in range(b.get_step() - steps, b.get_step())]


@pytest.mark.parametrize("small_first", [False, True])
def test_gathers_of_different_shared_memory_in_one_network(small_first):
    from knp_gb300 import GB300Backend
    from knp_gb300 import types as T

    steps = 12
    trains = []
    for mode, threshold in ((T.STEP_GRID, -1.0), (T.STEP_PHASES, 0.0), (T.STEP_GRID, 0.0)):
        with GB300Backend() as b:
            pop = _network(b, 200000, 3000, 400, 20, small_first, steps, mode, threshold)
            trains.append(_trains(b, pop, steps))
    assert sum(s.size for s in trains[0]) > 0
    for got in trains[1:]:
        for x, y in zip(got, trains[0]):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("mode", ["STEP_GRID", "STEP_PHASES"])
def test_a_smaller_backend_built_later_leaves_the_larger_one_running(mode):
    from knp_gb300 import GB300Backend
    from knp_gb300 import types as T

    with GB300Backend() as large, GB300Backend() as alone, GB300Backend() as small:
        pop = _network(alone, 200000, 3000, 400, 20, False, 20, getattr(T, mode), 0.0)
        ref = _trains(alone, pop, 20)
        _network(large, 200000, 3000, 400, 20, False, 20, getattr(T, mode), 0.0)
        got = _trains(large, pop, 10)
        small_pop = _network(small, 100000, 3000, 400, 6, False, 10, getattr(T, mode), 0.0)
        _trains(small, small_pop, 10)
        got += _trains(large, pop, 10)
    for x, y in zip(got, ref):
        np.testing.assert_array_equal(x, y)
