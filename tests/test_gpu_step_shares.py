"""How the step kernels share out work, at the edges: gathers whose delays come in groups and whose windows
are cut between blocks, and projections of short rows with long ones among them. Dyadic weights: every form
gives the same spikes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _trains(n, fan_in, d_hi, threshold, mode, steps=14, p_in=0.35):
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    pop, rec, inp, chan = (T.uid_from_int(5200 + i) for i in range(4))
    with GB300Backend() as b:
        b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))])
        b.generate_projection(inp, T.NULL_UID, pop, T.GEN_ONE_TO_ONE, n, n, 256, 256, 1, 1, 5, 10)
        b.generate_fixed_fan_in_projection(rec, pop, pop, n, n, fan_in, -32, 32, 1, d_hi, 5, 20)
        b.subscribe(inp, [chan])
        b.record_spikes(pop)
        b.set_pull_threshold(rec, threshold)
        b.set_step_mode(mode)
        b._init()
        b.generate_bernoulli_schedule(chan, n, p_in, 0, steps, 9)
        b.step(steps)
        return [b.spikes(pop, t) for t in range(steps)], b.counters()


# Fewer and more windows than blocks, a last window of one neuron, delays below, at and past the bitmaps that a
# block holds at a time.
@pytest.mark.parametrize("n,fan_in,d_hi", [(3000, 400, 1), (3000, 400, 8), (2817, 400, 9), (40000, 60, 20), (45057, 48, 3),
                                           (300, 4000, 17)])
def test_gather_shares_equal_the_scatter(n, fan_in, d_hi):
    from knp_gb300 import types as T

    ref, counts = _trains(n, fan_in, d_hi, -1.0, T.STEP_GRID)
    assert sum(s.size for s in ref) > 0
    for mode in (T.STEP_GRID, T.STEP_PHASES):
        for threshold in (0.0, 0.2):
            got, c = _trains(n, fan_in, d_hi, threshold, mode)
            assert c == counts
            for a, b in zip(got, ref):
                np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("mode", ["STEP_PHASES", "STEP_FUSED", "STEP_GRID"])
def test_long_rows_among_short_ones_match_the_oracle(mode):
    from knp_gb300 import backend as B
    from knp_gb300 import network as N
    from knp_gb300 import types as T
    from oracle import oracle as orc

    rng = np.random.default_rng(2)
    n, n_in = 700, 6000
    # Most sources without a synapse or with one; some with 8, 9, 33 and 2000 (two synapses a row on average at most).
    per_row = (rng.random(n_in) < 0.6).astype(np.int64)
    per_row[[3, 40, 41, 77, 5999]] = [8, 9, 33, 2000, 31]
    pre = np.repeat(np.arange(n_in, dtype=np.uint32), per_row)
    pop, proj, chan = (T.uid_from_int(5300 + i) for i in range(3))
    pr = N.Projection(proj, T.DELTA, T.NULL_UID, pop, pre, rng.integers(0, n, pre.size).astype(np.uint32),
                      (rng.integers(-64, 129, pre.size) / 256.0).astype(np.float32),
                      rng.integers(1, 5, pre.size).astype(np.uint32))
    net = N.Network([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))], [pr], [(proj, chan)])
    trains = [np.sort(rng.choice(n_in, k, replace=False)).astype(np.uint32) for k in (6000, 0, 1, 31, 33, 3000, 700, 64)]
    trains[3] = np.array([3, 40, 41, 77, 5999], np.uint32)
    offs = np.concatenate([[0], np.cumsum([t.size for t in trains])]).astype(np.int64)
    sched = [N.SpikeSchedule(chan, offs, np.concatenate(trains))]
    ref, _ = orc.run(net, sched, 14)
    out, b = B.run(net, sched, 14, step_mode=getattr(T, mode))
    assert b.counters()[0] == sum(int(per_row[t].sum()) for t in trains)
    for t in range(14):
        np.testing.assert_array_equal(out[pop][t], ref[pop][t])
    b.close()
