"""The fused and the grid step kernel at the edges of their shares: populations around the number of the cluster's threads, more
rows than the tables hold, more sources than one look resolves, more descriptors than shared memory takes, rows
too long for the list. Their results are the per-phase kernels', bit for bit: sums are exact in any order (dyadic
weights, or the fixed-point ring)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(net, sched, steps, mode):
    from knp_gb300 import backend as B

    out, b = B.run(net, sched, steps, step_mode=mode)
    got = [out[p.uid] for p in net.populations], [b.read_weights(p.uid) for p in net.projections], b.counters()
    b.close()
    return got


def _same(net, sched, steps, modes=None):
    from knp_gb300 import types as T

    ref, ref_w, ref_c = _run(net, sched, steps, T.STEP_PHASES)
    assert ref_c[1] > 0
    for mode in modes or (T.STEP_FUSED, T.STEP_GRID):
        spikes, weights, counts = _run(net, sched, steps, mode)
        assert counts == ref_c
        for a, b in zip(spikes, ref):
            for t in range(steps):
                np.testing.assert_array_equal(a[t], b[t])
        for a, b in zip(weights, ref_w):
            np.testing.assert_array_equal(a, b)


def _schedule(N, chan, trains):
    offs = np.concatenate([[0], np.cumsum([t.size for t in trains])]).astype(np.int64)
    return N.SpikeSchedule(chan, offs, np.concatenate(trains).astype(np.uint32))


# A neuron a thread up to 8192 neurons (16 CTAs of 512 threads), then four; 9000 rows of every neuron's spike are
# more than 512 a CTA, and 9000 neurons' spike lists more than shared memory is given. Odd scale: weights that no
# FP32 sum holds exactly (the fixed-point ring).
@pytest.mark.parametrize("n,p_in,scale", [(1, 1.0, 256), (31, 0.8, 256), (33, 0.8, 250), (1000, 0.4, 250), (4097, 0.3, 256),
                                          (8192, 0.5, 256), (8193, 0.5, 250), (9000, 1.0, 256)])
def test_population_sizes(n, p_in, scale):
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(n)
    pop, inp, rec, chan = (T.uid_from_int(5400 + i) for i in range(4))
    ids = np.arange(n, dtype=np.uint32)
    fan = min(n, 24)
    drive = N.Projection(inp, T.DELTA, T.NULL_UID, pop, ids, ids, np.ones(n, np.float32), np.ones(n, np.uint32))
    back = N.Projection(rec, T.DELTA, pop, pop, rng.integers(0, n, n * fan).astype(np.uint32), np.repeat(ids, fan),
                        (rng.integers(-96, 97, n * fan) / scale).astype(np.float32),
                        rng.integers(0, 6, n * fan).astype(np.uint32))
    net = N.Network([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))], [drive, back], [(inp, chan)])
    trains = [np.flatnonzero(rng.random(n) < p_in) for _ in range(8)]
    trains[0] = ids
    _same(net, [_schedule(N, chan, trains)], 12)


# 33 sources are more than one look resolves; 120 projections' descriptors stay in global memory.
@pytest.mark.parametrize("n_proj", [1, 32, 33, 120])
def test_many_projections(n_proj):
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(n_proj)
    n, n_in = 500, 70
    a, b, chan = (T.uid_from_int(5500 + i) for i in range(3))
    projs, subs = [], []
    for k in range(n_proj):
        uid = T.uid_from_int(5600 + k)
        src = (T.NULL_UID, a, b)[k % 3] if k else T.NULL_UID
        rows = n_in if k % 3 == 0 else n
        m = (0, 1, 40, 900)[(k + 3) % 4]  # some without a synapse; most of the others' rows without one too
        w = np.abs(rng.integers(1, 200, m)) / 128.0
        projs.append(N.Projection(uid, T.DELTA, src, (a, b)[k % 2], rng.integers(0, rows, m).astype(np.uint32),
                                  rng.integers(0, n, m).astype(np.uint32), w.astype(np.float32),
                                  rng.integers(1, 9, m).astype(np.uint32),
                                  out_type=rng.integers(0, 2, m).astype(np.uint8) if k % 5 == 4 else None))
        if k % 3 == 0:
            subs.append((uid, chan))
    net = N.Network([N.Population(u, T.BLIFAT, T.blifat_defaults(n)) for u in (a, b)], projs, subs)
    trains = [np.flatnonzero(rng.random(n_in) < 0.5) for _ in range(10)]
    _same(net, [_schedule(N, chan, trains)], 16)


def test_a_row_longer_than_the_list():
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(1)
    n, n_in, long_row = 300, 700, (1 << 20) + 77
    per_row = np.full(n_in, 9, np.int64)
    per_row[[7, 31]] = long_row, 1 << 20  # one above the length that is walked by itself, one at it
    m = int(per_row.sum())
    pop, inp, chan = (T.uid_from_int(5800 + i) for i in range(3))
    pr = N.Projection(inp, T.DELTA, T.NULL_UID, pop, np.repeat(np.arange(n_in, dtype=np.uint32), per_row),
                      rng.integers(0, n, m).astype(np.uint32), (rng.integers(-3, 4, m) / 256.0).astype(np.float32),
                      rng.integers(1, 4, m).astype(np.uint32))
    net = N.Network([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))], [pr], [(inp, chan)])
    # A few rows are cut into parts; 100 are not on 16 CTAs, 700 not on any number.
    trains = [np.array(x) for x in ([7], [3, 7, 31], [31], list(range(100)), list(range(n_in)))]
    _same(net, [_schedule(N, chan, trains)], 10)


# Rows on either side of every cut of a 16- and a 152-CTA kernel (64 and 608 rows, halved six times), of odd lengths.
@pytest.mark.parametrize("n_spikes", [1, 2, 9, 10, 19, 33, 64, 65, 152, 153, 304, 608, 609])
def test_rows_cut_into_parts(n_spikes):
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(n_spikes)
    n, n_in = 400, 620
    per_row = rng.integers(0, 140, n_in)
    per_row[:5] = [0, 1, 31, 63, 65]
    m = int(per_row.sum())
    pop, inp, chan = (T.uid_from_int(5850 + i) for i in range(3))
    pr = N.Projection(inp, T.DELTA, T.NULL_UID, pop, np.repeat(np.arange(n_in, dtype=np.uint32), per_row),
                      rng.integers(0, n, m).astype(np.uint32), (rng.integers(20, 100, m) / 64.0).astype(np.float32),
                      rng.integers(1, 4, m).astype(np.uint32))
    net = N.Network([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))], [pr], [(inp, chan)])
    trains = [np.sort(rng.choice(n_in, n_spikes, replace=False)) for _ in range(5)] + [np.arange(n_in)[:n_spikes]]
    _same(net, [_schedule(N, chan, trains)], 10)


def test_more_rows_than_the_grid_kernel_tables_hold():
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(3)
    n = 160000  # 1024 rows a CTA are 155648
    pop, inp, rec, chan = (T.uid_from_int(5870 + i) for i in range(4))
    ids = np.arange(n, dtype=np.uint32)
    drive = N.Projection(inp, T.DELTA, T.NULL_UID, pop, ids, ids, np.ones(n, np.float32), np.ones(n, np.uint32))
    back = N.Projection(rec, T.DELTA, pop, pop, rng.integers(0, n, 3 * n).astype(np.uint32), np.repeat(ids, 3),
                        (rng.integers(-96, 97, 3 * n) / 256).astype(np.float32), rng.integers(1, 6, 3 * n).astype(np.uint32))
    net = N.Network([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))], [drive, back], [(inp, chan)])
    _same(net, [_schedule(N, chan, [ids, ids[::2], ids])], 6, [T.STEP_GRID])


# 10^7 synapses and more a step are 65536 a CTA: rows of 20011 of every third source, so that runs of 128 cross them.
@pytest.mark.parametrize("fixed", [False, True])
def test_long_lists(fixed):
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    n, n_in, steps = 20011, 1600, 6
    pop, inp, rec, chan = (T.uid_from_int(5880 + i) for i in range(4))
    got = []
    for mode in (T.STEP_PHASES, T.STEP_GRID):
        with GB300Backend() as b:
            b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))])
            b.generate_projection(inp, T.NULL_UID, pop, T.GEN_ALL_TO_ALL, n_in, n, -8, 9, 1, 4, 7, 10)
            b.generate_fixed_fan_in_projection(rec, pop, pop, n, n, 37, -32, 32, 1, 3, 8, 20)
            b.subscribe(inp, [chan])
            b.record_spikes(pop)
            if fixed:
                b.set_accumulator(pop, T.ACC_FIXED64)
            b.set_pull_threshold(rec, -1.0)
            b.set_step_mode(mode)
            b._init()
            trains = [np.arange(k % 3, n_in, 3) if k % 2 else np.arange(n_in) for k in range(steps)]
            offs = np.concatenate([[0], np.cumsum([t.size for t in trains])]).astype(np.int64)
            b.load_spike_schedule(N.SpikeSchedule(chan, offs, np.concatenate(trains).astype(np.uint32)), 0)
            b.step(steps)
            got.append(([b.spikes(pop, t) for t in range(steps)], b.counters()))
    (ref, ref_c), (spikes, counts) = got
    assert counts == ref_c and ref_c[1] > 0
    for a, c in zip(spikes, ref):
        np.testing.assert_array_equal(a, c)
