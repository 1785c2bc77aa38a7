"""Launches that several populations or projections share: more of them than a launch takes, with sizes at a block's
edges and with ones too large to share. The grid step kernel, which has no such launches, gives the same spikes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,fixed", [([300], False), ([1, 255, 256, 257], False), ([33, 600, 512, 40000, 64, 300], True),
                                         ([40000, 9], False)])
def test_shared_launches_equal_the_grid_kernel(sizes, fixed):
    from knp_gb300 import backend as B
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(len(sizes) + sizes[0])
    n_in = 500
    pops = [T.uid_from_int(5900 + i) for i in range(len(sizes))]
    chan = T.uid_from_int(5950)
    projs, subs = [], []
    for i, n in enumerate(sizes):
        for k, src in enumerate([T.NULL_UID, pops[i], pops[(i + 1) % len(sizes)]]):
            uid = T.uid_from_int(6000 + 3 * i + k)
            rows = n_in if k == 0 else sizes[i if k == 1 else (i + 1) % len(sizes)]
            m = 6 * n
            w = rng.integers(-40 if k else 0, 120, m) / (250.0 if fixed else 256.0)
            projs.append(N.Projection(uid, T.DELTA, src, pops[i], rng.integers(0, rows, m).astype(np.uint32),
                                      rng.integers(0, n, m).astype(np.uint32), w.astype(np.float32),
                                      rng.integers(1, 5, m).astype(np.uint32)))
            if k == 0:
                subs.append((uid, chan))
    net = N.Network([N.Population(u, T.BLIFAT, T.blifat_defaults(n)) for u, n in zip(pops, sizes)], projs, subs)
    trains = [np.flatnonzero(rng.random(n_in) < 0.6) for _ in range(8)]
    offs = np.concatenate([[0], np.cumsum([t.size for t in trains])]).astype(np.int64)
    sched = [N.SpikeSchedule(chan, offs, np.concatenate(trains).astype(np.uint32))]
    got = {}
    for mode in (T.STEP_PHASES, T.STEP_GRID):
        out, b = B.run(net, sched, 12, step_mode=mode)
        got[mode] = out, b.counters()
        b.close()
    assert got[T.STEP_PHASES][1] == got[T.STEP_GRID][1] and got[T.STEP_GRID][1][1] > 0
    for u in pops:
        for t in range(12):
            np.testing.assert_array_equal(got[T.STEP_PHASES][0][u][t], got[T.STEP_GRID][0][u][t])
