"""The fused step kernel with little shared memory, near the most, and past what it copies (descriptors of many
projections beside spike lists of 8192 neurons): its cluster is chosen for the launch's own need, and its spikes are
those of the per-phase kernels (dyadic weights)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100, 8192])
@pytest.mark.parametrize("n_proj", [1, 40, 60, 80, 100, 250])
def test_descriptors_and_lists_of_every_size(n, n_proj):
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    rng = np.random.default_rng(n_proj)
    pop, chan = T.uid_from_int(6400), T.uid_from_int(6401)
    parts = [(rng.integers(0, n, 300).astype(np.uint32), rng.integers(0, n, 300).astype(np.uint32),
              (rng.integers(-64, 257, 300) / 256.0).astype(np.float32), rng.integers(1, 5, 300).astype(np.uint32))
             for _ in range(n_proj)]
    out = []
    for mode in (T.STEP_FUSED, T.STEP_PHASES):
        with GB300Backend() as b:
            b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))])
            b.generate_projection(T.uid_from_int(6402), T.NULL_UID, pop, T.GEN_ONE_TO_ONE, n, n, 256, 256, 1, 1, 5, 10)
            b.subscribe(T.uid_from_int(6402), [chan])
            b.load_projections([N.Projection(T.uid_from_int(6410 + k), T.DELTA, pop, pop, *p) for k, p in enumerate(parts)])
            b.record_spikes(pop)
            b.set_step_mode(mode)
            b._init()
            b.generate_bernoulli_schedule(chan, n, 0.4, 0, 12, 9)
            b.step(5)
            b.step(7)
            out.append([b.spikes(pop, t) for t in range(12)])
    assert sum(s.size for s in out[0]) > 0
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
