"""Device memory of an input channel: a spike schedule's goes when a host message takes its place, and messages and
schedules may follow one another in any order (one-to-one projection, weight 1, delay 1: a neuron fires the step after
its source's message)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
N_NEURONS = 20000


def _backend():
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    pop, proj, chan = (T.uid_from_int(6500 + i) for i in range(3))
    b = GB300Backend()
    b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(N_NEURONS))])
    b.generate_projection(proj, T.NULL_UID, pop, T.GEN_ONE_TO_ONE, N_NEURONS, N_NEURONS, 256, 256, 1, 1, 1, 1)
    b.subscribe(proj, [chan])
    b.record_spikes(pop)
    b._init()
    return b, pop, chan


@pytest.mark.parametrize("generated", [True, False])
@pytest.mark.parametrize("length", [0, 5, 2048, 2049, 15000])
def test_a_message_frees_the_schedule_it_replaces(generated, length):
    from knp_gb300 import network as N

    b, pop, chan = _backend()
    steps = 4000
    if generated:
        b.generate_bernoulli_schedule(chan, N_NEURONS, 0.5, 0, steps, 3)
    else:
        train = np.arange(0, N_NEURONS, 2, dtype=np.uint32)
        b.load_spike_schedule(N.SpikeSchedule(chan, np.arange(steps + 1, dtype=np.int64) * train.size, np.tile(train, steps)))
    b.step(steps)
    b.synchronize()
    before = torch.cuda.mem_get_info()[0]  # about 160 MB of indexes
    sent = np.arange(7, 7 + length, dtype=np.uint32)
    for _ in range(2):
        t = b.get_step()
        b.send_spikes(chan, sent, t)
        b.step(2)
        np.testing.assert_array_equal(b.spikes(pop, t + 1), sent)
    assert torch.cuda.mem_get_info()[0] - before > 100 << 20
    b.close()


def test_messages_and_schedules_in_turn():
    from knp_gb300 import network as N

    b, pop, chan = _backend()
    rng = np.random.default_rng(5)
    pick = lambda k: np.sort(rng.choice(N_NEURONS, k, replace=False)).astype(np.uint32)  # noqa: E731
    for length in (3, 3000, 2, 5000, 2048, 1, 2049):
        sent, t = pick(length), b.get_step()
        b.send_spikes(chan, sent, t)
        b.step(2)
        np.testing.assert_array_equal(b.spikes(pop, t + 1), sent)
        if length % 2:
            trains = [pick(k) for k in (10, 0, 4000)]
            t = b.get_step()
            offs = np.concatenate([[0], np.cumsum([s.size for s in trains])]).astype(np.int64)
            b.load_spike_schedule(N.SpikeSchedule(chan, offs, np.concatenate(trains)), t)
        else:
            t = b.get_step()
            b.generate_bernoulli_schedule(chan, N_NEURONS, 0.3, t, 3, 11)
            trains = [N.bernoulli_schedule(chan, 11, N_NEURONS, t + 3, 0.3).at(t + k) for k in range(3)]
        b.step(4)
        for k, s in enumerate(trains):
            np.testing.assert_array_equal(b.spikes(pop, t + k + 1), s)
    b.close()
