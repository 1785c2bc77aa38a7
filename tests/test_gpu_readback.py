"""Spikes of a large population read back as lists made on the device (readback.cu), as bitmaps, and while
later steps are queued: every form gives the indexes that were sent in through a one-to-one projection
(weight 1, delay 1: a neuron fires the step after its source's message)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _backend(n, device_steps=None):
    from knp_gb300 import GB300Backend
    from knp_gb300 import network as N
    from knp_gb300 import types as T

    pop, proj, chan = (T.uid_from_int(4100 + i) for i in range(3))
    b = GB300Backend()
    b.load_populations([N.Population(pop, T.BLIFAT, T.blifat_defaults(n))])
    b.generate_projection(proj, T.NULL_UID, pop, T.GEN_ONE_TO_ONE, n, n, 256, 256, 1, 1, 1, 1)
    b.subscribe(proj, [chan])
    b.record_spikes(pop)
    b._init()
    return b, pop, chan


def _trains(n):
    """Messages: none, one neuron at either end, exactly as many spikes as the bitmap has words and one
    more (list and bitmap), a run denser than a segment's shared memory, every neuron, and a few at random."""
    w = (n + 31) // 32
    rng = np.random.default_rng(n)
    pick = lambda k: np.sort(rng.choice(n, k, replace=False)).astype(np.uint32)  # noqa: E731
    return [np.zeros(0, np.uint32), np.array([0], np.uint32), np.array([n - 1], np.uint32), pick(w), pick(w + 1),
            np.arange(100, 100 + min(5000, w), dtype=np.uint32), np.arange(n, dtype=np.uint32), pick(7), pick(w // 3)]


# Word counts below, at and past a segment, with a partial last word and segment.
@pytest.mark.parametrize("n", [32000, 32768, 32769, 200003])
@pytest.mark.parametrize("batch", [1, 4, 9])
def test_spikes_read_back_in_every_form(n, batch):
    from knp_gb300 import network as N

    b, pop, chan = _backend(n)
    trains = _trains(n)
    offs = np.concatenate([[0], np.cumsum([t.size for t in trains])]).astype(np.int64)
    b.load_spike_schedule(N.SpikeSchedule(chan, offs, np.concatenate(trains)))
    for first in range(0, 9, batch):
        b.step(min(batch, 9 - first))
    b.step(1)
    for t, sent in enumerate(trains):
        np.testing.assert_array_equal(b.spikes(pop, t + 1), sent, err_msg=f"step {t + 1}")
        out = np.full(max(1, sent.size // 2), 0xFFFFFFFF, np.uint32)
        assert b.spikes_capped(pop, t + 1, out) == sent.size
        np.testing.assert_array_equal(out[:sent.size], sent[:out.size])
    b.close()


def test_spikes_read_while_a_later_step_runs_and_messages_of_every_length():
    """Host messages below, at and past the length that goes out with its descriptor in one copy; each step
    is read while the next is queued, and the last one after."""
    b, pop, chan = _backend(40000)
    rng = np.random.default_rng(3)
    trains = [np.sort(rng.choice(40000, k, replace=False)).astype(np.uint32) for k in (2048, 2049, 0, 1, 30000, 2047, 5)]
    for t, sent in enumerate(trains):
        b.send_spikes(chan, sent, t)
        b._step()
        if t > 1:
            np.testing.assert_array_equal(b.spikes(pop, t - 1), trains[t - 2])
    b._step()
    for t in (len(trains) - 1, len(trains)):
        np.testing.assert_array_equal(b.spikes(pop, t), trains[t - 1])
    b.discard_spikes(len(trains))
    b.close()
