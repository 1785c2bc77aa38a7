"""The batched form's layer kernel at the sizes where its tiles, chunks, streams and steps end: spike
records, counts and events against a NumPy restatement of the LIF rules (lif_impl.h:33-86). Weights are
k/256 with |k| <= 64, so every input sum is exact in FP32 in any order and the NumPy FP32 recurrence
(the same product, sum and comparison per step) gives the same bits: the spikes have to be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(cfg):
    from knp_gb300 import batched as BT

    L = len(cfg.sizes) - 1
    f = np.float32
    par = [(f((cfg.leak or (1,) * L)[k]), f((cfg.threshold or (1,) * L)[k]), f((cfg.reset or (0,) * L)[k]),
            int((cfg.refract or (0,) * L)[k])) for k in range(L)]
    spikes, events = {}, 0
    counts = np.zeros((cfg.batch, cfg.sizes[-1]), np.int64)
    for b in range(cfg.batch):
        own = [cfg.sizes[k] if cfg.sample_sizes is None else int(cfg.sample_sizes[k][b]) for k in range(L + 1)]
        V = [np.zeros(n, f) for n in cfg.sizes[1:]]
        rc = [np.zeros(n, np.int64) for n in cfg.sizes[1:]]
        prev = [np.zeros(n, bool) for n in cfg.sizes]
        for t in range(int(cfg.steps[b])):
            now = [np.zeros(n, bool) for n in cfg.sizes]
            now[0][BT.input_spikes(cfg, b, t)] = True
            for k in range(L):
                leak, thr, reset, period = par[k]
                current = (cfg.weights[k].astype(np.float64) @ prev[k]).astype(f)
                free = rc[k] == 0
                v = (V[k] * leak).astype(f) + current
                fire = free & (v > thr) & (np.arange(cfg.sizes[k + 1]) < own[k + 1])
                V[k] = np.where(fire, reset, np.where(free, v, V[k])).astype(f)
                rc[k] = np.where(fire, period, np.where(free, 0, rc[k] - 1))
                now[k + 1] = fire
            for k in range(L):
                events += int(now[k].sum()) * own[k + 1]
            counts[b] += now[L]
            for k in range(L + 1):
                spikes[k, b, t] = np.nonzero(now[k])[0]
            prev = now
    return spikes, counts, events


# Sizes at and one off a K block (16), a chunk (64), a stage (128), a neuron tile (128) and a tile pair
# (256); steps at and one off a padded run (8), a scan block (32) and a stream tile (128); batches of one
# sample, of one stream more than a pair's two, and of more samples than streams.
@pytest.mark.parametrize("sizes,batch,t_lo,t_hi,leak,refract", [
    ((15, 127, 1), 1, 1, 1, 1.0, 0), ((16, 128, 2), 2, 8, 8, 1.0, 0), ((17, 129, 33), 3, 7, 9, 0.9, 0),
    ((63, 255, 31), 5, 31, 33, 1.0, 0), ((64, 256, 65), 4, 32, 32, 0.75, 2), ((65, 257, 16), 3, 127, 129, 1.0, 0),
    ((127, 300), 2, 128, 128, 1.0, 1), ((128, 40, 40, 40, 5), 3, 15, 40, 0.9, 0), ((129, 64, 10), 160, 1, 40, 1.0, 0),
    ((400, 513, 12), 2, 250, 260, 1.0, 0)])
@pytest.mark.parametrize("segment_steps", [0, 13])
def test_batched_layers_equal_the_lif_rules(sizes, batch, t_lo, t_hi, leak, refract, segment_steps):
    from knp_gb300 import batched as BT

    cfg = BT.dense_config(seed=len(sizes) + batch + t_hi, batch=batch, sizes=sizes, t_lo=t_lo, t_hi=t_hi, rate_max=0.4)
    rng = np.random.default_rng(7)
    L = len(sizes) - 1
    cfg.weights = [(rng.integers(-24, 65, w.shape) / 256.0).astype(np.float32) for w in cfg.weights]
    cfg.leak, cfg.refract, cfg.reset = (leak,) * L, (refract,) * L, (0.125,) * L
    if batch == 3:
        cfg.sample_sizes = np.array([[max(1, n - 5 * b) for b in range(batch)] for n in sizes], np.uint32)
    ref, ref_counts, ref_events = _reference(cfg)
    counts, rec, events, _ = BT.run(cfg, record=True, segment_steps=segment_steps)
    for (k, b, t), idx in ref.items():
        np.testing.assert_array_equal(BT.spikes_from_bits(rec[k][t, b], sizes[k]), idx, err_msg=f"{k, b, t}")
    np.testing.assert_array_equal(counts, ref_counts)
    assert events == ref_events
