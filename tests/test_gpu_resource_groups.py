"""Resource-STDP training by a warp or by a block per neuron, at the edges: mean numbers of synapses around the one from
which a block takes a neuron and around a tile of the block's (1024), and weights so far apart that the additional
threshold's FP64 sum rounds, so that its terms have to be added in the reference's order."""
import sys
from dataclasses import replace
from pathlib import Path

import numpy as np
import pytest

from knp_gb300 import network as N
from knp_gb300 import types as T

sys.path.insert(0, str(Path(__file__).resolve().parent))
from test_gpu_resource_stdp import check_all, run_both  # noqa: E402

pytestmark = pytest.mark.gpu


def _with_more_synapses(net, more):
    """The network with a copy of its plastic projection's first `more` sources beside it."""
    pr = net.projections[0]
    take = pr.pre < more
    uid = T.uid_from_int(77001)
    copy = replace(pr, uid=uid, pre=pr.pre[take].copy(), post=pr.post[take].copy(), weight=pr.weight[take].copy(),
                   delay=pr.delay[take].copy(), rule=pr.rule[take].copy(),
                   out_type=None if pr.out_type is None else pr.out_type[take].copy())
    net.projections.insert(1, copy)
    net.subscriptions += [(uid, sender) for receiver, sender in net.subscriptions if receiver == pr.uid]


# Synapses of a neuron: n_in from the images, and as many again as `more`.
@pytest.mark.parametrize("n_in,more", [(33, 0), (127, 0), (128, 0), (784, 0), (600, 423), (600, 424), (600, 425), (784, 784),
                                       (64, 63)])
@pytest.mark.parametrize("apart", [False, True])
def test_training_at_the_edges_of_its_groups(n_in, more, apart):
    net, sched = N.resource_stdp_network(seed=n_in, samples=6, n_in=n_in, per_column=5, classes=4)
    if more:
        _with_more_synapses(net, more)
    if apart:
        w = net.projections[0].weight
        rng = np.random.default_rng(n_in)
        w[:] = np.where(rng.random(w.size) < 0.5, 0.09, rng.random(w.size).astype(np.float32) * np.float32(2.0**-40))
    g, b, o, oo = run_both(net, sched, 90)
    assert sum(x.size for x in g[net.populations[0].uid]) > 0
    check_all(net, g, b, o, oo)
    b.close()
