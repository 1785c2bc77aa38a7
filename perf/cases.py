"""The calls a user of this framework makes, as cases to be measured.

Six kinds, each through its public entry points:

network   a spiking network stepped by ``GB300Backend``: input spikes handed over (step by step, or as
          a window of steps), steps run, the population's spikes read back
stdp      one sample shown to an additive-STDP network, and its weights read
resource  one sample shown to a synaptic-resource-STDP network (three populations, seven projections)
batched   many feed-forward LIF samples in one ``BatchedPlan.run``
layer     one LIF layer forward and backward (``bptt.LIFLayerFn``)
train     one training iteration of a spiking MLP (``bptt.GraphedTrainStep``)
gemm      the BF16 matrix product under the last two (``bptt.gemm_tn``)

Every network has balanced recurrent weights or inhibition, so its activity stays at one level however
many passes it has run.
"""
import math

import numpy as np
import torch

from knp_gb300 import GB300Backend
from knp_gb300 import batched, bptt
from knp_gb300 import network as N
from knp_gb300 import types as T

BETA, THETA, SLOPE = 0.9, 1.0, 25.0
LEARNING_RATE = 1e-4
WARMUP_ITERATIONS = 3
SCHEDULE_STEPS = 20000
K_MAX = 32  # recurrent weights are k/256 with k uniform in [-K_MAX, K_MAX]


def listed():
    return [
        # One step of a small network driven spike message by spike message, as a control loop or an
        # executor with monitoring does: all latency.
        {"name": "online_small", "kind": "network", "n": 1000, "n_in": 100, "fan_in": 100, "p_in": 0.05,
         "delay": 5, "steps": 1, "online": True},
        # The same network left to run over a window of input that is on the device already.
        {"name": "window_small", "kind": "network", "n": 1000, "n_in": 100, "fan_in": 100, "p_in": 0.05,
         "delay": 5, "steps": 200, "online": False},
        # Learning: one 100-step image shown to the additive-STDP network (784 -> 800, lateral inhibition).
        {"name": "stdp_sample", "kind": "stdp", "n_in": 784, "n": 800, "steps": 100},
        # Learning: one 15-step image and its label shown to the resource-STDP network (784 -> 200 -> 10).
        {"name": "resource_sample", "kind": "resource", "n_in": 784, "per_column": 20, "classes": 10},
        # The large sparse network at the low rates such networks live at: a million neurons, a
        # thousand synapses each, half a per cent of them firing.
        {"name": "sparse_1m", "kind": "network", "n": 1000000, "n_in": 0, "fan_in": 1000, "p_in": 0.01, "delay": 20,
         "steps": 20, "online": False},
        # A smaller one in a state of high activity (about a third of the neurons fire each step).
        {"name": "dense_200k", "kind": "network", "n": 200000, "n_in": 0, "fan_in": 1000, "p_in": 0.3, "delay": 20,
         "steps": 5, "online": False},
        # Inference over a data set's batch with uneven sample lengths, output spike counts read.
        {"name": "batched_256", "kind": "batched", "sizes": "784-1000-1000-10", "batch": 256, "t_lo": 50,
         "t_hi": 200, "rate": 0.2, "uneven": False, "record": False},
        # A few small instances of uneven layer widths, with every spike train recorded and read.
        {"name": "batched_uneven_40", "kind": "batched", "sizes": "96-128-64-10", "batch": 40, "t_lo": 10,
         "t_hi": 30, "rate": 0.3, "uneven": True, "record": True},
        # One iteration of surrogate-gradient training of a small classifier, as its graph replays it.
        {"name": "train_784_512", "kind": "train", "sizes": "784-512-512-10", "batch": 128, "T": 32},
        # A layer inside a model of one's own, forward and backward, at sizes no tile divides.
        {"name": "layer_ragged", "kind": "layer", "T": 25, "batch": 50, "n_in": 700, "n_out": 333},
        # And a wide one, where the matrix products carry the time.
        {"name": "layer_wide", "kind": "layer", "T": 64, "batch": 256, "n_in": 2048, "n_out": 2048},
        # The matrix product alone, large.
        {"name": "gemm_8192", "kind": "gemm", "M": 8192, "N": 8192, "K": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["network", "network", "network", "stdp", "resource", "batched", "batched", "layer", "layer",
                       "train", "gemm"])
    if kind == "network":
        scale = rng.choice(["small", "sparse", "dense"])
        if scale == "small":
            online = rng.random() < 0.5
            return {"kind": kind, "n": _log(rng, 100, 6000), "n_in": _log(rng, 20, 400), "fan_in": _log(rng, 20, 300),
                    "p_in": rng.uniform(0.02, 0.1), "delay": rng.randint(1, 8),
                    "steps": _log(rng, 1, 10) if online else _log(rng, 20, 500), "online": online}
        if scale == "sparse":
            return {"kind": kind, "n": _log(rng, 50000, 1000000), "n_in": 0, "fan_in": _log(rng, 100, 1000),
                    "p_in": math.exp(rng.uniform(math.log(0.004), math.log(0.015))), "delay": rng.randint(4, 25),
                    "steps": _log(rng, 5, 20), "online": False}
        return {"kind": kind, "n": _log(rng, 50000, 200000), "n_in": 0, "fan_in": _log(rng, 200, 1000),
                "p_in": rng.uniform(0.25, 0.5), "delay": rng.randint(4, 20), "steps": _log(rng, 2, 5), "online": False}
    if kind == "stdp":
        return {"kind": kind, "n_in": rng.randint(300, 784), "n": rng.randint(300, 900), "steps": _log(rng, 30, 120)}
    if kind == "resource":
        return {"kind": kind, "n_in": rng.randint(300, 784), "per_column": rng.randint(10, 24),
                "classes": rng.randint(4, 12)}
    if kind == "batched":
        sizes = [rng.randint(100, 1000) for _ in range(rng.randint(2, 3))] + [rng.randint(4, 40)]
        lo = _log(rng, 5, 50)
        return {"kind": kind, "sizes": "-".join(str(x) for x in sizes), "batch": _log(rng, 8, 256), "t_lo": lo,
                "t_hi": lo + _log(rng, 5, 120), "rate": rng.uniform(0.1, 0.3), "uneven": rng.random() < 0.3,
                "record": False}
    if kind == "layer":
        return {"kind": kind, "T": _log(rng, 4, 64), "batch": _log(rng, 8, 256), "n_in": _log(rng, 100, 2048),
                "n_out": _log(rng, 10, 2048)}
    if kind == "train":
        hidden = _log(rng, 100, 800)
        return {"kind": kind, "sizes": "%d-%d-%d-10" % (rng.randint(200, 800), hidden, hidden),
                "batch": _log(rng, 16, 192), "T": rng.randint(8, 48)}
    return {"kind": kind, "M": _log(rng, 64, 8192), "N": _log(rng, 64, 8192), "K": _log(rng, 64, 8192)}


def _sizes(case):
    return tuple(int(x) for x in case["sizes"].split("-"))


def _rate(case):
    """The firing rate a network of this case settles at: a neuron fires when one background spike
    (weight 1) and recurrent input not below 0 arrive, or recurrent input alone reaches the threshold."""
    var = case["fan_in"] * K_MAX * (K_MAX + 1) / 3 / 256.0 ** 2
    p, r = (0.0, 0.05) if case["n_in"] else (case["p_in"], case["p_in"])
    mean = case["n_in"] * case["p_in"] * 0.125 if case["n_in"] else 0.0
    in_var = case["n_in"] * case["p_in"] * 0.021
    for _ in range(50):
        sd = math.sqrt(max(var * r + in_var, 1e-9))
        r = p * 0.53 + (1 - p) * 0.5 * math.erfc((1.0 - mean) / sd / math.sqrt(2))
    return r


# ------------------------------------------------------------------------------------- networks


class _Network:
    """A backend loaded with one population, its input projection and its recurrent projection."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        n, n_in, fan_in = case["n"], case["n_in"], case["fan_in"]
        self.pop, rec, inp, self.chan = (T.uid_from_int(10 * (seed % 1000000) + i) for i in (1, 2, 3, 4))
        b = self.backend = GB300Backend()
        b.load_populations([N.Population(self.pop, T.BLIFAT, T.blifat_defaults(n))])
        if n_in:  # all-to-all input, k in [0, 64], delays 1..4
            b.generate_projection(inp, T.NULL_UID, self.pop, T.GEN_ALL_TO_ALL, n_in, n, 0, 64, 1, 4, seed, 10)
        else:  # background drive, one source per neuron, weight 1, delay 1
            b.generate_projection(inp, T.NULL_UID, self.pop, T.GEN_ONE_TO_ONE, n, n, 256, 256, 1, 1, seed, 10)
        b.generate_fixed_fan_in_projection(rec, self.pop, self.pop, n, n, fan_in, -K_MAX, K_MAX, 1, case["delay"], seed,
                                           20)
        b.subscribe(inp, [self.chan])
        b.record_spikes(self.pop)
        b._init()
        self.scheduled_to = 0
        self.room = min(n, int(2.0 * _rate(case) * n) + 100)
        if case["online"]:
            self.messages = N.bernoulli_schedule(self.chan, seed, n_in or n, 256, case["p_in"])
            for _ in range(16):
                self.step_online()
        else:
            self.window(min(40, 2 * case["delay"]))  # past the first delays: every step is an ordinary one

    def step_online(self):
        b = self.backend
        t = b.get_step()
        b.send_spikes(self.chan, self.messages.at(t % 256), t)
        b._step()
        return self.read(t, 1)

    def window(self, steps):
        b = self.backend
        t = b.get_step()
        if t + steps > self.scheduled_to:
            self.scheduled_to = t + max(steps, SCHEDULE_STEPS)
            b.generate_bernoulli_schedule(self.chan, self.case["n_in"] or self.case["n"], self.case["p_in"], t,
                                          self.scheduled_to - t, self.seed)
        b.step(steps)
        return self.read(t, steps)

    def read(self, t, steps):
        return _trains(self.backend, self.pop, self.room, t, steps)


def _trains(backend, pop, room, t, steps):
    """Spike trains of the steps t .. t + steps - 1: the number of spikes of each, and their ascending
    indexes in rows of ``room``, the rest of a row zero."""
    rows = np.zeros((steps, room), np.uint32)
    return [np.array([backend.spikes_capped(pop, t + k, rows[k]) for k in range(steps)], np.int64), rows]


def _part(sched, first, steps):
    """Steps [first, first + steps) of a schedule, as a schedule of its own."""
    offs = sched.offsets[first:first + steps + 1]
    return N.SpikeSchedule(sched.sender, offs - offs[0], sched.indexes[offs[0]:offs[-1]])


class _Learner:
    """A plastic network and its samples' input, shown one sample per pass in turn."""

    def __init__(self, case, seed):
        if case["kind"] == "stdp":
            self.samples, self.steps = 4, case["steps"]
            net, self.scheds = N.stdp_network(seed, case["n_in"], case["n"], self.samples, self.steps)
        else:
            self.samples, self.steps = 2 * case["classes"], 15
            net, self.scheds = N.resource_stdp_network(seed, self.samples, case["n_in"], case["per_column"],
                                                       case["classes"], steps_per_sample=self.steps)
        self.pops = [(p.uid, p.size) for p in net.populations]
        self.plastic = net.projections[0].uid
        self.backend = GB300Backend()
        self.backend.load_network(net)
        self.backend._init()
        self.shown = 0

    def show(self):
        b, t = self.backend, self.backend.get_step()
        first = (self.shown % self.samples) * self.steps
        self.shown += 1
        for s in self.scheds:
            b.load_spike_schedule(_part(s, first, self.steps), t)
        b.step(self.steps)
        out = [_trains(b, u, n, t, self.steps) for u, n in self.pops]
        return {"spikes": out, "weights": b.read_weights(self.plastic)}


# ------------------------------------------------------------------------------------- the cases


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _layer_inputs(case, seed):
    g = _generator(seed)
    t, b, n, m = case["T"], case["batch"], case["n_in"], case["n_out"]
    rates = torch.rand(b, n, generator=g, device="cuda") * 0.3
    x = (torch.rand(t, b, n, generator=g, device="cuda") < rates).float()
    w = torch.randn(n, m, generator=g, device="cuda") * (2.0 / n) ** 0.5
    d = torch.randn(t, b, m, generator=g, device="cuda") / (t * b)
    return x, w, d


def prepare(case, seed):
    kind = case["kind"]
    if kind == "network":
        return {"case": case, "net": _Network(case, seed)}
    if kind in ("stdp", "resource"):
        return {"case": case, "net": _Learner(case, seed)}
    if kind == "batched":
        make = batched.uneven_config if case["uneven"] else batched.dense_config
        cfg = make(seed, case["batch"], _sizes(case), case["t_lo"], case["t_hi"], case["rate"])
        return {"case": case, "plan": batched.BatchedPlan(cfg, record=case["record"])}
    if kind == "layer":
        x, w, d = _layer_inputs(case, seed)
        return {"case": case, "x": x.requires_grad_(), "w": w.requires_grad_(), "d": d}
    if kind == "train":
        sizes = _sizes(case)
        x, labels = bptt.make_batch(case["T"], case["batch"], sizes[0], sizes[-1], seed=seed)
        model = bptt.SpikingMLP(sizes, BETA, THETA, seed=seed)
        opt = torch.optim.SGD(model.parameters(), lr=LEARNING_RATE)
        return {"case": case, "model": model, "step": bptt.GraphedTrainStep(model, opt, x, labels, WARMUP_ITERATIONS)}
    g = _generator(seed)
    a = torch.randn(case["M"], case["K"], generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(case["N"], case["K"], generator=g, device="cuda").to(torch.bfloat16)
    return {"case": case, "a": a, "b": b}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "network":
        net = state["net"]
        if case["online"]:
            return [net.step_online() for _ in range(case["steps"])]
        return net.window(case["steps"])
    if kind in ("stdp", "resource"):
        return state["net"].show()
    if kind == "batched":
        plan = state["plan"]
        events, _ = plan.run()
        out = {"events": events, "counts": plan.counts()}
        if case["record"]:
            out["record"] = [r for _, r in sorted(plan.record().items())]
        return out
    if kind == "layer":
        s = bptt.LIFLayerFn.apply(state["x"], state["w"], BETA, THETA, 8, False, SLOPE)
        dx, dw = torch.autograd.grad(s, (state["x"], state["w"]), state["d"])
        return {"spikes": s.detach(), "dx": dx, "dw": dw}
    if kind == "train":
        loss = state["step"]()
        return {"loss": loss.detach(), "weights": [p.detach() for p in state["model"].parameters()]}
    return bptt.gemm_tn(state["a"], state["b"])


def work(case):
    kind = case["kind"]
    if kind == "network":
        # A neuron's potential, threshold and counter and its input read and written; a synaptic event's
        # target, weight and delay read.
        r = _rate(case)
        events = case["n"] * r * case["fan_in"] + case["p_in"] * (case["n_in"] * case["n"] or case["n"])
        return {"bytes": case["steps"] * (32 * case["n"] + 9 * events), "flops": case["steps"] * events}
    if kind == "stdp":
        # About 1.2 % of the inputs and one neuron fire each step.
        events = 0.012 * case["n_in"] * case["n"] + case["n"]
        return {"bytes": case["steps"] * (64 * case["n"] + 9 * events) + 4 * case["n_in"] * case["n"],
                "flops": case["steps"] * events}
    if kind == "resource":
        n = case["classes"] * case["per_column"]  # about 1.6 % of the inputs fire each step
        events = 0.016 * case["n_in"] * n
        return {"bytes": 15 * (64 * n + 9 * events) + 4 * case["n_in"] * n, "flops": 15 * events}
    if kind == "batched":
        s = _sizes(case)
        rows = case["batch"] * (case["t_lo"] + case["t_hi"]) / 2
        pairs = sum(a * b for a, b in zip(s[:-1], s[1:]))
        bits = rows * sum(s) / 8 if case["record"] else 0
        return {"bytes": 2 * pairs + 4 * case["batch"] * (s[0] + s[-1]) + bits, "flops": 2 * rows * pairs}
    if kind == "layer":
        rows, n, m = case["T"] * case["batch"], case["n_in"], case["n_out"]
        # Spikes in and their gradient, spikes out and their gradient, weights and their gradient; three products.
        return {"bytes": 4 * (2 * rows * n + 2 * rows * m + 2 * n * m), "flops": 6 * rows * n * m}
    if kind == "train":
        s = _sizes(case)
        rows = case["batch"] * case["T"]
        pairs = sum(a * b for a, b in zip(s[:-1], s[1:]))
        return {"bytes": 4 * rows * s[0] + 12 * pairs, "flops": 2 * rows * (3 * pairs - s[0] * s[1])}
    m, n, k = case["M"], case["N"], case["K"]
    return {"bytes": 2 * (m * k + n * k) + 4 * m * n, "flops": 2 * m * n * k}


# ------------------------------------------------------------------------------------- in 64 bits


def _lif64(current):
    """Spikes and membrane values before the reset, over the steps of ``current`` [T, B, n]."""
    beta = float(np.float32(BETA))
    v = torch.zeros_like(current[0])
    us, ss = [], []
    for x in current:
        u = beta * v + x
        s = (u > THETA).double()
        v = u - THETA * s
        us.append(u)
        ss.append(s)
    return torch.stack(us), torch.stack(ss)


def _lif64_backward(us, ds):
    beta = float(np.float32(BETA))
    dv = torch.zeros_like(us[0])
    out = [None] * us.shape[0]
    for t in range(us.shape[0] - 1, -1, -1):
        g = 0.5 * SLOPE / (1.0 + SLOPE * (us[t] - THETA).abs()) ** 2
        du = ds[t] * g + dv * (1.0 - THETA * g)
        dv = beta * du
        out[t] = du
    return torch.stack(out)


def _layer64(x, w):
    """Forward of one layer: the weights take part as BF16 values."""
    wb = w.float().to(torch.bfloat16).double()
    us, s = _lif64(x @ wb)
    return wb, us, s


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        x, w, d = (v.double() for v in _layer_inputs(case, seed))
        wb, us, s = _layer64(x, w)
        di = _lif64_backward(us, d)
        return {"spikes": s, "dx": di @ wb.t(), "dw": x.flatten(0, 1).t() @ di.flatten(0, 1)}
    if kind == "train":
        sizes = _sizes(case)
        g = torch.Generator(device="cpu").manual_seed(seed)
        rates = torch.rand(case["batch"], sizes[0], generator=g) * 0.3
        x = (torch.rand(case["T"], case["batch"], sizes[0], generator=g) < rates).double().cuda()
        labels = torch.randint(0, sizes[-1], (case["batch"],), generator=g).cuda()
        g = torch.Generator(device="cpu").manual_seed(seed)
        ws = [(torch.randn(a, b, generator=g) * (2.0 / a) ** 0.5).double().cuda()
              for a, b in zip(sizes[:-1], sizes[1:])]
        for _ in range(WARMUP_ITERATIONS + 1):
            acts, saved = [x], []
            for w in ws:
                wb, us, s = _layer64(acts[-1], w)
                saved.append((wb, us))
                acts.append(s)
            counts = acts[-1].sum(0)
            loss = torch.nn.functional.cross_entropy(counts, labels)
            one_hot = torch.nn.functional.one_hot(labels, sizes[-1]).double()
            ds = ((counts.softmax(1) - one_hot) / case["batch"]).expand_as(acts[-1])
            for k in range(len(ws) - 1, -1, -1):
                wb, us = saved[k]
                di = _lif64_backward(us, ds)
                ds = di @ wb.t()
                ws[k] = ws[k] - LEARNING_RATE * (acts[k].flatten(0, 1).t() @ di.flatten(0, 1))
        return {"loss": loss, "weights": ws}
    if kind == "gemm":
        state = prepare(case, seed)
        return state["a"].double() @ state["b"].double().t()
    return None  # spikes and weights that are sums of table entries: compared as they are
