"""The single-barrier step loop, which run() and step() take for networks of
moderate degree, against the oracle and against the other loops: the same
fire stream, state and weights, bit for bit, at the edges of its shapes
(words of 32 neurons round the CTAs, one cluster up to 2048 neurons, a warp's
list of 128 groups), for every neuron type it holds, and across switches
between the loops in the middle of a simulation."""
import numpy as np
import pytest

import nemosim_b200 as nb
import oracle as O
from tests import nets

pytestmark = pytest.mark.gpu


def typed_network(mod, n, fanout, dmax, rate, seed):
    """n neurons of every type but Kuramoto, interleaved ids, random signs."""
    rng = np.random.default_rng(seed)
    net = mod.Network()
    ids = (rng.permutation(n) + 10).astype(np.uint32)
    parts = np.array_split(ids, 5)
    types = [net.add_neuron_type(t) for t in ("Izhikevich", "IF_curr_exp", "PoissonSource", "Input", "IzhikevichRS")]
    if len(parts[0]):
        net.add_neuron(types[0], parts[0], *nets.exc_neuron_args(0.0)[:4], rng.choice([0.0, 4.0], len(parts[0])), -13.0, -65.0)
    if len(parts[1]):
        net.add_neuron(types[1], parts[1], -65.0, -65.0, 1.0, 20.0, 2.0, 5.0, 5.0, -50.0, 0.0, -65.0, 0.0, 0.0, 1000.0)
    if len(parts[2]):
        net.add_neuron(types[2], parts[2], np.float32(rate))
    if len(parts[3]):
        net.add_neuron(types[3], parts[3])
    if len(parts[4]):
        net.add_neuron(types[4], parts[4], -13.0, -65.0)
    src = np.repeat(ids, fanout)
    tgt = rng.choice(ids, len(src)).astype(np.uint32)
    w = (rng.lognormal(0.0, 1.0, len(src)) * rng.choice([1, 1, 1, -1], len(src))).astype(np.float32)
    net.add_synapse(src, tgt, rng.integers(1, dmax + 1, len(src)).astype(np.uint32), w,
                    (rng.random(len(src)) < 0.6).astype(np.uint8))
    return net, parts


def conf(mod, stdp):
    return nets.standard_stdp(mod) if stdp else mod.Configuration()


def assert_same_state(sp, so, parts):
    for t, ns in ((0, 2), (1, 4), (4, 2)):
        if len(parts[t]):
            a, b = sp.type_state(t, ns, len(parts[t])), so.type_state(t, ns, len(parts[t]))
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) or np.array_equal(a, b, equal_nan=True)


# one word and part of one, one CTA more or fewer words, both sides of the
# cluster's limit and of one word per CTA (4736), one delay and the longest,
# groups beyond a warp's list (rate 1: every delay of every source pending)
@pytest.mark.parametrize("n,fanout,dmax,rate,stdp", [
    (5, 3, 1, 0.5, False), (32, 6, 63, 0.3, False), (33, 20, 44, 0.3, True), (511, 40, 20, 0.1, True),
    (2047, 30, 20, 0.05, True), (2048, 50, 1, 0.05, False), (2049, 50, 20, 0.05, True), (4736, 20, 10, 0.05, True),
    (4737, 20, 10, 0.05, False), (300, 60, 60, 1.0, False), (3000, 60, 44, 1.0, True), (20000, 12, 33, 0.02, True)])
def test_matches_oracle(n, fanout, dmax, rate, stdp):
    (pn, parts), (on, _) = typed_network(nb, n, fanout, dmax, rate, 3), typed_network(O, n, fanout, dmax, rate, 3)
    sp, so = nb.Simulation(pn, conf(nb, stdp)), O.Simulation(on, conf(O, stdp))
    for steps in (1, 2, 57, 40):
        cp, _, ip = sp.run(steps, 19 if stdp else 0, 0.7, max_ids=steps * n + 1)
        co, io = so.run(steps, 19 if stdp else 0, 0.7, max_ids=steps * n + 1)
        assert np.array_equal(cp, co) and np.array_equal(ip, io)
    assert_same_state(sp, so, parts)
    if stdp:
        assert np.array_equal(sp.weights_fx(n * fanout), so.weights_fx(n * fanout))


@pytest.mark.parametrize("n", [700, 3000])
@pytest.mark.parametrize("stdp", [True, False])
def test_switching_loops_mid_run(n, stdp):
    """run() and step() through every loop in turn: pending deliveries, STDP
    not yet accumulated and noise drawn ahead pass from each to the next."""
    (pn, parts), (on, _) = typed_network(nb, n, 40, 30, 0.1, 4), typed_network(O, n, 40, 30, 0.1, 4)
    sp, so = nb.Simulation(pn, conf(nb, stdp)), O.Simulation(on, conf(O, stdp))
    rng = np.random.default_rng(2)
    ids = np.concatenate(parts)

    def run(steps):
        cp, _, ip = sp.run(steps, 7 if stdp else 0, 1.0, max_ids=steps * n + 1)
        co, io = so.run(steps, 7 if stdp else 0, 1.0, max_ids=steps * n + 1)
        assert np.array_equal(cp, co) and np.array_equal(ip, io)

    def step(count, no_alloc=False):
        for k in range(count):
            f = rng.choice(ids, k % 9, replace=False).tolist()
            i = [(int(a), 20.0) for a in rng.choice(ids, 5, replace=False)] if k % 2 else None
            want = so.step(f, i)
            got = sp.step_no_alloc(f, i)[1] if no_alloc else sp.step(f, i)
            assert list(got) == list(want)
            if stdp and k % 4 == 3:
                sp.apply_stdp(0.9)
                so.apply_stdp(0.9)

    for _ in range(2):
        run(23)
        step(11)
        step(3, no_alloc=True)
        run(9)
        sp.set_persistent(False)
        run(15)
        step(6)
        sp.set_persistent(True)
        step(7)
        sp.set_resident_step(0)
        step(5)
        run(1)
        sp.set_resident_step(200)
        step(4)
        sp.trace_phases(3)  # three steps of the persistent loop
        so.run(3, 0, 1.0, max_ids=3 * n + 1)
        run(12)
    sp.autotune(5)
    run(20)
    sp.set_launch(64, 128)  # the persistent loop from here on
    run(20)
    step(5)
    assert_same_state(sp, so, parts)
    if stdp:
        assert np.array_equal(sp.weights_fx(n * 40), so.weights_fx(n * 40))


@pytest.mark.parametrize("fanout", [399, 400, 401])
def test_degree_limit(fanout):
    """The largest out-degree of the loop and the next one."""
    sp, so = (nb.Simulation(nb.example_random(1500, fanout, 20, False), nb.Configuration()),
              O.Simulation(O.example_random(1500, fanout, 20, False), O.Configuration()))
    cp, _, ip = sp.run(150, max_ids=150 * 1500)
    co, io = so.run(150, max_ids=150 * 1500)
    assert np.array_equal(cp, co) and np.array_equal(ip, io)


@pytest.mark.parametrize("n,fanout,dmax,rate,stdp", [
    (3, 450, 5, 0.5, True), (33, 401, 44, 0.3, True), (700, 500, 20, 0.05, False), (4737, 410, 40, 0.02, True),
    (300, 420, 63, 1.0, False), (300, 420, 44, 1.0, True)])
def test_balanced_form_matches_oracle(n, fanout, dmax, rate, stdp):
    """The two-barrier form of large degrees, with steps between runs."""
    (pn, parts), (on, _) = typed_network(nb, n, fanout, dmax, rate, 8), typed_network(O, n, fanout, dmax, rate, 8)
    sp, so = nb.Simulation(pn, conf(nb, stdp)), O.Simulation(on, conf(O, stdp))
    ids = np.concatenate(parts)
    for k, steps in enumerate((1, 2, 57, 40)):
        cp, _, ip = sp.run(steps, 19 if stdp else 0, 0.7, max_ids=steps * n + 1)
        co, io = so.run(steps, 19 if stdp else 0, 0.7, max_ids=steps * n + 1)
        assert np.array_equal(cp, co) and np.array_equal(ip, io)
        for j in range(5):
            i = [(int(ids[j % n]), 15.0)]
            assert list(sp.step([int(ids[0])], i)) == list(so.step([int(ids[0])], i))
        if k == 1:
            assert list(sp.step_no_alloc()[1]) == list(so.step())
        if k == 2:
            sp.set_persistent(False)
            assert list(sp.run(9, max_ids=9 * n + 1)[2]) == list(so.run(9, max_ids=9 * n + 1)[1])
            sp.set_persistent(True)
    assert_same_state(sp, so, parts)
    if stdp:
        assert np.array_equal(sp.weights_fx(n * fanout), so.weights_fx(n * fanout))


def test_many_synapses_onto_one_neuron():
    """A target whose in-degree exceeds the 65536 arrivals of the cluster's
    split sums, all of them in the same step, with weights of both signs and
    beyond 16 bits."""
    def network(mod):
        net = mod.Network()
        t, i = net.add_neuron_type("PoissonSource"), net.add_neuron_type("Izhikevich")
        src = np.arange(200, dtype=np.uint32)
        net.add_neuron(t, src, np.float32(1.0))
        net.add_neuron(i, np.arange(200, 210, dtype=np.uint32), *nets.exc_neuron_args(1.0))
        s = np.repeat(src, 340)
        w = np.where(np.arange(len(s)) % 2, 3.0001, -2.9999).astype(np.float32)
        net.add_synapse(s, np.full(len(s), 205, np.uint32), np.ones(len(s), np.uint32), w, np.zeros(len(s), np.uint8))
        return net
    sp, so = nb.Simulation(network(nb), nb.Configuration()), O.Simulation(network(O), O.Configuration())
    cp, _, ip = sp.run(40, max_ids=40 * 210)
    co, io = so.run(40, max_ids=40 * 210)
    assert np.array_equal(cp, co) and np.array_equal(ip, io)
    assert np.array_equal(sp.type_state(1, 2, 10).view(np.uint32), so.type_state(1, 2, 10).view(np.uint32))


@pytest.mark.parametrize("stdp", [True, False])
@pytest.mark.parametrize("n", [1, 127, 129, 3000])
def test_fused_step_matches_oracle(n, stdp):
    """The same step as one kernel per step (two-launch mode): without and
    with graphs of 100 steps, and followed by the other loops."""
    fanout = min(n, 40)
    (pn, parts), (on, _) = typed_network(nb, n, fanout, 25, 0.1, 6), typed_network(O, n, fanout, 25, 0.1, 6)
    sp, so = nb.Simulation(pn, conf(nb, stdp)), O.Simulation(on, conf(O, stdp))
    sp.set_persistent(False)
    for k, steps in enumerate((1, 2, 99, 100, 231, 30)):
        if k == 4:
            sp.set_graphs(False)
        if k == 5:
            sp.set_persistent(True)
        period = 110 if stdp else 0
        cp, _, ip = sp.run(steps, period, 0.7, max_ids=steps * n + 1)
        co, io = so.run(steps, period, 0.7, max_ids=steps * n + 1)
        assert np.array_equal(cp, co) and np.array_equal(ip, io)
        got, want = sp.step([int(parts[0][0])] if len(parts[0]) else None), so.step([int(parts[0][0])] if len(parts[0]) else None)
        assert list(got) == list(want)
        sp.set_persistent(k >= 4)
    assert_same_state(sp, so, parts)
    if stdp:
        assert np.array_equal(sp.weights_fx(n * fanout), so.weights_fx(n * fanout))
