"""Networks whose neurons fire often: the single-barrier form of the step loop
stands back for the loops that deal deliveries to all warps, and returns when
the network has calmed down -- in run() and in nemo_step, with the same
results throughout."""
import numpy as np
import pytest

import nemosim_b200 as nb
from tests import nets

pytestmark = pytest.mark.gpu


def network(n, fanout, rate):
    """Half Poisson sources, half Izhikevich neurons, random signs."""
    net = nb.Network()
    rng = np.random.default_rng(n)
    ids = np.arange(n, dtype=np.uint32)
    net.add_neuron(net.add_neuron_type("PoissonSource"), ids[:n // 2], np.float32(rate))
    net.add_neuron(net.add_neuron_type("Izhikevich"), ids[n // 2:], *nets.exc_neuron_args(0.0)[:4], 4.0, -13.0, -65.0)
    src = np.repeat(ids, fanout)
    net.add_synapse(src, rng.integers(0, n, len(src)).astype(np.uint32), rng.integers(1, 21, len(src)).astype(np.uint32),
                    rng.normal(0.0, 0.3, len(src)).astype(np.float32), np.ones(len(src), np.uint8))
    return net


def set_rates(sims, n, rate):
    for s in sims:
        for i in range(n // 2):
            s.set_neuron_parameter(i, 0, rate)


def same(a, b, steps, period, n):
    ra, rb = a.run(steps, period, 0.1, max_ids=steps * n), b.run(steps, period, 0.1, max_ids=steps * n)
    assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[1], rb[1]) and np.array_equal(ra[2], rb[2])


def same_end(a, b, n, fanout, stdp):
    x, y = a.type_state(1, 2, n - n // 2), b.type_state(1, 2, n - n // 2)
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    if stdp:
        assert np.array_equal(a.weights_fx(n * fanout), b.weights_fx(n * fanout))


@pytest.mark.parametrize("stdp", [False, True])
@pytest.mark.parametrize("n,form", [(600, "local_run_kernel<1>"), (3000, "local_run_kernel<2>")])
def test_run(n, form, stdp):
    fanout, period = 60, 25 if stdp else 0
    a, b = (nb.Simulation(network(n, fanout, 0.7), nets.standard_stdp(nb) if stdp else nb.Configuration()) for _ in range(2))
    b.set_launch(64, 128)  # the persistent loop throughout
    assert a.step_kernel() == form
    same(a, b, 20, period, n)
    assert a.step_kernel() == form  # too few steps to judge
    same(a, b, 700, period, n)
    assert a.step_kernel() == "run_kernel"
    set_rates((a, b), n, 0.01)
    same(a, b, 100, period, n)
    assert a.step_kernel() == form
    same(a, b, 700, period, n)
    assert a.step_kernel() == form
    set_rates((a, b), n, 0.7)
    for steps in (1, 2, 30, 1, 40):  # delays up to 20 ms fill first
        same(a, b, steps, period, n)
    assert a.step_kernel() == "run_kernel"
    same(a, b, 50, period, n)
    same_end(a, b, n, fanout, stdp)


@pytest.mark.parametrize("stdp", [False, True])
@pytest.mark.parametrize("n,form", [(600, "local_run_kernel<1>"), (3000, "local_run_kernel<2>")])
def test_nemo_step(n, form, stdp):
    """The busiest warp's load comes with the answers."""
    fanout = 60
    a, b = (nb.Simulation(network(n, fanout, 0.7), nets.standard_stdp(nb) if stdp else nb.Configuration()) for _ in range(2))
    b.set_resident_step(0)
    rng = np.random.default_rng(1)

    def steps(count, reward_every):
        for k in range(count):
            f = rng.choice(n, k % 8, replace=False).tolist()
            assert list(a.step(f)) == list(b.step(f))
            if stdp and k % reward_every == reward_every - 1:
                a.apply_stdp(0.1)
                b.apply_stdp(0.1)

    assert a.step_kernel() == form
    steps(100, 40)
    assert a.step_kernel() == "run_kernel"
    steps(30, 3)
    set_rates((a, b), n, 0.01)
    steps(70, 40)
    assert a.step_kernel() == form
    steps(100, 1)  # a launch per step: the window spans launches
    assert a.step_kernel() == form
    set_rates((a, b), n, 0.7)
    steps(100, 1)
    assert a.step_kernel() == "run_kernel"
    assert a.step_events() == b.step_events()
    same_end(a, b, n, fanout, stdp)


def test_calm_after_a_resident_loop_of_a_very_busy_network():
    """What the loop had counted when it was stopped, a hundred rounds a step,
    does not weigh on the calm network later."""
    n, fanout = 600, 390
    a, b = (nb.Simulation(network(n, fanout, 1.0), nb.Configuration()) for _ in range(2))
    b.set_resident_step(0)
    assert [list(a.step()) for _ in range(70)] == [list(b.step()) for _ in range(70)]
    assert a.step_kernel() == "run_kernel"
    set_rates((a, b), n, 0.001)
    assert [list(a.step()) for _ in range(200)] == [list(b.step()) for _ in range(200)]
    assert a.step_kernel() == "local_run_kernel<1>"


def test_two_launch_shape_of_a_large_learning_network():
    """Without a shape of the caller's, the two-launch step of a large network
    with STDP takes wider partitions while the network fires often."""
    n, sources = 230_000, 11_500
    rng = np.random.default_rng(3)

    def build():
        net = nb.Network()
        ids = np.arange(n, dtype=np.uint32)
        net.add_neuron(net.add_neuron_type("PoissonSource"), ids[:sources], np.float32(0.6))
        net.add_neuron(net.add_neuron_type("IzhikevichRS"), ids[sources:], -13.0, -65.0)
        r = np.random.default_rng(4)
        # a hub of out-degree 401: not one kernel per step
        src = np.concatenate([np.repeat(ids, 3), np.full(398, 9)]).astype(np.uint32)
        net.add_synapse(src, r.integers(0, n, len(src)).astype(np.uint32), r.integers(1, 21, len(src)).astype(np.uint32),
                        np.full(len(src), 2.0, np.float32), np.ones(len(src), np.uint8))
        return nb.Simulation(net, nets.standard_stdp(nb))

    a, b = build(), build()
    b.set_persistent(False)
    b.set_launch(256, 256)
    assert a.step_kernel() == "update_kernel" and a.launch() == (128, 128)
    a.set_launch(*a.launch())  # changes nothing
    same(a, b, 130, 50, n)
    wide = a.launch()
    assert wide[0] > 256 and wide[1] > 256
    same(a, b, 130, 50, n)
    assert a.launch() == wide
    for s in (a, b):
        for i in rng.permutation(sources).tolist():
            s.set_neuron_parameter(i, 0, 0.001)
    same(a, b, 130, 50, n)
    assert a.launch() == (128, 128)
    same(a, b, 30, 0, n)
    assert list(a.step([5])) == list(b.step([5]))
    a.set_launch(96, 96)
    same(a, b, 20, 0, n)
    assert a.launch() == (96, 96)
    assert np.array_equal(a.weights_fx(3 * n + 398), b.weights_fx(3 * n + 398))
