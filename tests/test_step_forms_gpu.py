"""Which form of the step loop a network takes, on both sides of each rule,
and that this form -- not another that stepped in for it -- gives the
oracle's fire stream and its state, bit for bit."""
import numpy as np
import pytest

import nemosim_b200 as nb
import oracle as O
from tests import nets
from tests.test_single_barrier_gpu import conf, typed_network

pytestmark = pytest.mark.gpu

CLUSTER, GRID, BALANCED = "local_run_kernel<1>", "local_run_kernel<2>", "balanced_run_kernel"


def same_bits(a, b):
    """NaN for NaN, whatever its payload, and every other value by its bits."""
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return np.array_equal(np.where(np.isnan(a), np.float32(np.nan), a).view(np.uint32),
                          np.where(np.isnan(b), np.float32(np.nan), b).view(np.uint32))


def assert_same(sp, so, parts, steps, period, n):
    cp, _, ip = sp.run(steps, period, 0.7, max_ids=steps * n + 1)
    co, io = so.run(steps, period, 0.7, max_ids=steps * n + 1)
    assert np.array_equal(cp, co) and np.array_equal(ip, io)
    for t, ns in ((0, 2), (1, 4), (4, 2)):
        if len(parts[t]):
            assert same_bits(sp.type_state(t, ns, len(parts[t])), so.type_state(t, ns, len(parts[t])))


# 2048 neurons | one cluster; out-degree 400 and, with STDP, a plastic
# in-degree of 320 (224 beyond 12288 neurons and for one kernel per step):
# the single barrier.  Largest plastic in-degrees of these networks, in turn:
# 49, 292, 294, 415, 200, 234.
@pytest.mark.parametrize("n,fanout,dmax,stdp,form,one_kernel", [
    (1, 1, 1, False, CLUSTER, True), (2048, 40, 20, False, CLUSTER, True), (2049, 40, 20, False, GRID, True),
    (700, 400, 20, False, CLUSTER, True), (700, 401, 20, False, BALANCED, False), (2048, 40, 20, True, CLUSTER, True),
    (2500, 400, 20, True, GRID, False), (2500, 401, 20, True, BALANCED, False), (500, 600, 20, True, BALANCED, False),
    (13000, 250, 10, True, GRID, True), (13000, 300, 10, True, BALANCED, False)])
def test_form_and_results(n, fanout, dmax, stdp, form, one_kernel):
    (pn, parts), (on, _) = typed_network(nb, n, fanout, dmax, 0.05, 6), typed_network(O, n, fanout, dmax, 0.05, 6)
    sp, so = nb.Simulation(pn, conf(nb, stdp)), O.Simulation(on, conf(O, stdp))
    assert sp.step_kernel() == form
    assert_same(sp, so, parts, 60, 25 if stdp else 0, n)
    after = sp.step_kernel()
    assert after in (form, "run_kernel")  # the latter where those steps were busy
    sp.set_persistent(False)
    assert sp.step_kernel() == ("fused_step_kernel" if one_kernel else "update_kernel")
    assert_same(sp, so, parts, 30, 25 if stdp else 0, n)
    sp.set_launch(64, 96)
    assert sp.step_kernel() == "update_kernel"
    sp.set_persistent(True)
    assert sp.step_kernel() == after
    sp.set_launch(64, 96)
    assert sp.step_kernel() == "run_kernel"
    assert_same(sp, so, parts, 30, 25 if stdp else 0, n)


def test_types_beyond_the_forms():
    net = nb.Network()
    k = net.add_neuron_type("Kuramoto")
    net.add_neuron(k, np.arange(40, dtype=np.uint32), np.float32(0.1), np.float32(0.0))
    net.add_synapse(np.array([0], np.uint32), np.array([1], np.uint32), np.ones(1, np.uint32), np.full(1, 0.1, np.float32),
                    np.zeros(1, np.uint8))
    sim = nb.Simulation(net, nb.Configuration())
    assert sim.step_kernel() == "run_kernel"
    sim.set_persistent(False)
    assert sim.step_kernel() == "update_kernel"


@pytest.mark.parametrize("persistent", [True, False])
@pytest.mark.parametrize("n,fanout", [(700, 40), (3000, 40), (700, 450)])
def test_setting_the_reported_shape_changes_nothing(n, fanout, persistent):
    a, b = (nb.Simulation(nb.example_random(n, fanout, 20, True), nets.standard_stdp(nb)) for _ in range(2))
    for s in (a, b):
        s.set_persistent(persistent)
    form, shape = a.step_kernel(), a.launch()
    a.set_launch(*shape)
    assert (a.step_kernel(), a.launch()) == (form, shape) == (b.step_kernel(), b.launch())
    ra, rb = a.run(130, 50, 1.0), b.run(130, 50, 1.0)
    assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[2], rb[2])
    a.set_launch(96, 192)
    assert a.launch() == (96, 192) and a.step_kernel() == ("run_kernel" if persistent else "update_kernel")
    a.set_launch(*a.launch())
    assert a.launch() == (96, 192) and a.step_kernel() == ("run_kernel" if persistent else "update_kernel")
    a.autotune(5)
    ra, rb = a.run(130, 50, 1.0), b.run(130, 50, 1.0)
    assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[2], rb[2])


def noisy_network(n, noisy, hub):
    """n Izhikevich neurons, the first `noisy` with input noise, three synapses
    each and, with a hub, one of out-degree 401 (the balanced form)."""
    net = nb.Network()
    sigma = np.where(np.arange(n) < noisy, 6.0, 0.0).astype(np.float32)
    ids = np.arange(n, dtype=np.uint32)
    net.add_neuron(net.add_neuron_type("Izhikevich"), ids, *nets.exc_neuron_args(0.0)[:4], sigma, -13.0, -65.0)
    rng = np.random.default_rng(n)
    src = np.concatenate([np.repeat(ids, 3), np.full(398 if hub else 0, 5)]).astype(np.uint32)
    net.add_synapse(src, rng.integers(0, n, len(src)).astype(np.uint32), rng.integers(1, 21, len(src)).astype(np.uint32),
                    np.full(len(src), 4.0, np.float32), np.zeros(len(src), np.uint8))
    return net


# words of 32 neurons per CTA, neurons beyond, the noisy share; 27, 28, 29 and
# 30 worker warps leave 4, 3, 2 and 1 warps for the noise (a word of 32 neurons
# costs a draw when one of them is noisy)
@pytest.mark.parametrize("words,more,noisy,hub,form", [
    (28, 0, 1.0, False, GRID), (28, 1, 1.0, False, "run_kernel"), (28, 1, 0.5, False, GRID), (30, 0, 0.25, False, GRID),
    (30, 0, 0.5, False, "run_kernel"), (30, 0, 0.0, False, GRID), (27, 0, 1.0, True, BALANCED), (27, 1, 1.0, True, "run_kernel"),
    (27, 1, 0.5, True, BALANCED)])
def test_noise_limit(words, more, noisy, hub, form):
    import torch
    n = words * 32 * torch.cuda.get_device_properties(0).multi_processor_count + more
    a, b = (nb.Simulation(noisy_network(n, int(noisy * n), hub), nb.Configuration()) for _ in range(2))
    assert a.step_kernel() == form
    b.set_persistent(False)
    b.set_launch(256, 256)
    for steps in (1, 60):
        ra, rb = a.run(steps, max_ids=steps * n), b.run(steps, max_ids=steps * n)
        assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[2], rb[2])
        # served by the same form up to 29 worker warps
        assert [list(a.step([k])) for k in range(10)] == [list(b.step([k])) for k in range(10)]
    assert noisy == 0 or ra[0].sum() > 0
    assert same_bits(a.type_state(0, 2, n), b.type_state(0, 2, n))


@pytest.mark.parametrize("n,fanout", [(700, 450), (20_001, 420), (40_001, 420)])
def test_brief_runs_of_the_balanced_form(n, fanout):
    """Segments on both sides of the length from which the balanced form pays
    (one step per 20000 neurons, two at least), one after the other."""
    a, b = (nb.Simulation(nb.example_random(n, fanout, 20, True), nets.standard_stdp(nb)) for _ in range(2))
    assert a.step_kernel() == BALANCED
    b.set_launch(256, 384)
    assert b.step_kernel() == "run_kernel"
    for steps, period in ((60, 0), (1, 0), (1, 1), (2, 0), (3, 1), (1, 0), (12, 2), (3, 0), (15, 4), (40, 0)):
        ra, rb = a.run(steps, period, 0.5, max_ids=steps * n), b.run(steps, period, 0.5, max_ids=steps * n)
        assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[1], rb[1]) and np.array_equal(ra[2], rb[2])
        assert list(a.step([5])) == list(b.step([5]))
    assert ra[0].sum() > 0
    assert same_bits(a.type_state(0, 2, n), b.type_state(0, 2, n))
    assert np.array_equal(a.weights_fx(n * fanout), b.weights_fx(n * fanout))


def test_resident_launches_of_one_step():
    """The balanced form gives way to the persistent loop after launches that
    served one step, and returns after one that served more."""
    n, fanout = 900, 430
    a, b = (nb.Simulation(nb.example_random(n, fanout, 20, True), nets.standard_stdp(nb)) for _ in range(2))
    assert a.step_kernel() == BALANCED
    b.set_resident_step(0)
    for length in (1, 1, 1, 5, 1, 1, 30, 2, 1, 1, 1, 7):
        for k in range(length):
            f, i = [k, 3 * k + 1], [(n - 1 - k, 12.0)] if k % 2 else None
            assert list(a.step(f, i)) == list(b.step(f, i))
        for s in (a, b):
            s.apply_stdp(0.5)
            s.set_neuron_state(7, 0, -12.0)
        ra, rb = a.run(2, max_ids=2 * n), b.run(2, max_ids=2 * n)
        assert np.array_equal(ra[2], rb[2])
    assert same_bits(a.type_state(0, 2, n), b.type_state(0, 2, n))
    assert np.array_equal(a.weights_fx(n * fanout), b.weights_fx(n * fanout))
