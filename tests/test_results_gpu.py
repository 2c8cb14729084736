"""Results that leave the device: run()'s fire stream, counts and events,
the state rows and the weights in network iteration order, at the sizes where
their kernels' tiles and staging memory end.  Whole numbers: equal to the
oracle's."""
import numpy as np
import pytest

import nemosim_b200 as nb
import oracle as O
from tests import nets

pytestmark = pytest.mark.gpu


def firing_network(mod, n, rate, stride, seed):
    """n Poisson sources with scattered ids, each connected to its neighbour."""
    net = mod.Network()
    t = net.add_neuron_type("PoissonSource")
    ids = (np.random.default_rng(seed).permutation(n) * stride + 3).astype(np.uint32)
    net.add_neuron(t, ids, np.float32(rate))
    net.add_synapse(ids, np.roll(ids, 1), np.full(n, 2, np.uint32), np.full(n, 0.5, np.float32), np.zeros(n, np.uint8))
    return net


# one neuron, a bit-vector word more or less, a tile of 512 words more or
# less; every neuron firing every step, so that 1100 steps (two ring lengths)
# exceed the staging memory many times and a tile exceeds its shared ids
@pytest.mark.parametrize("n,rate,stride,steps", [(1, 1.0, 1, 1100), (31, 1.0, 7, 40), (33, 1.0, 1, 1100), (500, 0.3, 2, 1100),
                                                 (16384, 0.02, 1, 60), (16385, 1.0, 3, 40), (33000, 0.2, 1, 25)])
def test_fire_stream(n, rate, stride, steps):
    sp = nb.Simulation(firing_network(nb, n, rate, stride, 5), nb.Configuration())
    so = O.Simulation(firing_network(O, n, rate, stride, 5), O.Configuration())
    for part in (steps, 7):
        cp, ep, ip = sp.run(part, max_ids=part * n + 1)
        co, io = so.run(part, max_ids=part * n + 1)
        assert np.array_equal(cp, co) and np.array_equal(ep, cp) and np.array_equal(ip, io)


# an answer of one word of neurons or many, on both sides of the 4096 ids it
# carries word by word
@pytest.mark.parametrize("n,stride", [(1, 1), (33, 3), (1024, 1), (1025, 2), (4096, 1), (4097, 1), (9000, 2)])
def test_step_answers(n, stride):
    sp = nb.Simulation(firing_network(nb, n, 1.0, stride, 5), nb.Configuration())
    so = O.Simulation(firing_network(O, n, 1.0, stride, 5), O.Configuration())
    for _ in range(4):
        assert list(sp.step()) == list(so.step())
    assert sp.step_events() == 4 * n


def test_fire_stream_longer_than_the_callers_buffer():
    sp = nb.Simulation(firing_network(nb, 100, 1.0, 1, 5), nb.Configuration())
    with pytest.raises(nb.NemoError):
        sp.run(10, max_ids=999)
    assert len(sp.run(10, max_ids=1000)[2]) == 1000


@pytest.mark.parametrize("count", [2, 5])
def test_batch_stream_of_interleaved_types(count):
    """Networks of several types, listed in different orders, are not
    contiguous in a batch: their streams come back in each one's own order."""
    def network(mod, k):
        net = mod.Network()
        names = ["PoissonSource", "Izhikevich"] if k % 2 else ["Izhikevich", "PoissonSource"]
        for i, name in enumerate(names):
            t = net.add_neuron_type(name)
            ids = np.arange(40 + 11 * k, dtype=np.uint32) * 2 + i
            if name == "PoissonSource":
                net.add_neuron(t, ids, np.float32(0.2))
            else:
                net.add_neuron(t, ids, *nets.exc_neuron_args(5.0))
        net.add_synapse(ids, np.roll(ids, 1), np.full(len(ids), 1 + k, np.uint32), np.full(len(ids), 3.0, np.float32),
                        np.zeros(len(ids), np.uint8))
        return net
    batch = nb.Batch([network(nb, k) for k in range(count)], nb.Configuration())
    counts, _, ids = batch.run(120)
    for k, (c, i) in enumerate(batch.streams(counts, ids)):
        co, io = O.Simulation(network(O, k), O.Configuration()).run(120, max_ids=120 * 300)
        assert np.array_equal(c, co) and np.array_equal(i, io)


@pytest.mark.parametrize("device", [True, False])
@pytest.mark.parametrize("queried", [True, False])
@pytest.mark.parametrize("scattered", [True, False])
def test_weights_and_state(device, queried, scattered):
    """Weights in network iteration order after learning, from a device-built
    and a host-built network, before and after a synapse query, with global
    ids in and out of local order."""
    def network(mod):
        if not scattered:
            return mod.example_random(700, 50, 20, True)
        return nets.create_ring(mod, mod.Network(), 777, n0=5, plastic=True, nstep=3)
    conf_p, conf_o = nets.standard_stdp(nb), nets.standard_stdp(O)
    conf_p.set_device_construction(device)
    net = network(nb)
    sp, so = nb.Simulation(net, conf_p), O.Simulation(network(O), conf_o)
    n = 700 if not scattered else 777
    first = 0 if not scattered else 5
    if queried:
        assert len(sp.get_synapses_from(first)) == (50 if not scattered else 1)
    for _ in range(2):
        sp.run(60, 30, 1.0)
        so.run(60, 30, 1.0, max_ids=60 * n)
        nsyn = sp.synapse_count()
        assert np.array_equal(sp.weights_fx(nsyn), so.weights_fx(nsyn))
        assert np.array_equal(sp.type_state(0, 2, n).view(np.uint32), so.type_state(0, 2, n).view(np.uint32))
