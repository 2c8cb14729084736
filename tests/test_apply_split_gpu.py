"""applyStdp with its items dealt to several warps: the weights of the oracle,
bit for bit, at the edges of the split (1, 2, 4, ... warps an item, items
shorter than the mean, a last word of few neurons, all synapses onto one
neuron)."""
import numpy as np
import pytest

import nemosim_b200 as nb
import oracle as O
from tests import nets
from tests.test_single_barrier_gpu import typed_network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,fanout", [(32, 13), (32, 14), (33, 20), (65, 27), (320, 54), (1000, 100), (257, 300)])
def test_weights(n, fanout):
    (pn, _), (on, _) = typed_network(nb, n, fanout, 20, 0.1, 6), typed_network(O, n, fanout, 20, 0.1, 6)
    sp = nb.Simulation(pn, nets.standard_stdp(nb))
    so = O.Simulation(on, nets.standard_stdp(O))
    for reward in (1.0, 0.3, -0.5):  # the first call also clamps
        sp.run(40, 0, 0.0)
        so.run(40, 0, 0.0)
        sp.apply_stdp(reward)
        so.apply_stdp(reward)
        assert np.array_equal(sp.weights_fx(n * fanout), so.weights_fx(n * fanout))


def test_one_target():
    def build(mod):
        net = mod.Network()
        t = net.add_neuron_type("PoissonSource")
        z = net.add_neuron_type("Izhikevich")
        ids = np.arange(700, dtype=np.uint32)
        net.add_neuron(t, ids[:699], np.float32(0.1))
        net.add_neuron(z, ids[699:], *nets.exc_neuron_args(0.0)[:4], 4.0, -13.0, -65.0)
        src = np.repeat(ids[:699], 5)
        net.add_synapse(src, np.full(len(src), 699, np.uint32), np.arange(len(src), dtype=np.uint32) % 20 + 1,
                        np.full(len(src), 0.7, np.float32), np.ones(len(src), np.uint8))
        return net, len(src)

    (pn, m), (on, _) = build(nb), build(O)
    sp, so = nb.Simulation(pn, nets.standard_stdp(nb)), O.Simulation(on, nets.standard_stdp(O))
    for _ in range(2):
        sp.run(60, 20, 0.8)
        so.run(60, 20, 0.8)
        assert np.array_equal(sp.weights_fx(m), so.weights_fx(m))
