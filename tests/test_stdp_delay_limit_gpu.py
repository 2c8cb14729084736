"""STDP with a delay of exactly 64 ms, which an empty post-fire window allows:
the pre-synaptic history of such a synapse is not shifted at all (a shift by
64 acts as one by 0), newest spike included, so its weight follows spikes of
the same millisecond.  At 63 ms, the neighbouring delay, every step form holds."""
import numpy as np
import pytest

import nemosim_b200 as nb
import oracle as O
from tests import nets

pytestmark = pytest.mark.gpu


def network(mod, n, fanout, dmax, seed):
    """n Poisson sources (nothing is delivered at a maximum delay of 64),
    a third of the synapses at the longest delay."""
    rng = np.random.default_rng(seed)
    net = mod.Network()
    ids = (rng.permutation(n) + 5).astype(np.uint32)
    net.add_neuron(net.add_neuron_type("PoissonSource"), ids, np.float32(0.2))
    src = np.repeat(ids, fanout)
    dly = np.where(rng.random(len(src)) < 1 / 3, dmax, rng.integers(1, dmax + 1, len(src))).astype(np.uint32)
    dly[0] = dmax
    net.add_synapse(src, rng.choice(ids, len(src)).astype(np.uint32), dly, rng.uniform(0.5, 2.0, len(src)).astype(np.float32),
                    np.ones(len(src), np.uint8))
    return net


def conf(mod):
    c = mod.Configuration()
    dt = np.arange(1, 21, dtype=np.float32)
    c.set_stdp_function((0.01 * np.exp(-dt / 20)).astype(np.float32), np.zeros(0, np.float32), -10.0, 10.0)
    return c


@pytest.mark.parametrize("dmax", [63, 64])
@pytest.mark.parametrize("n,fanout", [(700, 20), (3000, 12), (60, 500)])
@pytest.mark.parametrize("form", ["run", "step", "kernel_per_step", "two_launches"])
def test_weights_match_the_oracle(n, fanout, dmax, form):
    sp = nb.Simulation(network(nb, n, fanout, dmax, 5), conf(nb))
    so = O.Simulation(network(O, n, fanout, dmax, 5), conf(O))
    if form == "kernel_per_step":
        sp.set_persistent(False)
    if form == "two_launches":
        sp.set_persistent(False)
        sp.set_launch(64, 64)
    for _ in range(2):
        if form == "step":
            for _ in range(90):
                assert list(sp.step()) == list(so.step())
            for s in (sp, so):
                s.apply_stdp(0.5)
        else:
            cp, _, ip = sp.run(130, 65, 0.5, max_ids=130 * n)
            co, io = so.run(130, 65, 0.5, max_ids=130 * n)
            assert cp.sum() > 0 and np.array_equal(cp, co) and np.array_equal(ip, io)
    a, b = sp.weights_fx(n * fanout), so.weights_fx(n * fanout)
    assert len(np.unique(b)) > n
    assert np.array_equal(a, b), int((a != b).sum())
