"""The step loop of one cluster (up to 2048 neurons) over tens of thousands of
barriers, in run() and in nemo_step's resident form: a delivery that an update
does not wait for loses the spike of a ring for good, and changes the fire
stream of a random network."""
import numpy as np
import pytest

import nemosim_b200 as nb
from tests import nets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 700, 2048])
def test_ring_keeps_its_spike(n):
    sim = nb.Simulation(nets.create_ring(nb, nb.Network(), n), nb.Configuration())
    assert list(sim.step([0])) == [0]
    steps = 20_000
    counts, _, ids = sim.run(steps, max_ids=2 * steps)
    assert np.array_equal(counts, np.ones(steps))
    assert np.array_equal(ids, (1 + np.arange(steps)) % n)
    for k in range(3000):
        fired = list(sim.step())
        assert fired == [(steps + 1 + k) % n], (k, fired)


@pytest.mark.parametrize("n,fanout", [(64, 30), (1000, 100), (2047, 60)])
def test_long_run_matches_the_persistent_loop(n, fanout):
    a, b = (nb.Simulation(nb.example_random(n, fanout, 20, True), nets.standard_stdp(nb)) for _ in range(2))
    b.set_launch(64, 128)  # the persistent loop
    steps = 10_000
    ra, rb = (s.run(steps, 500, 0.01, max_ids=steps * n) for s in (a, b))
    assert ra[0].sum() > 0
    assert np.array_equal(ra[0], rb[0]) and np.array_equal(ra[2], rb[2])
    assert [list(a.step([k % n])) for k in range(1000)] == [list(b.step([k % n])) for k in range(1000)]
    assert np.array_equal(a.type_state(0, 2, n).view(np.uint32), b.type_state(0, 2, n).view(np.uint32))
    assert np.array_equal(a.weights_fx(n * fanout), b.weights_fx(n * fanout))
