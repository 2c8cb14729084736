"""The bounded waits of every form of the step loop: with a limit of zero
polls (tests/test_bounded_waits_gpu.py) a wait of one cluster, of the grid
and of the balanced form runs out at once on a healthy GPU, in run() and in
nemo_step's resident loop; the call reports it and the device goes on."""
import pytest

import nemosim_b200 as nb
from tests import nets
from tests.test_bounded_waits_gpu import NEMO_CUDA_ERROR, fresh_sim_is_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resident", [False, True])
@pytest.mark.parametrize("n,fanout,form", [
    (700, 60, "local_run_kernel<1>"), (3000, 60, "local_run_kernel<2>"), (3000, 450, "balanced_run_kernel"),
    (3000, 60, "run_kernel")])
def test_wait_runs_out(n, fanout, form, resident):
    sim = nb.Simulation(nb.example_random(n, fanout, 20, True), nets.standard_stdp(nb))
    if form == "run_kernel":
        sim.set_launch(64, 128)
    assert sim.step_kernel() == form
    sim.set_wait_limit(0)
    with pytest.raises(nb.NemoError) as e:
        if resident:
            for _ in range(10):
                sim.step([1])
        else:
            sim.run(300, 100, 1.0)
    assert e.value.code == NEMO_CUDA_ERROR
    assert "wait timed out" in str(e.value)
    del sim
    fresh_sim_is_bitexact()


@pytest.mark.parametrize("limit", [1 << 24, 0xffffffff])
@pytest.mark.parametrize("n,fanout", [(700, 60), (3000, 450)])
def test_long_limits_do_not_run_out(n, fanout, limit):
    a, b = (nb.Simulation(nb.example_random(n, fanout, 20, True), nets.standard_stdp(nb)) for _ in range(2))
    b.set_wait_limit(limit)
    ra, rb = a.run(300, 100, 1.0), b.run(300, 100, 1.0)
    assert ra[2].tolist() == rb[2].tolist()
    assert [list(a.step()) for _ in range(20)] == [list(b.step()) for _ in range(20)]
