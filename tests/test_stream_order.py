"""Device memory is filled in the order that its readers rely on.

A simulation's stream does not wait for the legacy default stream, so a plain
cudaMemcpy into memory that the stream has zeroed (or that its kernels read
next) is ordered against neither: an upload can be overwritten by the zeros
that were queued before it.  Uploads therefore go through the stream.  The
first tests look for the unordered calls in the native sources (CPU); the
others construct small simulations many times over, whose tables of ids
would come out as zeros (GPU)."""
import os
import re

import numpy as np
import pytest

import nemosim_b200 as nb
from tests import nets

CSRC = os.path.join(os.path.dirname(os.path.abspath(nb.__file__)), "csrc")


def calls(source, name):
    text = open(os.path.join(CSRC, source)).read()
    return [" ".join(m.split()) for m in re.findall(r"\b%s\s*\([^;]*;" % name, text)]


@pytest.mark.parametrize("source", ["simulation.cu", "construction.cu", "bptt.cu"])
def test_no_upload_beside_the_stream(source):
    assert calls(source, "cudaMemcpyAsync")
    assert [c for c in calls(source, "cudaMemcpy") if "HostToDevice" in c] == []


@pytest.mark.parametrize("source", ["simulation.cu", "construction.cu", "bptt.cu"])
def test_no_zeros_beside_the_stream(source):
    """The barrier of the step loops is cleared after a wait gave up, and the
    next launch counts its arrivals in it; the differentiable loops count from
    the zeros of a new model, on whatever stream they are called."""
    assert calls(source, "cudaMemset") == []


@pytest.mark.gpu
def test_id_tables_of_fresh_simulations():
    """1000 fresh rings with scattered ids: a table of zeros answers 0 for
    every fired neuron."""
    n, n0, nstep = 1000, 1_000_000, 4
    for k in range(1000):
        sim = nb.Simulation(nets.create_ring(nb, nb.Network(), n, n0, False, nstep), nb.Configuration())
        got = [list(sim.step([n0 + nstep * 7]))] + [list(sim.step()) for _ in range(3)]
        want = [[n0 + nstep * (7 + i)] for i in range(4)]
        assert got == want, (k, got, want)


@pytest.mark.gpu
def test_stream_order_of_fresh_batches():
    """200 fresh batches whose networks are not contiguous in the union
    (each has neurons of two types): ids and per-network counts."""
    sizes = [7, 40, 33]

    def network(n):
        net = nb.Network()
        t, i = net.add_neuron_type("PoissonSource"), net.add_neuron_type("Input")
        ids = np.arange(10, 10 + 2 * n, dtype=np.uint32)
        net.add_neuron(t, ids[:n], np.float32(1.0))
        net.add_neuron(i, ids[n:])
        net.add_synapse(ids[:n], ids[n:], np.ones(n, np.uint32), np.ones(n, np.float32), np.zeros(n, np.uint8))
        return net

    counts0 = np.array([sizes] * 3)
    ids0 = np.concatenate([np.arange(10, 10 + n) for n in sizes] * 3)
    for k in range(200):
        batch = nb.Batch([network(n) for n in sizes], nb.Configuration())
        counts, _, ids = batch.run(3)
        assert counts.tolist() == counts0.tolist(), k
        assert ids.tolist() == ids0.tolist(), k


@pytest.mark.gpu
def test_first_pass_of_a_fresh_model_on_a_side_stream():
    """100 fresh differentiable models, each called at once on a stream that
    does not wait for the legacy one."""
    import torch
    from nemosim_b200.bptt import DifferentiableNetwork
    net = DifferentiableNetwork.random(200, 20, seed=2)
    gen = torch.Generator(device="cuda").manual_seed(1)
    noise = 6.0 * torch.randn((40, 4, 200), generator=gen, device="cuda")
    target = torch.zeros((40, 4, 32), device="cuda")
    W, a, b = net.tensors("cuda")
    torch.cuda.synchronize()
    side, want = torch.cuda.Stream(), None
    for k in range(100):
        with torch.cuda.stream(side):
            model = net.model(trials=4, ms=40, readout=32, checkpoint_ms=20)
            loss = model.loss(W, a, b, noise, target)
            got = [loss.detach(), *torch.autograd.grad(loss, (W, a, b))]
            side.synchronize()
        want = want or got
        assert all(torch.equal(x, y) for x, y in zip(got, want)), k
    assert float(want[0]) > 0 and float(want[1].abs().max()) > 0
