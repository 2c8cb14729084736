"""The differentiable mode where neurons fire several times in a millisecond:
inputs come from spike counts, 32 synapses at a time."""
import pytest
import torch

from tests.test_bptt_gpu import TOL, reference, relerr, setup

pytestmark = pytest.mark.gpu


# in-degrees around 32 and 64 and of 100 and 2500, one to 20 trials (every split of a list's four sums over lanes), more
# neurons than a CTA's warps hold
@pytest.mark.parametrize("neurons,fanout,ms,trials,readout", [
    (70, 31, 20, 4, 10), (70, 33, 20, 1, 10), (90, 64, 20, 20, 10), (500, 100, 15, 7, 40), (40, 2500, 12, 4, 8),
    (6000, 20, 12, 1, 60), (76_000, 5, 10, 1, 60), (4800, 13, 12, 16, 60)])
def test_counts_match_autograd(neurons, fanout, ms, trials, readout):
    dev, net, model, noise, target = setup(neurons=neurons, fanout=fanout, ms=ms, trials=trials, readout=readout,
                                           smooth=False, ckpt=7, state_dtype=torch.float64)
    noise, target = noise * 60.0, target + 1.0
    W, a, b = net.tensors(dev)
    loss = model.loss(W, a, b, noise, target)
    loss.backward()
    l64, gW, ga, gb = reference(net, dev, noise, target, readout, False)
    ours = [relerr(loss.detach(), l64), relerr(W.grad, gW), relerr(a.grad, ga), relerr(b.grad, gb)]
    assert all(e <= TOL for e in ours), ours
