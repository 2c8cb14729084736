"""The differentiable mode: the hand-written BPTT adjoint against PyTorch
autograd of the same unrolled dynamics in float64 (the FP64 oracle,
oracle/bptt_torch.py) and against finite differences of the smooth forward.

The relative error of a gradient vector is ||g - g64|| / ||g64||.  With
float64 state the adjoint must match the FP64 oracle to 1e-4.  With float32
state the gradient carries the rounding of a float32 evaluation, which the
spike upstroke amplifies (PyTorch's own float32 autograd of the same model
is off by about 1e-2 on these networks), so that mode must be no worse than
PyTorch float32 autograd on the same GPU."""
import numpy as np
import pytest
import torch

from nemosim_b200.bptt import DifferentiableNetwork
from oracle import bptt_torch as R

pytestmark = pytest.mark.gpu

TOL = 1e-4


def setup(neurons=256, fanout=24, ms=80, trials=4, readout=32, smooth=True, ckpt=20, seed=1,
          state_dtype=torch.float32):
    dev = torch.device("cuda", 0)
    net = DifferentiableNetwork.random(neurons, fanout, max_delay=10, seed=seed)
    teacher = DifferentiableNetwork.random(neurons, fanout, max_delay=10, seed=seed + 100)
    g = torch.Generator(device="cpu").manual_seed(seed)
    noise = (5.0 * torch.randn((ms, trials, neurons), generator=g)).to(dev)
    tmodel = teacher.model(trials, ms, readout, ckpt, smooth)
    Wt, at, bt = teacher.tensors(dev, requires_grad=False)
    target = tmodel.readout_trains(Wt, at, bt, noise)
    model = net.model(trials, ms, readout, ckpt, smooth, state_dtype=state_dtype)
    return dev, net, model, noise, target


def reference(net, dev, noise, target, readout, smooth, dtype=torch.float64):
    W, a, b = net.tensors(dev, dtype=dtype)
    c, d = net.constants(dev, dtype=dtype)
    st = R.Structure(net.source, net.target, net.delay, net.neurons, dev)
    loss = R.loss(W, a, b, c, d, noise.to(dtype), target.to(dtype), st, readout, smooth)
    loss.backward()
    return loss.detach(), W.grad, a.grad, b.grad


def relerr(x, ref):
    x = x.double()
    ref = ref.double()
    return float((x - ref).norm() / ref.norm().clamp_min(1e-300))


@pytest.mark.parametrize("smooth", [True, False])
def test_fp64_state_gradient_matches_fp64_autograd(smooth):
    dev, net, model, noise, target = setup(smooth=smooth, state_dtype=torch.float64)
    W, a, b = net.tensors(dev)
    loss = model.loss(W, a, b, noise, target)
    loss.backward()
    l64, gW, ga, gb = reference(net, dev, noise, target, 32, smooth)
    errs = [relerr(W.grad, gW), relerr(a.grad, ga), relerr(b.grad, gb)]
    print(f"smooth={smooth} fp64 state: loss {float(loss):.6g} vs {float(l64):.6g}; "
          f"rel. err. W {errs[0]:.2e} a {errs[1]:.2e} b {errs[2]:.2e}")
    assert abs(float(loss) - float(l64)) <= TOL * abs(float(l64))
    assert max(errs) <= TOL, errs


@pytest.mark.parametrize("smooth", [True, False])
def test_fp32_state_gradient_no_worse_than_fp32_autograd(smooth):
    dev, net, model, noise, target = setup(smooth=smooth)
    W, a, b = net.tensors(dev)
    loss = model.loss(W, a, b, noise, target)
    loss.backward()
    l64, gW, ga, gb = reference(net, dev, noise, target, 32, smooth)
    _, tW, ta, tb = reference(net, dev, noise, target, 32, smooth, dtype=torch.float32)
    ours = [relerr(W.grad, gW), relerr(a.grad, ga), relerr(b.grad, gb)]
    torch32 = [relerr(tW, gW), relerr(ta, ga), relerr(tb, gb)]
    print(f"smooth={smooth} fp32 state rel. err. {['%.2e' % e for e in ours]}, "
          f"torch fp32 autograd {['%.2e' % e for e in torch32]}")
    assert abs(float(loss) - float(l64)) <= TOL * abs(float(l64))
    for e, t in zip(ours, torch32):
        assert e <= max(TOL, 2.0 * t), (ours, torch32)


def test_gradient_matches_finite_differences():
    """Central differences of the smooth float64 forward along random
    directions agree with the adjoint's directional derivative (float64
    state).  a and b move every neuron at once, and the loss is smooth in
    them only on a scale of about 1e-6, hence the smaller step there."""
    dev, net, model, noise, target = setup(smooth=True, neurons=128, fanout=16, ms=60, state_dtype=torch.float64)
    W, a, b = net.tensors(dev)
    model.loss(W, a, b, noise, target).backward()
    c, d = net.constants(dev, dtype=torch.float64)
    st = R.Structure(net.source, net.target, net.delay, net.neurons, dev)
    W64, a64, b64 = (t.detach().double() for t in (W, a, b))
    n64, t64 = noise.double(), target.double()
    gen = torch.Generator(device="cpu").manual_seed(7)
    for name, base, grad, step in (("W", W64, W.grad, 1e-6), ("a", a64, a.grad, 1e-7), ("b", b64, b.grad, 1e-7)):
        direction = torch.randn(base.shape, generator=gen, dtype=torch.float64).to(dev)
        direction /= direction.norm()
        eps = step * max(1.0, float(base.abs().max()))
        args = {"W": W64, "a": a64, "b": b64}

        def f(x):
            kw = dict(args)
            kw[name] = x
            return float(R.loss(kw["W"], kw["a"], kw["b"], c, d, n64, t64, st, 32, True))
        fd = (f(base + eps * direction) - f(base - eps * direction)) / (2 * eps)
        ad = float((grad.double() * direction).sum())
        print(f"{name}: finite difference {fd:.8g}, adjoint {ad:.8g}")
        assert abs(fd - ad) <= 1e-3 * abs(fd) + 1e-12, (name, fd, ad)


@pytest.mark.parametrize("state_dtype", [torch.float32, torch.float64])
def test_checkpoint_interval_does_not_change_gradients(state_dtype):
    dev, net, model, noise, target = setup(smooth=True, ckpt=20, state_dtype=state_dtype)
    m2 = net.model(4, 80, 32, 7, True, state_dtype=state_dtype)
    W, a, b = net.tensors(dev)
    model.loss(W, a, b, noise, target).backward()
    W2, a2, b2 = net.tensors(dev)
    m2.loss(W2, a2, b2, noise, target).backward()
    assert torch.equal(W.grad, W2.grad) and torch.equal(a.grad, a2.grad) and torch.equal(b.grad, b2.grad)


def test_options_are_checked():
    from nemosim_b200 import NemoError, lib
    src = np.zeros(1, np.uint32)
    h = lib().nemo_b200_bptt_new(4, 1, 10, 1, 5, 1, src, src, np.ones(1, np.uint32), 4, 0)
    assert not h
    with pytest.raises(ValueError):
        DifferentiableNetwork.random(8, 2).model(1, 10, 1, state_dtype=torch.float16)
    assert NemoError is not None


def test_full_size_speed_vs_torch_autograd():
    """The differentiable configuration at full size (4096 neurons x 200
    synapses, 500 ms, 16 trials, 256 readouts, checkpoints every 50 ms): one
    gradient step of the adjoint, with float32 and with float64 state,
    against PyTorch float32 autograd of the same model on the same GPU."""
    import time
    dev, net, model, noise, target = setup(neurons=4096, fanout=200, ms=500, trials=16, readout=256,
                                           smooth=False, ckpt=50)
    times = {}
    for dtype in (torch.float32, torch.float64):
        m = net.model(16, 500, 256, 50, False, state_dtype=dtype)
        W, a, b = net.tensors(dev)
        for _ in range(2):
            W.grad = a.grad = b.grad = None
            m.loss(W, a, b, noise, target).backward()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(3):
            W.grad = a.grad = b.grad = None
            m.loss(W, a, b, noise, target).backward()
        torch.cuda.synchronize()
        times[dtype] = (time.perf_counter() - t0) / 3
        del m
    W32, a32, b32 = net.tensors(dev)
    c32, d32 = net.constants(dev)
    st = R.Structure(net.source, net.target, net.delay, net.neurons, dev)
    R.loss(W32, a32, b32, c32, d32, noise, target, st, 256, False).backward()  # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(2):
        W32.grad = a32.grad = b32.grad = None
        R.loss(W32, a32, b32, c32, d32, noise, target, st, 256, False).backward()
    torch.cuda.synchronize()
    theirs = (time.perf_counter() - t0) / 2
    ours32, ours64 = times[torch.float32], times[torch.float64]
    print(f"adjoint fp32 state {ours32 * 1e3:.1f} ms, fp64 state {ours64 * 1e3:.1f} ms, "
          f"torch autograd {theirs * 1e3:.1f} ms, speedup {theirs / ours32:.1f}x / {theirs / ours64:.1f}x")
    assert theirs / ours32 >= 10.0
    assert theirs / ours64 >= 10.0


def test_full_size_accuracy_vs_fp64_autograd():
    """The gradient error at full size (4096 x 200, 500 ms, 16 trials, 256
    readouts, hard threshold): the adjoint with float64 state within TOL of
    float64 autograd, and with float32 state no worse than twice PyTorch's
    own float32 autograd of the same model (both against float64)."""
    dev, net, _, noise, target = setup(neurons=4096, fanout=200, ms=500, trials=16, readout=256,
                                       smooth=False, ckpt=50)
    l64, gW, ga, gb = reference(net, dev, noise, target, 256, False)
    _, tW, ta, tb = reference(net, dev, noise, target, 256, False, dtype=torch.float32)
    torch32 = [relerr(tW, gW), relerr(ta, ga), relerr(tb, gb)]
    del tW, ta, tb
    errs = {}
    for dtype in (torch.float64, torch.float32):
        m = net.model(16, 500, 256, 50, False, state_dtype=dtype)
        W, a, b = net.tensors(dev)
        loss = m.loss(W, a, b, noise, target)
        loss.backward()
        errs[dtype] = (abs(float(loss) - float(l64)) / abs(float(l64)),
                       [relerr(W.grad, gW), relerr(a.grad, ga), relerr(b.grad, gb)])
        del m
    for dtype, (lerr, e) in errs.items():
        print(f"full size, {dtype} state: loss rel. err. {lerr:.2e}; gradient rel. err. W {e[0]:.2e} "
              f"a {e[1]:.2e} b {e[2]:.2e}")
    print(f"full size, torch float32 autograd: W {torch32[0]:.2e} a {torch32[1]:.2e} b {torch32[2]:.2e}")
    lerr64, e64 = errs[torch.float64]
    assert lerr64 <= TOL and max(e64) <= TOL, e64
    lerr32, e32 = errs[torch.float32]
    assert lerr32 <= TOL
    for e, t in zip(e32, torch32):
        assert e <= max(TOL, 2.0 * t), (e32, torch32)


# (neurons, fanout, ms, trials, readout, noise scale): a lane's 1 to 4 trials,
# groups of 16 (17, 33 trials), one neuron, fewer neurons than warps, more
# than a CTA's warps hold, lists and windows beyond shared memory, and noise
# so strong that neurons fire several times in a ms
LOOP_SHAPES = [(1, 1, 12, 1, 1, 1.0), (7, 3, 30, 2, 7, 1.0), (33, 9, 30, 3, 5, 1.0), (130, 17, 40, 5, 10, 1.0),
               (100, 40, 30, 8, 10, 1.0), (64, 64, 25, 13, 64, 1.0), (90, 20, 25, 17, 9, 1.0), (65, 33, 20, 33, 8, 1.0),
               (2100, 5, 15, 6, 40, 1.0), (40, 2500, 12, 4, 8, 1.0), (40, 30000, 12, 2, 8, 0.2), (60, 20, 20, 16, 10, 60.0),
               (60, 20, 20, 3, 10, 60.0)]


@pytest.mark.parametrize("state_dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("shape", LOOP_SHAPES)
def test_loops_match_autograd_at_their_edges(shape, state_dtype):
    """Loss and gradients of the hard threshold over the shapes of the
    forward and adjoint loops, with targets away from the trains (a loss that
    vanishes has no relative error).  float64 state: TOL.  float32 state: no
    worse than twice PyTorch's own float32 autograd, as above."""
    neurons, fanout, ms, trials, readout, scale = shape
    dev, net, model, noise, target = setup(neurons=neurons, fanout=fanout, ms=ms, trials=trials, readout=readout,
                                           smooth=False, ckpt=7, state_dtype=state_dtype)
    noise, target = noise * scale, target + 1.0
    W, a, b = net.tensors(dev)
    loss = model.loss(W, a, b, noise, target)
    loss.backward()
    l64, gW, ga, gb = reference(net, dev, noise, target, readout, False)
    ours = [relerr(loss.detach(), l64), relerr(W.grad, gW), relerr(a.grad, ga), relerr(b.grad, gb)]
    bound = [TOL] * 4
    if state_dtype == torch.float32:
        l32, tW, ta, tb = reference(net, dev, noise, target, readout, False, dtype=torch.float32)
        bound = [max(TOL, 2.0 * e) for e in (relerr(l32, l64), relerr(tW, gW), relerr(ta, ga), relerr(tb, gb))]
    assert all(e <= t for e, t in zip(ours, bound)), (ours, bound)


def test_a_weight_that_is_not_finite_reaches_its_target_without_a_spike():
    """inf x 0 is NaN: the target's state is NaN from the first delivery on
    (so it never fires and the loss stays finite), and so is the gradient of
    every weight into it, whether or not the source fired."""
    dev, net, model, noise, target = setup(neurons=40, fanout=8, ms=20, trials=4, readout=40, smooth=False,
                                           state_dtype=torch.float64)
    W, a, b = net.tensors(dev)
    with torch.no_grad():
        W[5] = float("inf")
    loss = model.loss(W, a, b, 0 * noise, target)  # no noise: nothing fires
    loss.backward()
    into = torch.as_tensor(net.target == net.target[5], device=dev)
    assert bool(torch.isfinite(loss)) and bool(torch.isnan(W.grad[into]).all())
    with torch.no_grad():
        W[5] = 0.1
    W.grad = None
    model.loss(W, a, b, noise, target).backward()  # the next pass is not affected
    assert bool(torch.isfinite(W.grad).all())


def test_loops_under_graph_capture():
    """Forward and backward captured in a CUDA graph and replayed on other
    inputs give the eager results."""
    dev, net, model, noise, target = setup(neurons=300, fanout=20, ms=30, trials=4, readout=20, smooth=False,
                                           state_dtype=torch.float64)
    W, a, b = net.tensors(dev, requires_grad=False)
    other = noise.flip(1).contiguous()
    want = (model.forward_raw(W, a, b, other, target),) + model.backward_raw(W, a, b, other, target)
    want = [x.clone() for x in want]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        model.forward_raw(W, a, b, noise, target)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = (model.forward_raw(W, a, b, noise, target),) + model.backward_raw(W, a, b, noise, target)
    for _ in range(2):
        noise.copy_(other)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
