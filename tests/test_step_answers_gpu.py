"""The answers of nemo_step's resident loops: every fired neuron of a step
comes back, in order, whatever their number -- up to 32 words of neurons
(answered by one warp) and beyond, up to 4096 ids (word by word) and beyond
(in a buffer of their own)."""
import os
import re

import numpy as np
import pytest

import nemosim_b200 as nb

CSRC = os.path.join(os.path.dirname(os.path.abspath(nb.__file__)), "csrc")


def test_polled_words_are_written_whole():
    """The host takes each word of an answer as it appears, while the kernel
    runs: no ordinary store writes one."""
    text = open(os.path.join(CSRC, "simulation.cu")).read()
    assert re.findall(r"ctl->(?:reply|ids)\[[^;=]*\]\s*=[^=]", text) == []
    assert len(re.findall(r"st_relaxed_sys_u64\(&ctl->(?:reply|ids)\[", text)) >= 6


@pytest.mark.gpu
@pytest.mark.parametrize("persistent_shape", [False, True])
@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 5000])
def test_every_fired_neuron_is_answered(n, persistent_shape):
    net = nb.Network()
    rng = np.random.default_rng(n)
    ids = (rng.permutation(n) * 3 + 7).astype(np.uint32)
    net.add_neuron(net.add_neuron_type("Input"), ids)
    sim = nb.Simulation(net, nb.Configuration())
    if persistent_shape:
        sim.set_launch(64, 128)  # the persistent loop
    for count in (0, 1, n // 2, 4095, 4096, 4097, n, 2, n, 0):
        if count > n:
            continue
        chosen = np.sort(rng.choice(n, count, replace=False))
        assert list(sim.step(ids[chosen].tolist())) == ids[chosen].tolist(), count
