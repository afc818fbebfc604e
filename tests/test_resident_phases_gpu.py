"""Stepping through the resident launch, whose cycles are gathered while the
host has their firing: every way a stay can begin and end (idle, a run, an
applyStdp, a stimulus too long for a command, a state read), with and without
STDP, against the oracle: firing of every cycle, membrane potentials, weights."""

import os
import time

import numpy as np
import pytest

from nemo_b200 import netgen
from nemo_b200.nemo import Configuration, Library, Network, Simulation

pytestmark = pytest.mark.gpu

ORACLE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_build",
                      "libnemo_oracle.so")


# (neurons, synapses per neuron, largest delay, STDP): one block, few blocks,
# more blocks than SMs would hold; only delay-1 synapses
@pytest.mark.parametrize("n,m,dmax,stdp", [(20, 10, 3, True), (900, 80, 20, True), (5200, 60, 7, True),
                                           (5200, 60, 20, False), (700, 100, 1, True)])
def test_stays_match_the_oracle(n, m, dmax, stdp):
    spec = netgen.izhikevich_random(n, m, dmax=dmax, seed=n + m, stdp=stdp)
    sims = []
    for lib in (Library(), Library(ORACLE)):
        net = Network(lib)
        for p in spec.populations:
            net.add_neuron(net.add_neuron_type(p.type_name), p.idx, *p.args)
        ids = net.add_synapse(spec.source, spec.target, spec.delay, spec.weight, spec.plastic)
        conf = Configuration(lib)
        if stdp:
            pre, post = netgen.standard_stdp()
            conf.set_stdp_function(pre, post, 0.0, 1.0, 0.0, -1.0)
        if sims:
            conf.set_cpu_backend()
        sims.append(Simulation(net, conf))
    gpu, ref = sims
    rng = np.random.default_rng(n)

    def steps(count, fstim=0, istim=0):
        for _ in range(count):
            f = rng.choice(n, size=min(n, fstim), replace=False).astype(np.uint32)
            i = [(int(k), 12.5) for k in rng.choice(n, size=min(n, istim), replace=False)]
            assert np.array_equal(gpu.step(f, i), ref.step(f, i))

    for _ in range(3):
        steps(7, fstim=3)
        time.sleep(0.01)                       # the stay ends idle
        steps(1, fstim=1, istim=2)
        assert gpu.get_membrane_potential(n // 2) == ref.get_membrane_potential(n // 2)
        steps(2)
        assert gpu.run(5).tolist() == [len(ref.step()) for _ in range(5)]
        steps(9, fstim=2)
        if stdp:
            gpu.apply_stdp(1.0)
            ref.apply_stdp(1.0)
        steps(2, fstim=1)
        steps(2, fstim=40)                     # staged, a launch of its own
        steps(3, fstim=2)
        if stdp:
            gpu.apply_stdp(-0.5)
            ref.apply_stdp(-0.5)
    some = ids[::max(1, len(ids) // 3000)]
    assert np.array_equal(gpu.get_weights(some), np.array([ref.get_synapse_weight(k) for k in some], np.float32))
