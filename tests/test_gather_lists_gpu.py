"""The gather's block-to-block lists and unit sizes: networks whose synapses
stay near their source (a block is reached by few others, some blocks by none)
and networks of large buckets (units of fewer than 32 sources), against the
oracle: every cycle's firing, and the weights after learning."""

import os

import numpy as np
import pytest

from nemo_b200 import netgen
from nemo_b200.nemo import Configuration, Library, Network, Simulation

pytestmark = pytest.mark.gpu

ORACLE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_build",
                      "libnemo_oracle.so")


def _spec(n, m, reach, dmax, seed):
    """m synapses per neuron to targets at most `reach` indices away (0: any);
    the last third of the neurons has none."""
    spec = netgen.izhikevich_random(n, 0, seed=seed)
    rng = np.random.default_rng(seed)
    senders = n - n // 3
    src = np.repeat(np.arange(senders, dtype=np.uint32), m)
    if reach:
        tgt = (src + rng.integers(-reach, reach + 1, src.size)) % senders
    else:
        tgt = rng.integers(0, n, src.size)
    spec.source, spec.target = src, tgt.astype(np.uint32)
    spec.delay = rng.integers(1, dmax + 1, src.size).astype(np.uint32)
    inh = src >= int(senders * 0.8)
    spec.weight = np.where(inh, -rng.random(src.size), 0.5 * rng.random(src.size)).astype(np.float32) * np.float32(100.0 / m)
    spec.plastic = (~inh).astype(np.uint8)
    return spec


# (neurons, synapses per neuron, reach, largest delay): units of 32 sources
# with few lists; of 16, 8 and 4 sources; one block
@pytest.mark.parametrize("shape", [(9000, 40, 150, 9), (4800, 400, 60, 3), (640, 500, 0, 12), (2000, 1500, 0, 5),
                                   (70, 3000, 0, 20), (33, 900, 0, 2)])
def test_firing_and_weights_match_the_oracle(shape):
    n, m, reach, dmax = shape
    spec = _spec(n, m, reach, dmax, seed=sum(shape))
    pre, post = netgen.standard_stdp()
    sims = []
    for lib in (Library(), Library(ORACLE)):
        net = Network(lib)
        for p in spec.populations:
            net.add_neuron(net.add_neuron_type(p.type_name), p.idx, *p.args)
        ids = net.add_synapse(spec.source, spec.target, spec.delay, spec.weight, spec.plastic)
        conf = Configuration(lib)
        conf.set_stdp_function(pre, post, 0.0, 4.0, 0.0, -4.0)
        if len(sims):
            conf.set_cpu_backend()
        sims.append(Simulation(net, conf))
    gpu, ref = sims
    fired = 0
    for base in (0, 30, 60):
        first = gpu.run(30)
        expected = [ref.step() for _ in range(30)]
        assert first.tolist() == [len(f) for f in expected]
        fired += int(first.sum())
        for c, f in enumerate(expected):
            assert np.array_equal(gpu.fired_at(base + c), f), (base + c)
        gpu.apply_stdp(1.0)
        ref.apply_stdp(1.0)
    assert fired > 0
    some = ids[::max(1, len(ids) // 2000)]
    assert np.array_equal(gpu.get_weights(some), np.array([ref.get_synapse_weight(i) for i in some], np.float32))
