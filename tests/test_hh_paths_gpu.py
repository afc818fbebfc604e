"""The Hodgkin-Huxley update where it leaves its straight-line substep:
voltages at and around the rates' singular points (-55 and -40 mV, where a rate
is 0 / 0), exponents out of the fast range, neurons that are infinite or NaN
(beside ordinary ones of the same warp), a last warp that is not full. State
and firing bit for bit as the oracle, through single steps and through a
device-resident run."""

import os

import numpy as np
import pytest

from nemo_b200 import netgen
from nemo_b200.nemo import Configuration, Library, Network, Simulation

pytestmark = pytest.mark.gpu

ORACLE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_build",
                      "libnemo_oracle.so")


def _pair(n, seed, volts):
    rng = np.random.default_rng(seed)
    f32 = np.float32
    v = rng.uniform(-90.0, 50.0, n).astype(f32)
    v[: min(n, len(volts))] = np.array(volts[:n], f32)
    rng.shuffle(v)
    gates = [rng.uniform(0.0, 1.0, n).astype(f32) for _ in range(3)]
    pop = netgen.Population("HH", np.arange(n, dtype=np.uint32), [v] + gates + [np.zeros(n, f32)])
    sims = []
    for lib in (Library(), Library(ORACLE)):
        net = netgen.NetSpec([pop]).build(Network(lib))
        conf = Configuration(lib)
        if sims:
            conf.set_cpu_backend()
        sims.append(Simulation(net, conf))
    return sims


def _state(sim, n):
    a = np.array([[sim.get_neuron_state(i, k) for k in range(5)] for i in range(n)], np.float32)
    return np.where(np.isnan(a), np.uint32(0x7fc00000), a.view(np.uint32))


SINGULAR = [-55.0, -40.0, -65.0, -54.999996, -55.000004, -40.000004, -39.999996]
EXTREME = [1e4, -1e4, 760.0, -860.0, 3e38, float("inf"), float("-inf"), float("nan"), float("nan"), 1e-30]


@pytest.mark.parametrize("n,volts", [(1, SINGULAR), (7, SINGULAR), (37, SINGULAR + EXTREME), (130, EXTREME)])
def test_state_and_firing_match_the_oracle(n, volts):
    gpu, ref = _pair(n, n, volts)
    rng = np.random.default_rng(n)
    for c in range(14):
        # the currents are conductances here; some large
        istim = [(int(i), float(rng.choice([0.0, 3.0, 20.0, 4000.0]))) for i in rng.integers(0, n, 1 + n // 8)]
        istim = list(dict(istim).items())
        assert np.array_equal(gpu.step([], istim), ref.step([], istim)), c
    assert np.array_equal(_state(gpu, n), _state(ref, n))
    fired = gpu.run(4)
    assert fired.tolist() == [len(ref.step()) for _ in range(4)]
    assert np.array_equal(_state(gpu, n), _state(ref, n))
