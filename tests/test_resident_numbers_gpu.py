"""Resident stepping when its command numbers run out: a library whose last
number is 40 (the product's is 2^31 - 2, ten hours of one loop), against the
oracle. A stay ends at the last number, with its cycle gathered, and the next
one starts at 1 again."""

import os
import subprocess

import numpy as np
import pytest

import nemo_b200.build as b
from nemo_b200 import netgen
from nemo_b200.nemo import Configuration, Library, Network, Simulation

pytestmark = pytest.mark.gpu

ORACLE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_build",
                      "libnemo_oracle.so")


@pytest.fixture(scope="module")
def numbers_lib(tmp_path_factory):
    b.build()
    path = tmp_path_factory.mktemp("numbers")
    objs = [os.path.join(b.BUILD, f) for f in sorted(os.listdir(b.BUILD))
            if f.endswith(".o") and f != "simulation.cpp.o"]
    obj, lib = str(path / "simulation.o"), str(path / "libnemo_b200_numbers.so")
    subprocess.check_call([b.CXX] + b.CXX_FLAGS + ["-DNEMO_B200_RESIDENT_LAST=40u", "-c",
                                                  os.path.join(b.CSRC, "simulation.cpp"), "-o", obj])
    subprocess.check_call([b.CXX, obj] + objs + b.LINK + ["-o", lib])
    lib = Library(lib)
    lib.add_plugin_path(os.path.join(b.HERE, "plugins"))
    return lib


@pytest.mark.parametrize("n,m,stdp", [(900, 80, True), (5200, 60, False)])
def test_numbers_start_again(numbers_lib, n, m, stdp):
    spec = netgen.izhikevich_random(n, m, dmax=12, seed=n, stdp=stdp)
    sims = []
    for lib in (numbers_lib, Library(ORACLE)):
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
    # long commands among short ones: every chunk of the mailbox is used again
    stim = [rng.choice(n, size=int(rng.choice([0, 1, 2, 25])), replace=False) for _ in range(200)]
    expected = [ref.step(f) for f in stim]
    for c, f in enumerate(stim):
        assert np.array_equal(gpu.step(f), expected[c]), c
    if stdp:
        gpu.apply_stdp(1.0)
        ref.apply_stdp(1.0)
    some = ids[::max(1, len(ids) // 2000)]
    assert np.array_equal(gpu.get_weights(some), np.array([ref.get_synapse_weight(k) for k in some], np.float32))
