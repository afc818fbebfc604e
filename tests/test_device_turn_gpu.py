"""Simulations and the differentiable form on one device at once, from several
threads: a stepping simulation (which stays on the device), one that runs many
cycles a call, gradient passes. Everything comes out as it does alone, and
nobody waits for another caller's loop to end."""

import threading
import time

import numpy as np
import pytest
import torch

from nemo_b200 import netgen
from nemo_b200.lif import LIFNetwork, lif_backward, lif_forward, poisson_bits
from nemo_b200.nemo import Configuration, Library, Network, Simulation

pytestmark = pytest.mark.gpu


def _simulation(n, seed):
    spec = netgen.izhikevich_random(n, 60, dmax=9, seed=seed, stdp=True)
    lib = Library()
    net = spec.build(Network(lib))
    conf = Configuration(lib)
    pre, post = netgen.standard_stdp()
    conf.set_stdp_function(pre, post, 0.0, 1.0, 0.0, -1.0)
    return Simulation(net, conf)


def _step(sim, n, count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for c in range(count):
        out.append(sim.step(rng.integers(0, n, 2)))
        if c % 100 == 99:
            sim.apply_stdp(1.0)
    return np.concatenate(out)


def _run(sim, count):
    return np.concatenate([sim.run(25) for _ in range(count)])


def _gradient(args):
    net, w, bits, trials, d = args
    counts, saved = lif_forward(net, w, bits, trials)
    return counts, lif_backward(net, w, bits, trials, saved, d)


def _problem(n):
    net = LIFNetwork.random(n, 20, 30, 5, seed=n, checkpoint=25)
    bits, _ = poisson_bits(60, 30, 7, rate_hz=90.0, seed=n)
    d = torch.tensor(np.random.default_rng(n).normal(size=(7, 6)), dtype=torch.float32, device="cuda")
    return net, net.initial_weights(seed=n, scale_rec=0.3, scale_in=1.0), bits, 7, d


def test_everything_at_once():
    problem = _problem(2100)
    alone = _step(_simulation(900, 1), 900, 600, 1), _step(_simulation(5200, 2), 5200, 300, 2), \
        _run(_simulation(5200, 3), 20), _gradient(problem)
    torch.cuda.synchronize()
    sims = _simulation(900, 1), _simulation(5200, 2), _simulation(5200, 3)
    got, errors = {}, []

    def gradients():
        with torch.cuda.stream(torch.cuda.Stream()):
            out = [_gradient(problem) for _ in range(40)]
            torch.cuda.current_stream().synchronize()
        return out

    def call(key, f, *args):
        try:
            got[key] = f(*args)
        except Exception as e:   # reported by the main thread
            errors.append((key, e))

    jobs = [(0, _step, sims[0], 900, 600, 1), (1, _step, sims[1], 5200, 300, 2), (2, _run, sims[2], 20), (3, gradients)]
    threads = [threading.Thread(target=call, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(3):
        assert len(alone[k]) > 0 and np.array_equal(got[k], alone[k]), k
    for counts, dw in got[3]:
        assert torch.equal(counts, alone[3][0]) and torch.equal(dw, alone[3][1])


def test_a_gradient_does_not_wait_for_a_stepping_loop():
    problem, sim = _problem(2100), _simulation(900, 4)
    _gradient(problem)
    torch.cuda.synchronize()
    stop = threading.Event()
    steps = [0]

    def loop():
        while not stop.is_set():
            sim.step()
            steps[0] += 1

    t = threading.Thread(target=loop)
    t.start()
    try:
        time.sleep(0.2)
        before, start = steps[0], time.monotonic()
        for _ in range(20):
            counts, dw = _gradient(problem)
            torch.cuda.synchronize()
        took, during = time.monotonic() - start, steps[0] - before
    finally:
        stop.set()
        t.join()
    # a pass takes about 1 ms alone; a wait gives up after 10 s
    assert took < 5.0 and torch.isfinite(dw).all() and counts.sum() > 0
    assert before > 0 and during > 0
