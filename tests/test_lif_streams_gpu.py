"""The differentiable form where its one-launch kernels step aside or take
turns: under CUDA graph capture (its steps are then separate launches), on two
streams at once (its cooperative grids run one after another), and from two
threads whose calls need different amounts of shared memory."""

import threading

import numpy as np
import pytest
import torch

from nemo_b200.lif import LIFNetwork, lif_backward, lif_forward, poisson_bits

pytestmark = pytest.mark.gpu

# float32 sums of up to 1e4 terms: 2^-24 * sqrt(1e4) = 6e-6 relative, times 4
REL = 2.4e-5


def _problem(n, seed, steps=60, trials=7):
    net = LIFNetwork.random(n, 20, 30, 5, seed=seed, checkpoint=25)
    w = net.initial_weights(seed=seed, scale_rec=0.3, scale_in=1.0)
    bits, _ = poisson_bits(steps, 30, trials, rate_hz=90.0, seed=seed)
    d = torch.tensor(np.random.default_rng(seed).normal(size=(trials, steps // net.bin_steps)), device="cuda")
    return net, w, bits, trials, d.to(torch.float32)


def _pass(net, w, bits, trials, d):
    counts, saved = lif_forward(net, w, bits, trials)
    return counts, saved[0], lif_backward(net, w, bits, trials, saved, d)


def _same(got, want):
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert want[0].sum() > 0 and want[2].norm() > 0
    assert (got[2].double() - want[2].double()).norm() <= REL * want[2].double().norm()


@pytest.mark.parametrize("n", [31, 300, 2100])
def test_captured_pass_matches(n):
    args = _problem(n, seed=n)
    want = _pass(*args)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _pass(*args)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    _same(got, want)


def test_two_streams():
    problems = [_problem(n, seed=n) for n in (900, 2100)]
    want = [_pass(*p) for p in problems]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in problems]
    got = [[], []]
    for _ in range(4):
        for i, (s, p) in enumerate(zip(streams, problems)):
            with torch.cuda.stream(s):
                got[i].append(_pass(*p))
    torch.cuda.synchronize()
    for i in range(2):
        for g in got[i]:
            _same(g, want[i])


def test_two_threads_with_different_checkpoints():
    # a network whose backward steps launch by launch and takes no turn; the
    # segments' kernels use shared memory by the checkpoint interval (64 steps:
    # 66 KB; 2 steps: 3 KB)
    n, steps, trials = 40000, 64, 32
    rng = np.random.default_rng(3)
    tgt, pre = rng.integers(0, n, 3 * n), np.concatenate([rng.integers(0, n, 2 * n), n + rng.integers(0, 50, n)])
    bits, _ = poisson_bits(steps, 50, trials, rate_hz=100.0, seed=3)
    errors, grads = [], {}

    def work(checkpoint, calls):
        try:
            net = LIFNetwork(n, 50, tgt, pre, checkpoint=checkpoint, bin_steps=8)
            w = net.initial_weights(seed=3, scale_in=1.0)
            with torch.cuda.stream(torch.cuda.Stream()):
                d = torch.full((trials, steps // 8), 0.5, device="cuda")
                _, saved = lif_forward(net, w, bits, trials)
                for _ in range(calls):
                    g = lif_backward(net, w, bits, trials, saved, d)
                torch.cuda.current_stream().synchronize()
            grads[checkpoint] = g
        except Exception as e:   # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in ((64, 30), (2, 60))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    # the same terms, grouped by segment
    assert grads[2].norm() > 0
    assert (grads[64].double() - grads[2].double()).norm() <= REL * grads[2].double().norm()
