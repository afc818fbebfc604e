"""The differentiable form past its kernels' shared memory, and at the sizes
where a direction goes back to a launch per step: against the captured pass,
which runs launch by launch and keeps nothing in shared memory. Spikes and
counts are equal; gradients to rounding."""

import numpy as np
import pytest
import torch

from nemo_b200.lif import LIFNetwork, lif_backward, lif_forward, poisson_bits

pytestmark = pytest.mark.gpu


def _net(n, chans, n_rec, n_in, checkpoint, seed):
    """Random synapses: in- and out-degrees differ, a pair may have several."""
    rng = np.random.default_rng(seed)
    tgt = rng.integers(0, n, n_rec + n_in)
    pre = np.concatenate([rng.integers(0, n, n_rec), n + rng.integers(0, chans, n_in)])
    return LIFNetwork(n, chans, tgt, pre, checkpoint=checkpoint)


def _problem(net, steps, trials, seed):
    w = net.initial_weights(seed=seed, scale_in=1.0)
    bits, _ = poisson_bits(steps, net.n_in, trials, rate_hz=150.0, seed=seed)
    d = np.random.default_rng(seed).normal(size=(trials, steps // net.bin_steps))
    return net, w, bits, trials, torch.tensor(d, dtype=torch.float32, device="cuda")


def _pass(net, w, bits, trials, d):
    counts, saved = lif_forward(net, w, bits, trials)
    return counts, saved[0], lif_backward(net, w, bits, trials, saved, d)


def _captured(args):
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _pass(*args)
    graph.replay()
    torch.cuda.synchronize()
    return out


def _check(args, passes=1):
    net, _, bits, _, _ = args
    want = _captured(args)
    assert want[0].sum() > 0 and torch.isfinite(want[2]).all() and want[2].norm() > 0
    # a weight's gradient sums gu over its spikes, gu sums a source's synapses
    # each step: float32 sums of up to fan-out x steps terms on both sides,
    # random-walk rounding of 2^-24 sqrt(terms) relative, times 4
    fan = net._post.numel() / net.n
    rel = 4 * 2.0 ** -24 * np.sqrt(max(fan, 1.0) * bits.shape[0])
    for _ in range(passes):
        got = _pass(*args)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        assert (got[2].double() - want[2].double()).norm() <= rel * want[2].double().norm()


@pytest.fixture(scope="module")
def dense():
    return _net(600, 20, 2_400_000, 6_000, checkpoint=20, seed=5)


@pytest.mark.parametrize("trials", [5, 13, 27])
def test_entries_through_the_ring(dense, trials):
    # 4,000 synapses a neuron: a block's share of 60 sources is 240 KB, more
    # than a block has, at rows of 8, 16 and 32 trials; several passes, as the
    # ring is used anew every step
    _check(_problem(dense, 40, trials, seed=trials), passes=4)


@pytest.mark.parametrize("n,n_rec,trials", [
    (5000, 4_100_000, 9),    # 27,900 synapses a block, more than its room; two neurons a warp
    (11000, 33_000, 32),     # nine parts of 32-trial rows (from 10,233 neurons on)
    (20000, 60_000, 32),     # sixteen parts; more rows to finish than a block has threads
    (37091, 80_000, 32),     # the largest network of 32 trials in one launch
    (37092, 80_000, 32),     # the backward step by step
    (48000, 90_000, 8),      # the forward step by step, the backward in 12 parts of 8-trial rows
    (65600, 90_000, 5),      # both step by step
])
def test_sizes_at_the_limits(n, n_rec, trials):
    net = _net(n, 20, n_rec, n, checkpoint=15, seed=n)
    _check(_problem(net, 40, trials, seed=trials))
