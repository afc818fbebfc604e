"""The differentiable form over the sizes where its kernels change course:
checkpoint intervals above and below the 64-step parts of the event lists, a
last segment and a last part that are shorter, steps in which a unit spikes in
more than 32 (step, trial) pairs of a part, neurons without synapses, one to 32
trials, no recurrent synapse. The float64 reference differentiates the
kernel's own spike trains."""

import numpy as np
import pytest
import torch

import lif_reference as ref
from nemo_b200.lif import LIFNetwork, lif_bptt, lif_forward, poisson_bits, rate_loss, sinusoid_target

pytestmark = pytest.mark.gpu

BIN = 10

# (neurons, channels, recurrent synapses, input synapses, steps, trials,
# checkpoint, input rate in Hz)
SHAPES = [
    (3, 4, 0, 20, 60, 1, 60, 400.0),         # three neurons, no recurrent synapse
    (33, 5, 300, 60, 130, 3, 130, 100.0),    # one segment of three parts
    (100, 7, 1500, 300, 200, 32, 65, 900.0),  # parts of 33 and 32 steps; dense spikes: lists over 32 codes
    (257, 40, 4000, 2600, 90, 9, 64, 60.0),  # a full part, a short last segment
    (300, 0, 6000, 0, 60, 16, 7, 0.0),       # no input channels, nothing spikes
    (640, 33, 20000, 6000, 70, 31, 10, 80.0),
]


@pytest.mark.parametrize("shape", SHAPES)
def test_gradient_and_spikes_match_float64(shape):
    n, chans, n_rec, n_in, steps, trials, checkpoint, rate = shape
    rng = np.random.default_rng(sum(shape[:7]))
    # random targets: in-degrees differ, some neurons have no synapse
    tgt = rng.integers(0, n, n_rec + n_in)
    pre = np.concatenate([rng.integers(0, n, n_rec), n + rng.integers(0, max(chans, 1), n_in)])
    net = LIFNetwork(n, chans, tgt, pre, checkpoint=checkpoint, bin_steps=BIN)
    w = net.initial_weights(seed=1, scale_rec=0.35, scale_in=1.2)
    bits, ins = poisson_bits(steps, chans, trials, rate_hz=rate, seed=2)
    target = sinusoid_target(steps // BIN, BIN)
    wg = w.clone().requires_grad_(True)
    counts = lif_bptt(wg, bits, net, trials)
    rate_loss(counts, n, BIN, target).backward()
    _, saved = lif_forward(net, w, bits, trials)
    words = saved[0].cpu().numpy().view(np.uint32)
    assert trials == 32 or not np.any(words >> np.uint32(trials))
    spikes = np.stack([(words >> np.uint32(b)) & 1 for b in range(trials)], axis=2).astype(bool)
    assert rate == 0.0 or spikes.any()
    # the float64 potential along these trains crosses the threshold where
    # the kernel spikes, up to the rounding of a float32 sum
    w64 = torch.tensor(w.cpu().numpy().astype(np.float64), requires_grad=True)
    c64 = ref.counts(net, w64, ins, trials, spikes=spikes)
    assert np.array_equal(c64.detach().numpy(), counts.detach().cpu().numpy().astype(np.float64))
    pre_t, tgt_t = torch.as_tensor(net.pres), torch.as_tensor(net.targets)
    v = torch.zeros(n, trials, dtype=torch.float64)
    prev = torch.zeros(n, trials, dtype=torch.float64)
    for t in range(steps):
        x = torch.cat([prev, torch.as_tensor(ins[t].astype(np.float64))])[pre_t]
        u = net.beta * v + torch.zeros(n, trials, dtype=torch.float64).index_add(0, tgt_t, x * w64.detach()[:, None])
        s = torch.as_tensor(spikes[t].astype(np.float64))
        clear = (u - net.theta).abs() > 1e-4
        assert torch.equal((u >= net.theta)[clear], (s > 0)[clear]), t
        v, prev = u - net.theta * s, s
    rate_loss(c64, n, BIN, target.cpu().double()).backward()
    g, g64 = wg.grad.cpu().numpy().astype(np.float64), w64.grad.numpy()
    if rate == 0.0:
        assert not g.any() and not g64.any()
        return
    # float32 sums of up to 1e4 terms and an adjoint of up to 200 steps:
    # random-walk rounding of 2^-24 * sqrt(1e4) = 6e-6 relative, times 4
    assert np.linalg.norm(g - g64) <= 2.4e-5 * np.linalg.norm(g64)
