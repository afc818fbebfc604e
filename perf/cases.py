"""The work that users of the library have it do, as cases that can be timed
and whose outputs can be compared.

Spiking simulation (``nemo_b200.nemo``), Izhikevich networks as the random
benchmark network of ``netgen`` (80% excitatory, thalamic noise, uniform
targets and delays):

* ``step``  -- a closed loop: ``Simulation.step`` every millisecond with a
  firing stimulus in and the fired neurons out, ``apply_stdp`` at the end of
  the pass where the network learns;
* ``run``   -- device-resident: ``Simulation.run`` of many cycles, then
  ``apply_stdp`` and (small networks) the learned weights read back;
* ``mixed`` -- a closed loop over Izhikevich, IF_curr_exp, QIF and HH
  populations, every neuron stimulated at random each cycle;
* ``batch`` -- many independent networks advanced together
  (``nemo_b200_new_batch``, ``nemo_b200_run_graph``).

Differentiable form (``nemo_b200.lif``):

* ``lif``   -- spike counts of a recurrent LIF network, and with ``grad`` the
  gradient of a rate loss with respect to every synapse's weight.

Simulation results are whole numbers and fixed-point weights, equal bit for
bit in every correct implementation; the differentiable form computes in
float32.
"""

import ctypes
import math

import numpy as np
import torch

from nemo_b200 import netgen
from nemo_b200.lif import LIFNetwork, lif_bptt, lif_forward, rate_loss, sinusoid_target
from nemo_b200.nemo import Configuration, Library, Network, Simulation

KAPPA = 10.0
TAU_M = 20.0
BIN = 10


def listed():
    return [
        # the 1000-neuron example network in a closed loop: the smallest call, latency counts
        dict(name="step-1k", kind="step", n=1000, m=100, dmax=20, stdp=False, stim=1, cycles=50),
        # a learning network in a closed loop
        dict(name="step-20k-stdp", kind="step", n=20000, m=1000, dmax=20, stdp=True, stim=1, cycles=100),
        # the example network learning on the device, its weights read after every update
        dict(name="run-1k-weights", kind="run", n=1000, m=100, dmax=20, stdp=True, weights=True, cycles=100),
        # an ordinary static network of an odd size, run on the device
        dict(name="run-30k", kind="run", n=30011, m=300, dmax=15, stdp=False, weights=False, cycles=100),
        # the benchmark: 1e8 synapses with STDP, an update every 100 ms
        dict(name="run-100k-stdp", kind="run", n=100000, m=1000, dmax=20, stdp=True, weights=False, cycles=100),
        # mixed neuron models under a random stimulus (the Hodgkin-Huxley update is most of a cycle)
        dict(name="mixed-50k", kind="mixed", iz=20000, lif=15000, qif=10000, hh=5000, m=500, dmax=10, p=0.005,
             cycles=20),
        # a parameter sweep: independent networks of 500 to 20000 neurons in one simulation
        dict(name="batch-64", kind="batch", count=64, lo=500, hi=20000, m=100, dmax=20, cycles=100),
        # a gradient step of a toy network: launches count
        dict(name="lif-300", kind="lif", grad=True, n=300, fan=30, chans=40, infan=10, ragged=False, steps=120,
             trials=8, rate=60.0, checkpoint=25),
        # an ordinary gradient step
        dict(name="lif-2k", kind="lif", grad=True, n=2000, fan=200, chans=500, infan=50, ragged=False, steps=100,
             trials=32, rate=10.0, checkpoint=50),
        # the benchmark's gradient step
        dict(name="lif-10k", kind="lif", grad=True, n=10000, fan=200, chans=500, infan=50, ragged=False, steps=500,
             trials=32, rate=10.0, checkpoint=50),
        # evaluation of a trained network: forward only, odd sizes, in-degrees that differ
        dict(name="lif-eval-3k", kind="lif", grad=False, n=3001, fan=120, chans=77, infan=30, ragged=True, steps=250,
             trials=17, rate=20.0, checkpoint=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "mixed", "batch", "lif", "lif", "lif"])
    if kind == "step":
        n = _log(rng, 200, 20000)
        return dict(kind=kind, n=n, m=_log(rng, 20, min(n, 1000)), dmax=rng.randint(2, 24), stdp=rng.random() < 0.5,
                    stim=rng.choice([0, 1, 5, 40]), cycles=rng.randint(30, 100))
    if kind == "run":
        n = _log(rng, 500, 60000)
        m = _log(rng, 30, min(n, 600))
        stdp = rng.random() < 0.6
        return dict(kind=kind, n=n, m=m, dmax=rng.randint(2, 24), stdp=stdp, weights=stdp and n * m <= 200000,
                    cycles=rng.randint(50, 200))
    if kind == "mixed":
        return dict(kind=kind, iz=_log(rng, 500, 20000), lif=_log(rng, 300, 15000), qif=_log(rng, 200, 10000),
                    hh=_log(rng, 50, 5000), m=_log(rng, 20, 300), dmax=rng.randint(2, 12), p=0.005,
                    cycles=rng.randint(10, 20))
    if kind == "batch":
        lo = _log(rng, 200, 2000)
        return dict(kind=kind, count=rng.randint(8, 64), lo=lo, hi=_log(rng, lo + 1, 15000), m=_log(rng, 30, 100),
                    dmax=rng.randint(2, 24), cycles=rng.randint(50, 100))
    n = _log(rng, 100, 8000)
    steps = BIN * rng.randint(5, 40)
    return dict(kind=kind, grad=rng.random() < 0.75, n=n, fan=_log(rng, 10, min(n - 1, 250)),
                chans=_log(rng, 20, 600), infan=rng.randint(5, 20) if rng.random() < 0.5 else 20,
                ragged=rng.random() < 0.5, steps=steps, trials=rng.choice([1, 5, 8, 16, 31, 32, 32]),
                rate=rng.choice([10.0, 20.0, 60.0]), checkpoint=rng.choice([10, 25, 33, 50, 100]))


# ---- spiking simulation ----

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _random_synapses(spec, n, m, dmax, n_exc_end, n_inh, stdp, w_exc, w_inh, seed):
    """m synapses per neuron to uniform targets, delays U{1..dmax}; neurons
    [n_exc_end, n_exc_end + n_inh) are inhibitory."""
    g = _generator(seed)
    total = n * m
    src = torch.arange(n, device="cuda", dtype=torch.int32).repeat_interleave(m)
    tgt = torch.randint(0, n, (total,), generator=g, device="cuda", dtype=torch.int32)
    dly = torch.randint(1, dmax + 1, (total,), generator=g, device="cuda", dtype=torch.int32)
    w = torch.rand(total, generator=g, device="cuda")
    inh = (src >= n_exc_end) & (src < n_exc_end + n_inh)
    w = torch.where(inh, -w_inh * w, w_exc * w)
    spec.source = src.cpu().numpy().view(np.uint32)
    spec.target = tgt.cpu().numpy().view(np.uint32)
    spec.delay = dly.cpu().numpy().view(np.uint32)
    spec.weight = w.cpu().numpy()
    spec.plastic = (~inh).to(torch.uint8).cpu().numpy() if stdp else np.zeros(total, np.uint8)
    return spec


def _izhikevich(n, m, dmax, stdp, seed, **kw):
    spec = netgen.izhikevich_random(n, 0, seed=seed, **kw)
    n_exc = int(n * 0.8)
    return _random_synapses(spec, n, m, dmax, n_exc, n - n_exc, stdp, 0.5, 1.0, seed)


def _simulation(spec, stdp, write_only):
    net = Network(Library())
    for p in spec.populations:
        net.add_neuron(net.add_neuron_type(p.type_name), p.idx, *p.args)
    ids = net.add_synapse(spec.source, spec.target, spec.delay, spec.weight, spec.plastic)
    conf = Configuration(net.lib)
    if stdp:
        pre, post = netgen.standard_stdp()
        conf.set_stdp_function(pre, post, 0.0, 1.0, 0.0, -1.0)
    if write_only:
        conf.set_write_only_synapses()
    return Simulation(net, conf), ids


def _prepare_batch(case, seed):
    lib = Library()
    d = lib.dll
    d.nemo_b200_new_batch.restype = ctypes.c_void_p
    d.nemo_b200_new_batch.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t, ctypes.c_void_p]
    d.nemo_b200_run_graph.argtypes = [ctypes.c_void_p, ctypes.c_uint, ctypes.c_uint, ctypes.POINTER(ctypes.c_int)]
    d.nemo_b200_cycle.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint64)]
    d.nemo_b200_batch_fired_at.argtypes = [ctypes.c_void_p, ctypes.c_uint64,
                                           ctypes.POINTER(ctypes.POINTER(ctypes.c_uint)),
                                           ctypes.POINTER(ctypes.POINTER(ctypes.c_size_t))]
    sizes = netgen.batched_sizes(case["count"], case["lo"], case["hi"], seed=3)
    sig = np.random.default_rng(4).uniform(3.0, 7.0, size=case["count"])
    nets = []
    for j, n in enumerate(sizes):
        spec = _izhikevich(int(n), min(case["m"], int(n)), case["dmax"], False, 1000 * seed + j,
                           sigma_exc=float(sig[j]), sigma_inh=float(0.4 * sig[j]))
        nets.append(spec.build(Network(lib)))
    conf = Configuration(lib)
    handles = (ctypes.c_void_p * len(nets))(*[x.handle for x in nets])
    conf.set_write_only_synapses()
    batch = d.nemo_b200_new_batch(handles, len(nets), conf.handle)
    if not batch:
        raise RuntimeError(d.nemo_strerror().decode())
    # owned by a Simulation object, which deletes the handle with itself
    sim = Simulation.__new__(Simulation)
    sim.lib, sim.handle = lib, batch
    return sim


def _neurons(case):
    if case["kind"] == "mixed":
        return case["iz"] + case["lif"] + case["qif"] + case["hh"]
    if case["kind"] == "batch":
        return int(netgen.batched_sizes(case["count"], case["lo"], case["hi"], seed=3).sum())
    return case["n"]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("step", "run"):
        spec = _izhikevich(case["n"], case["m"], case["dmax"], case["stdp"], seed)
        weights = kind == "run" and case["weights"]
        state["sim"], ids = _simulation(spec, case["stdp"], not weights)
        if weights:
            state["ids"] = ids
        state["raster"] = np.zeros((case["cycles"] if kind == "step" else 1, case["n"]), np.uint8)
        state["done"] = 0
        if kind == "step":
            rng = np.random.default_rng(seed + 1)
            state["stim"] = [rng.choice(case["n"], size=case["stim"], replace=False).astype(np.uint32)
                             for _ in range(case["cycles"])]
    elif kind == "mixed":
        n = _neurons(case)
        spec = netgen.mixed_plugins(case["iz"], case["lif"], case["qif"], case["hh"], m=0, dmax=case["dmax"], seed=seed)
        n_exc = int(case["iz"] * 0.8)
        _random_synapses(spec, n, case["m"], case["dmax"], n_exc, case["iz"] - n_exc, False, 0.3, 0.6, seed)
        state["sim"], _ = _simulation(spec, False, True)
        state["raster"] = np.zeros((case["cycles"], n), np.uint8)
        rng = np.random.default_rng(seed + 1)
        state["stim"] = [np.nonzero(rng.random(n) < case["p"])[0].astype(np.uint32) for _ in range(case["cycles"])]
    elif kind == "batch":
        state["sim"] = _prepare_batch(case, seed)
        sizes = netgen.batched_sizes(case["count"], case["lo"], case["hi"], seed=3)
        state["base"] = np.cumsum(sizes) - sizes
        state["raster"] = np.zeros((2, sizes.sum()), np.uint8)
    else:
        targets, pres, w, bits = _lif_inputs(case, seed)
        net = LIFNetwork(case["n"], case["chans"], targets, pres, tau_m=TAU_M, kappa=KAPPA,
                         checkpoint=case["checkpoint"], bin_steps=BIN)
        state["net"], state["bits"] = net, bits
        state["w"] = w.clone().requires_grad_(case["grad"])
        state["target"] = sinusoid_target(case["steps"] // BIN, BIN)
    return state


def _run_batch(state):
    sim, cycles = state["sim"], state["case"]["cycles"]
    lib, h = sim.lib, sim.handle
    lib.call("nemo_b200_run_graph", h, cycles, cycles, None)
    now = ctypes.c_uint64()
    lib.call("nemo_b200_cycle", h, ctypes.byref(now))
    fired = ctypes.POINTER(ctypes.c_uint)()
    offsets = ctypes.POINTER(ctypes.c_size_t)()
    # the last two cycles' firing of every instance
    raster = state["raster"]
    raster.fill(0)
    for k in (1, 2):
        lib.call("nemo_b200_batch_fired_at", h, now.value - k, ctypes.byref(fired), ctypes.byref(offsets))
        off = np.ctypeslib.as_array(offsets, shape=(state["case"]["count"] + 1,)).astype(np.int64)
        if off[-1]:
            own = np.ctypeslib.as_array(fired, shape=(int(off[-1]),))
            raster[k - 1, own + np.repeat(state["base"], np.diff(off))] = 1
    return {"fired": raster}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "mixed"):
        sim = state["sim"]
        fired = [sim.step(f) for f in state["stim"]]
        if case.get("stdp"):
            sim.apply_stdp(1.0)
        raster = state["raster"]
        raster.fill(0)
        for c, f in enumerate(fired):
            raster[c, f] = 1
        return {"fired": raster}
    if kind == "run":
        sim = state["sim"]
        out = {"count": sim.run(case["cycles"]).astype(np.int64), "fired": state["raster"]}
        state["done"] += case["cycles"]
        state["raster"].fill(0)
        state["raster"][0, sim.fired_at(state["done"] - 1)] = 1
        if case["stdp"]:
            sim.apply_stdp(1.0)
        if case["weights"]:
            out["weights"] = sim.get_weights(state["ids"])
        return out
    if kind == "batch":
        return _run_batch(state)
    if not case["grad"]:
        counts, saved = lif_forward(state["net"], state["w"], state["bits"], case["trials"])
        return {"counts": counts, "spikes": saved[0]}
    w = state["w"]
    w.grad = None
    counts = lif_bptt(w, state["bits"], state["net"], case["trials"])
    rate_loss(counts, case["n"], BIN, state["target"]).backward()
    return {"counts": counts.detach(), "grad": w.grad}


# ---- differentiable form: inputs and the 64-bit result ----

def _lif_inputs(case, seed):
    """Synapses by target (recurrent ones first), weights in that order, input
    spikes as words [steps][chans] (bit b: trial b). ``ragged``: a synapse's
    target is uniform, so that in-degrees differ (0 among them)."""
    n, fan, chans, infan = case["n"], case["fan"], case["chans"], case["infan"]
    g = _generator(seed)
    dev = "cuda"
    if case["ragged"]:
        t_rec = torch.randint(0, n, (n * fan,), generator=g, device=dev).sort().values
        t_in = torch.randint(0, n, (n * infan,), generator=g, device=dev).sort().values
    else:
        t_rec = torch.arange(n, device=dev).repeat_interleave(fan)
        t_in = torch.arange(n, device=dev).repeat_interleave(infan)
    p_rec = torch.randint(0, n - 1, t_rec.shape, generator=g, device=dev)
    p_rec = p_rec + (p_rec >= t_rec)   # not the target itself
    p_in = n + torch.randint(0, chans, t_in.shape, generator=g, device=dev)
    w_rec = torch.randn(t_rec.shape, generator=g, device=dev) / math.sqrt(fan)
    # an input drive of standard deviation 0.25 per step
    w_in = torch.randn(t_in.shape, generator=g, device=dev) * (0.25 / math.sqrt(infan * case["rate"] / 1000.0))
    targets, pres, w = torch.cat([t_rec, t_in]), torch.cat([p_rec, p_in]), torch.cat([w_rec, w_in])
    order = torch.argsort(targets, stable=True)
    targets, pres, w = targets[order], pres[order], w[order].contiguous()
    spikes = torch.rand((case["steps"], chans, case["trials"]), generator=g, device=dev) < case["rate"] / 1000.0
    words = (spikes.to(torch.int64) << torch.arange(case["trials"], device=dev)).sum(2)
    bits = torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)
    return targets.cpu().numpy(), pres.cpu().numpy(), w, bits


def exact(case, seed):
    """Simulation results are whole numbers: none. For the differentiable
    form the spike trains are those of the model in float32 (a threshold
    decided in 64 bits gives another trajectory, not a more exact one): sums
    in synapse order, every operation rounded once. The gradient of the
    counts along them is in 64 bits."""
    if case["kind"] != "lif":
        return None
    n, chans, T, B = case["n"], case["chans"], case["steps"], case["trials"]
    targets, pres, w, bits = _lif_inputs(case, seed)
    tgt, pre = torch.as_tensor(targets, device="cuda"), torch.as_tensor(pres, device="cuda")
    degree = torch.bincount(tgt, minlength=n)
    start = torch.cumsum(degree, 0) - degree
    slot = torch.arange(tgt.numel(), device="cuda") - start[tgt]
    D = int(degree.max())
    # synapses of each neuron in order, padded with weight 0 (adds nothing)
    pre_pad = torch.zeros((D, n), dtype=torch.int64, device="cuda")
    w_pad = torch.zeros((D, n, 1), device="cuda")
    pre_pad[slot, tgt] = pre
    w_pad[slot, tgt, 0] = w
    unit = torch.arange(B, device="cuda")
    X = torch.zeros((T, n + chans, B), device="cuda")     # presynaptic spikes of each step
    X[:, n:] = ((bits[:, :, None] >> unit) & 1).float()
    beta = float(np.float32(1.0) - np.float32(1.0) / np.float32(TAU_M))
    S = torch.zeros((T, n, B), device="cuda")
    v = torch.zeros((n, B), device="cuda")
    for t in range(T):
        if t:
            X[t, :n] = S[t - 1]
        current = torch.zeros((n, B), device="cuda")
        for d in range(D):
            current = current + w_pad[d] * X[t][pre_pad[d]]
        u = beta * v + current
        S[t] = (u >= 1.0).float()
        v = u - S[t]
    counts = S.double().sum(1).reshape(T // BIN, BIN, B).sum(1).T
    if not case["grad"]:
        return {"counts": counts, "spikes": None}
    w64 = w.double()
    rec = pre < n
    W = torch.sparse_coo_tensor(torch.stack([tgt, pre]), w64, (n, n + chans)).to_sparse_csr()
    Wt = torch.sparse_coo_tensor(torch.stack([pre[rec], tgt[rec]]), w64[rec], (n, n)).to_sparse_csr()
    U = torch.zeros((T, n, B), dtype=torch.float64, device="cuda")
    v = torch.zeros((n, B), dtype=torch.float64, device="cuda")
    for t in range(T):
        U[t] = beta * v + W @ X[t].double()
        v = U[t] - S[t].double()
    c = counts.clone().requires_grad_(True)
    target = sinusoid_target_64(T // BIN)
    ((c / (n * BIN / 1000.0) - target) ** 2).mean().backward()
    dc = c.grad
    G = torch.zeros((T, n, B), dtype=torch.float64, device="cuda")
    gu = None
    for t in reversed(range(T)):
        gs = dc[:, t // BIN].expand(n, B)
        gv = 0.0
        if gu is not None:
            gs = gs + Wt @ gu
            gv = beta * gu
        surrogate = 1.0 / (1.0 + KAPPA * (U[t] - 1.0).abs()) ** 2
        gu = surrogate * (gs - gv) + gv
        G[t] = gu
    del U
    grad = torch.zeros((D, n), dtype=torch.float64, device="cuda")
    for d in range(D):
        for t0 in range(0, T, 100):
            grad[d] += (G[t0:t0 + 100] * X[t0:t0 + 100][:, pre_pad[d]].double()).sum((0, 2))
    return {"counts": counts, "grad": grad[slot, tgt]}


def sinusoid_target_64(bins):
    t = (torch.arange(bins, device="cuda", dtype=torch.float64) + 0.5) * BIN / 1000.0
    return (20.0 + 10.0 * torch.sin(2.0 * math.pi * 4.0 * t)).float().double()


def tolerance(case):
    # simulation: integers and fixed-point weights. The differentiable form:
    # the spike trains are whole; the gradient, sums of up to 1e5 float32
    # terms, is 1e-7 to 6e-7 off its 64-bit value, and as far from the same
    # sums in another order; a network that hardly spikes has fewer, larger
    # terms.
    return {"rel": 1e-5} if case["kind"] == "lif" else "exact"


def work(case):
    kind = case["kind"]
    if kind == "lif":
        nnz, words = case["n"] * (case["fan"] + case["infan"]), case["steps"] * case["chans"]
        per_step = case["trials"] * case["steps"]
        flops = 0.05 * nnz * per_step       # a spike in twenty (synapse, trial) pairs adds its weight
        moved = 8 * nnz + 4 * words
        if case["grad"]:
            flops += 2.05 * case["n"] * case["fan"] * per_step   # the adjoint's w * gu, the gradient's sums
            moved += 4 * nnz
        return {"bytes": moved, "flops": flops}
    n, m, cycles = _neurons(case), case["m"], case["cycles"]
    # a network fires at some 7 Hz; the mixed network at 200
    rate = 0.2 if kind == "mixed" else 0.007
    per_cycle = 92 * n + 8 * rate * n * m
    moved = cycles * per_cycle
    if case.get("stdp"):
        plastic = 0.8 * n * m
        moved += cycles * 20 * rate * plastic + 20 * plastic
    # the HH model: 999 substeps of about 120 operations
    flops = 30 * cycles * n + (120e3 * cycles * case["hh"] if kind == "mixed" else 0)
    return {"bytes": moved, "flops": flops}
