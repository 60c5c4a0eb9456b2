"""The work that a user of this framework has it do, as cases that can be timed.

Each case is a dict of plain values.  ``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges,
``prepare(case, seed)`` makes what a program has in hand before the call (built simulation, model, weights, inputs),
``run(state)`` is one pass through the public entry points, ``work(case)`` the bytes and operations one pass cannot do
without, and ``exact(case, seed)`` the results in 64 bits where the path has such results.

Kinds of work:

* ``loop``     a closed control loop: external spikes in, ten steps, the call's output spikes out
* ``lif``      a static voltage-jump LIF network under Poisson drive, one ``run`` call and its raster
* ``batch``    many such networks of different sizes in one engine
* ``stdp``     current-based Izhikevich neurons with pair STDP: reset, one trial, raster and state (and learned weights)
* ``dense``    64 instances of an all-to-all LIF population sharing one weight matrix
* ``deliver``  one dense spike delivery from host spikes to host currents
* ``train``    one training step of the recurrent LIF network: encode rates to spikes, forward, loss, backward
* ``infer``    encode and forward of that network alone
"""
import math

import numpy as np
import torch

import neuronbridge_gb300 as nb
from neuronbridge_gb300 import workloads
from neuronbridge_gb300.adjoint import RecurrentLIF, poisson_inputs
from neuronbridge_gb300.dense import DensePopulations

DT = 0.1


def listed():
    return [
        # the smallest call: a robot controller that exchanges spikes with its network once per simulated millisecond
        {"name": "loop_500", "kind": "loop", "inputs": 64, "neurons": 500, "steps": 10},
        # a small network simulated for 100 ms; the sizes of the plain LIF benchmark
        {"name": "lif_1k", "kind": "lif", "neurons": 1000, "steps": 1000, "rate": 8000.0},
        # a parameter sweep: networks of 500 to 50,000 neurons in one engine, larger than the L2 cache
        {"name": "batch_16", "kind": "batch", "instances": 16, "lo": 500, "hi": 50000, "steps": 200},
        # a learning experiment that reads its weights after every trial
        {"name": "stdp_5k", "kind": "stdp", "neurons": 5000, "steps": 500, "weights": True},
        # the headline network (100,000 neurons, 10 million synapses), one 50 ms trial
        {"name": "stdp_100k", "kind": "stdp", "neurons": 100000, "steps": 500, "weights": False},
        # 64 all-to-all populations at the dense benchmark's size, and at an odd multiple of the tile
        {"name": "dense_8192", "kind": "dense", "neurons": 8192, "steps": 100, "precision": "split_bf16"},
        # the exact FP32 path of the same populations at a size the tests use
        {"name": "dense_fp32_2k", "kind": "dense", "neurons": 2048, "steps": 100, "precision": "fp32"},
        # one delivery from and to host memory, the form a co-simulator calls
        {"name": "deliver_1152", "kind": "deliver", "neurons": 1152, "precision": "split_bf16", "rate": 0.03},
        # the training benchmark's step: 256 inputs, 1,024 recurrent neurons, batch 128, 1,000 steps
        {"name": "train_b128", "kind": "train", "inputs": 256, "neurons": 1024, "outputs": 10, "batch": 128,
         "steps": 1000, "smooth": False},
        # a training step of a smaller model at a smaller batch
        {"name": "train_b32", "kind": "train", "inputs": 128, "neurons": 512, "outputs": 10, "batch": 32, "steps": 250,
         "smooth": False},
        # the smoothed (sigmoid) mode, at sizes that are no multiple of anything
        {"name": "smooth_b12", "kind": "train", "inputs": 50, "neurons": 300, "outputs": 7, "batch": 12, "steps": 60,
         "smooth": True},
        # evaluation of a trained model
        {"name": "infer_b64", "kind": "infer", "inputs": 200, "neurons": 1000, "outputs": 10, "batch": 64,
         "steps": 500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "lif", "batch", "stdp", "dense", "deliver", "train", "train", "smooth", "infer"])
    if kind == "loop":
        return {"kind": "loop", "inputs": _log(rng, 16, 256), "neurons": _log(rng, 100, 5000), "steps": _log(rng, 5, 50)}
    if kind == "lif":
        return {"kind": "lif", "neurons": _log(rng, 200, 8000), "steps": _log(rng, 50, 1000),
                "rate": float(rng.randrange(4000, 12001))}
    if kind == "batch":
        return {"kind": "batch", "instances": rng.randrange(4, 17), "lo": 500, "hi": _log(rng, 4000, 50000),
                "steps": _log(rng, 50, 200)}
    if kind == "stdp":
        n = _log(rng, 2000, 100000)
        return {"kind": "stdp", "neurons": n, "steps": _log(rng, 100, 500), "weights": n <= 10000}
    if kind == "dense":
        fp32 = rng.random() < 0.4
        return {"kind": "dense", "neurons": 256 * _log(rng, 4, 16 if fp32 else 32), "steps": _log(rng, 20, 100),
                "precision": "fp32" if fp32 else "split_bf16"}
    if kind == "deliver":
        fp32 = rng.random() < 0.4
        return {"kind": "deliver", "neurons": 256 * _log(rng, 2, 16) + (0 if fp32 else 128 * rng.randrange(2)),
                "precision": "fp32" if fp32 else "split_bf16", "rate": round(rng.uniform(0.01, 0.06), 4)}
    if kind == "infer":
        return {"kind": "infer", "inputs": _log(rng, 20, 300), "neurons": _log(rng, 64, 1024), "outputs": 10,
                "batch": _log(rng, 1, 128), "steps": _log(rng, 50, 1000)}
    smooth = kind == "smooth"
    tuned = not smooth and rng.random() < 0.3  # the benchmark's batch and a multiple of its tile
    neurons = 128 * rng.randrange(1, 9) if tuned else _log(rng, 64, 512)
    steps = _log(rng, 20, 60) if smooth else _log(rng, 50, 1000 if tuned else 250)
    most = max(2, min(64, int(2.2e9 / (neurons * neurons * steps))))
    return {"kind": "train", "inputs": _log(rng, 20, 256), "neurons": neurons, "outputs": rng.randrange(2, 20),
            "batch": 128 if tuned else _log(rng, 1, most), "steps": steps, "smooth": smooth}


# ------------------------------------------------------------------- inputs


def _lif_description(n, rate, rng):
    """n LIF neurons (80 % excitatory), mean in-degree 100, each with its own Poisson source."""
    src, tgt = workloads.lif_instance_arrays(n, int(rng.integers(1 << 30)))
    ids = np.arange(n, dtype=np.int32)
    inh = src >= (n * 4) // 5
    layers = [nb.NeuronLayer("TimeDrivenLIF_Voltage_jump", n, output=True, parameters=dict(workloads.LIF_PARAMS)),
              nb.NeuronLayer.poisson_rate(n, rate_bias_hz=rate, rate_gain_hz_per_current=0.0)]
    return nb.NetworkDescription.from_arrays(
        layers, np.concatenate([src, ids + n]), np.concatenate([tgt, ids]),
        np.concatenate([inh.astype(np.int32), np.zeros(n, np.int32)]),
        np.concatenate([np.where(inh, 2.5, 0.5).astype(np.float32), np.full(n, 0.5, np.float32)]),
        delay=np.concatenate([np.full(len(src), 15, np.int32), np.ones(n, np.int32)]))


def _batch_sizes(case):
    return np.rint(np.geomspace(case["lo"], case["hi"], case["instances"])).astype(np.int64)


def _loop(case, rng):
    """Input spikes -> LIF (plastic, 2 to 5 ms) and LIF -> LIF (1 to 3 ms)."""
    n_in, n = case["inputs"], case["neurons"]
    net = nb.Network()
    net.add_layer(nb.NeuronLayer.input_spike(n_in))
    net.add_layer(nb.NeuronLayer("TimeDrivenLIF_Voltage_jump", n, output=True, parameters=dict(workloads.LIF_PARAMS)))
    net.add_learning_rule(nb.LearningRule("STDP", {"Max_LTP": nb.float32(0.05), "LTP_tau": nb.float32(20.0),
                                                   "Max_LTD": nb.float32(0.06), "LTD_tau": nb.float32(20.0)}))
    src = np.repeat(np.arange(n_in, dtype=np.int32), 40)
    net.connect(nb.Connection(src, (n_in + rng.integers(0, n, len(src))).astype(np.int32), synapse_type=0, weight=4.0,
                              max_weight=8.0, delay=rng.integers(20, 51, len(src)).astype(np.int32), synapse_rule=0))
    src, tgt = workloads.lif_instance_arrays(n, int(rng.integers(1 << 30)), min(100.0, 0.1 * n))
    inh = src >= (n * 4) // 5
    net.connect(nb.Connection((n_in + src).astype(np.int32), (n_in + tgt).astype(np.int32),
                              synapse_type=inh.astype(np.int32), weight=np.where(inh, 2.0, 1.5).astype(np.float32),
                              delay=rng.integers(10, 31, len(src)).astype(np.int32)))
    when, who = np.nonzero(rng.random((case["steps"], n_in)) < 0.02)  # 200 Hz per input
    sim = nb.Simulation(net, nb.SimulationConfig(steps=case["steps"], timestep=DT))
    warm_when, warm_who = np.nonzero(rng.random((400, n_in)) < 0.02)
    sim.add_external_spikes(warm_when, warm_who)
    sim.run(400)  # the controller has been running: arrivals are in flight
    return {"sim": sim, "when": when.astype(np.int32), "who": who.astype(np.int32)}


def _dense_weights(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, n, generator=g, device="cuda") / math.sqrt(n)


def _spikes(case, seed):
    return (np.random.default_rng(seed).random((64, case["neurons"])) < case["rate"]).astype(np.uint8)


def _dense_layer():
    return nb.NeuronLayer("TimeDrivenLIF_Voltage_jump", 1, parameters=dict(workloads.LIF_PARAMS))


def _model(case, seed):
    smooth = case.get("smooth", False)
    # weights at which the recurrent neurons fire a few per cent of the steps, as a trained model's do
    return RecurrentLIF(case["inputs"], case["neurons"], case["outputs"], smooth=smooth,
                        weight_scale=10.0 if smooth else 20.0, slope=0.5 if smooth else 10.0, seed=seed)


def _rates(case, seed):
    g = torch.Generator().manual_seed(seed)
    lo, hi = (40.0, 400.0) if case.get("smooth", False) else (5.0, 50.0)
    return torch.empty(case["inputs"]).uniform_(lo, hi, generator=g).cuda()


def _labels(case, seed):
    return torch.randint(0, case["outputs"], (case["batch"],), generator=torch.Generator().manual_seed(seed)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    state = {"case": case}
    if kind == "loop":
        state.update(_loop(case, rng))
    elif kind == "lif":
        state["sim"] = nb.Simulation(_lif_description(case["neurons"], case["rate"], rng),
                                     nb.SimulationConfig(steps=case["steps"], timestep=DT))
    elif kind == "batch":
        parts = [_lif_description(int(n), float(rng.uniform(4000.0, 12000.0)), rng) for n in _batch_sizes(case)]
        state["sim"] = nb.Simulation.batch(parts, nb.SimulationConfig(steps=case["steps"], timestep=DT))
    elif kind == "stdp":
        net, cfg = workloads.izhikevich_stdp(n=case["neurons"], steps=case["steps"], seed=seed)
        state["sim"] = nb.Simulation(net, cfg, seed=seed)
    elif kind in ("dense", "deliver"):
        w = _dense_weights(case["neurons"], seed).cpu().numpy()
        state["pop"] = DensePopulations(w, _dense_layer(), precision=case["precision"])
        if kind == "deliver":
            state["s"] = _spikes(case, seed)
    else:
        state["model"] = _model(case, seed)
        state["rates"] = _rates(case, seed)
        state["labels"] = _labels(case, seed)
        state["seed"] = seed % 100003
    return state


def _raster(sim, neurons, steps):
    """The spikes of the call in arrays of a fixed size, zeros after the last: a refractory neuron (20 steps) fires at
    most every 21st step."""
    t, i = sim.spike_raster()
    out = np.zeros((2, neurons * (steps // 21 + 2)), np.int32)
    out[0, :len(t)] = t
    out[1, :len(i)] = i
    return {"count": len(t), "time": out[0], "neuron": out[1]}


def _encode(state):
    case = state["case"]
    return poisson_inputs(state["rates"], case["steps"], case["batch"], dt=1.0, seed=state["seed"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loop":
        sim = state["sim"]
        sim.clear_spikes()
        sim.add_external_spikes(state["when"] + sim.next_time, state["who"])
        sim.run(case["steps"])
        return {**_raster(sim, case["neurons"], case["steps"]), "v": sim.state_field(0)}
    if kind in ("lif", "batch"):
        sim = state["sim"]
        sim.clear_spikes()
        sim.run(case["steps"])
        neurons = case["neurons"] if kind == "lif" else int(_batch_sizes(case).sum())
        return {**_raster(sim, neurons, case["steps"] + 1), "v": sim.state_field(0)}
    if kind == "stdp":
        sim = state["sim"]
        sim.reset()
        sim.run(case["steps"])
        out = {**_raster(sim, case["neurons"], case["steps"] + 1), "v": sim.state_field(0), "u": sim.state_field(1)}
        if case["weights"]:
            out["synapses"] = sim.weights()
        return out
    if kind == "dense":
        pop = state["pop"]
        pop.run(case["steps"])
        v, last = pop.state()
        return {"v": v, "last": last, "spikes": pop.spikes(), "counts": pop.spike_counts()[-case["steps"]:]}
    if kind == "deliver":
        return state["pop"].deliver(state["s"])
    x = _encode(state)
    model = state["model"]
    if kind == "infer":
        with torch.no_grad():
            return model(x)
    model.zero_grad(set_to_none=True)
    y = model(x)
    torch.nn.functional.cross_entropy(y, state["labels"]).backward()
    return {"y": y.detach(), "grads": {name: q.grad for name, q in model.named_parameters()}}


# ---------------------------------------------------------- what it costs


def work(case):
    """Bytes: the state read and written once, the synapse records that the delivered events touch (8 bytes static, 32 read and 16
    written where they learn) or the weights once, inputs and results once.  Operations: those of the arithmetic
    named by the path (products count two per term)."""
    kind, n = case["kind"], case.get("neurons", 0)
    steps = case.get("steps", 1)
    if kind in ("loop", "lif", "batch"):
        if kind == "batch":
            n = int(_batch_sizes(case).sum())
        ev = n * steps * (100 * 0.012 + 0.8) if kind != "loop" else steps * 0.02 * case["inputs"] * 40
        return {"bytes": 16.0 * n + 8.0 * ev + 8.0 * n * steps * 0.012, "flops": 8.0 * n * steps + ev}
    if kind == "stdp":
        ev = n * steps * 0.064
        by = 24.0 * n + 48.0 * ev + 48.0 * ev + 8.0 * n * steps * 0.00064  # arrivals and post-synaptic updates
        if case["weights"]:
            by += 16.0 * 100 * n
        return {"bytes": by, "flops": 60.0 * n * steps + 8.0 * ev}
    if kind in ("dense", "deliver"):
        reads = 4.0 * n * n  # both BF16 halves, or FP32
        rows = 1.0 if case["precision"] == "split_bf16" else 1.0 - (1.0 - case.get("rate", 0.016)) ** 64
        dots = 2.0 * 64 * n * n * (2.0 if case["precision"] == "split_bf16" else 0.5 * case.get("rate", 0.016))
        if kind == "deliver":
            return {"bytes": reads * rows + 64.0 * n * 5, "flops": dots}
        return {"bytes": steps * (reads * rows + 64.0 * n * 2) + 64.0 * n * 13, "flops": steps * dots}
    b, c = case["batch"], case["inputs"]
    o = case["outputs"]
    fire = 0.03 if not case.get("smooth", False) else 1.0
    x_on = 0.0275 if not case.get("smooth", False) else 1.0
    fwd = 2.0 * steps * b * n * (fire * n + x_on * c) + 2.0 * b * n * o
    weights = 4.0 * (n * n + c * n + n * o)
    if kind == "infer":
        return {"bytes": 4.0 * steps * b * c * 2 + weights + 4.0 * b * o, "flops": fwd}
    bwd = 2.0 * steps * b * n * (n + n * fire + c * x_on)
    rec = 13.0 * steps * b * n  # the state the adjoint reads, written and read once
    return {"bytes": 4.0 * steps * b * c * 3 + 2 * rec + 2 * weights, "flops": fwd + bwd}


# ------------------------------------------------------------ in 64 bits


def _exact_smooth(case, seed):
    """The smoothed network and its gradients by autograd over plain FP64 tensor operations."""
    state = {"case": case, "rates": _rates(case, seed), "seed": seed % 100003}
    x = _encode(state).double()
    model = _model(case, seed)
    p = {name: q.detach().double().requires_grad_(True) for name, q in model.named_parameters()}
    T, B, N = case["steps"], case["batch"], case["neurons"]
    slope, rest, reset = 0.5, -65.0, -65.0
    a_out = math.exp(-1.0 / 20.0)
    v = torch.full((B, N), reset, dtype=torch.float64, device="cuda")
    s = torch.zeros_like(v)
    z = torch.zeros_like(v)
    for t in range(T):
        u = v + p["alpha"] * (rest - v) + x[t] @ p["w_in"] + s @ p["w_rec"]
        s = torch.sigmoid(slope * (u - p["theta"]))
        v = u - s * (u - reset)
        z = z + (1.0 - a_out ** (T - t)) / ((1.0 - a_out) * T) * s
    y = z @ p["w_out"]
    torch.nn.functional.cross_entropy(y, _labels(case, seed)).backward()
    return {"y": y.detach(), "grads": {name: q.grad for name, q in p.items()}}


def exact(case, seed):
    """A spiking trajectory has no value in 64 bits to compare with: a rounding moves a threshold crossing, and every
    later value with it.  The smoothed network and a single delivery have."""
    if case["kind"] == "deliver":
        w = _dense_weights(case["neurons"], seed).double()
        return (torch.from_numpy(_spikes(case, seed)).double().cuda() @ w).cpu().numpy()
    if case["kind"] == "train" and case["smooth"]:
        return _exact_smooth(case, seed)
    return None
