"""Edge cases of the step engine, bit-exact against the oracle: no synapses,
in-degree above the fast path's 1,024 (the general drain), more than 32
inline generator inputs, a one-step minimum delay (one step per launch),
very long delays, and the raster capacity error."""
import numpy as np
import pytest

import neuronbridge_gb300 as nb
from neuronbridge_gb300 import Connection, Network, NeuronLayer, SimulationConfig, float32
from neuronbridge_gb300.workloads import LIF_PARAMS

pytestmark = pytest.mark.gpu


def _lif(n, **kw):
    return NeuronLayer("TimeDrivenLIF_Voltage_jump", n, parameters=dict(LIF_PARAMS, **kw.pop("params", {})), **kw)


def _check(net, cfg, steps, **sim_kw):
    import oracle

    sim = nb.Simulation(net, cfg, **sim_kw)
    sim.run(steps)
    o = oracle.OracleNet(net.to_native().flat(cfg.timestep))
    o.run(steps)
    d = net.to_native()
    keep = np.repeat(d.layer_output, d.layer_count)
    t, i = o.spikes()
    t, i = t[keep[i]], i[keep[i]]
    order = np.lexsort((i, t))
    st, si = sim.spike_raster()
    assert np.array_equal(st, t[order]) and np.array_equal(si, i[order])
    assert np.array_equal(sim.state_field(0), o.state(0).astype(np.float32))
    assert sim.num_events == o.num_events
    return sim


def test_no_synapses_constant_current(oracle_lib):
    net = Network().add_layer(_lif(64, output=True, params={"I_ext": float32(20.0)}))
    sim = _check(net, SimulationConfig(steps=3000, timestep=0.1), 3000)
    assert len(sim.spike_raster()[0]) > 0 and sim.num_events == 0


def test_in_degree_above_fast_path(oracle_lib):
    """Targets with 1,500 in-synapses (47 mask words) drain through the
    general path; sources are LIF neurons driven by Poisson generators."""
    rng = np.random.default_rng(4)
    net = Network()
    net.add_layer(_lif(2000))
    net.add_layer(_lif(20, output=True))
    net.add_layer(NeuronLayer.poisson_rate(2000, rate_bias_hz=6000.0, rate_gain_hz_per_current=0.0))
    ids = np.arange(2000, dtype=np.int32)
    net.connect(Connection(ids + 2020, ids, weight=0.6, delay=1))
    src = np.concatenate([rng.choice(2000, 1500, replace=False) for _ in range(20)]).astype(np.int32)
    tgt = np.repeat(np.arange(2000, 2020), 1500).astype(np.int32)
    typ = (rng.random(len(src)) < 0.2).astype(np.int32)
    net.connect(Connection(src, tgt, synapse_type=typ, weight=0.05, delay=rng.integers(2, 9, len(src)).astype(np.int32)))
    sim = _check(net, SimulationConfig(steps=1500, timestep=0.1), 1500)
    assert np.any(sim.spike_raster()[1] >= 2000)


def test_many_generator_inputs(oracle_lib):
    """40 inline Poisson generator inputs per target (> 32: general path)."""
    net = Network()
    net.add_layer(_lif(50, output=True))
    net.add_layer(NeuronLayer.poisson_rate(400, rate_bias_hz=900.0, rate_gain_hz_per_current=0.0))
    rng = np.random.default_rng(5)
    src = (50 + np.concatenate([rng.choice(400, 40, replace=False) for _ in range(50)])).astype(np.int32)
    tgt = np.repeat(np.arange(50), 40).astype(np.int32)
    net.connect(Connection(src, tgt, weight=1.2, delay=rng.integers(1, 4, len(src)).astype(np.int32)))
    sim = _check(net, SimulationConfig(steps=2000, timestep=0.1), 2000)
    assert len(sim.spike_raster()[0]) > 0


def test_one_step_delay_and_long_delays(oracle_lib):
    """Recurrent delay 1 (B = 1: one step per launch) next to 3,000-step
    delays (a 3,001-slot ring)."""
    rng = np.random.default_rng(6)
    net = Network()
    net.add_layer(_lif(300, output=True))
    net.add_layer(NeuronLayer.poisson_rate(300, rate_bias_hz=7000.0, rate_gain_hz_per_current=0.0))
    ids = np.arange(300, dtype=np.int32)
    net.connect(Connection(ids + 300, ids, weight=0.5, delay=1))
    s, t = rng.integers(0, 300, 3000).astype(np.int32), rng.integers(0, 300, 3000).astype(np.int32)
    net.connect(Connection(s, t, weight=0.4, delay=np.where(rng.random(3000) < 0.5, 1, 3000).astype(np.int32)))
    sim = _check(net, SimulationConfig(steps=7000, timestep=0.1), 7000)
    assert sim.block_steps == 1


def test_raster_capacity_overflow_is_an_error():
    net = Network().add_layer(_lif(64, output=True, params={"I_ext": float32(20.0)}))
    sim = nb.Simulation(net, SimulationConfig(steps=3000, timestep=0.1), spike_capacity=10)
    with pytest.raises(nb.NbgError, match="capacity"):
        sim.run(3000)


def test_weights_of_more_synapses_than_a_gather_chunk():
    """Weights come back in original connection order in chunks of 2^24 synapses; traces of a static network are 0."""
    from neuronbridge_gb300 import NetworkDescription, NeuronLayer
    from neuronbridge_gb300.workloads import LIF_PARAMS

    n, s = 5000, (1 << 24) + 70_001
    rng = np.random.default_rng(2)
    w = rng.random(s, dtype=np.float32)
    d = NetworkDescription.from_arrays([NeuronLayer("TimeDrivenLIF_Voltage_jump", n, parameters=dict(LIF_PARAMS))],
                                       rng.integers(0, n, s, dtype=np.int32), rng.integers(0, n, s, dtype=np.int32),
                                       np.zeros(s, np.int32), w, delay=np.full(s, 3, np.int32))
    sim = nb.Simulation(d, nb.SimulationConfig(steps=1, timestep=0.1))
    got = sim.weights()
    assert np.array_equal(got["weight"], w)
    assert not got["apre"].any() and not got["apost"].any() and not got["last_update"].any()


def test_a_reset_is_complete_when_the_next_call_starts():
    """Trials of a network whose ring takes longer to clear than a run call takes to start: every trial after a reset
    records the same spikes."""
    from neuronbridge_gb300 import workloads

    net, cfg = workloads.izhikevich_stdp(n=60_000, in_degree=100, steps=120, seed=6)
    sim = nb.Simulation(net, cfg, seed=6)
    first = None
    for _ in range(12):
        sim.reset()
        sim.run(120)
        t, i = sim.spike_raster()
        if first is None:
            first = t.copy(), i.copy()
        assert len(t) > 0 and np.array_equal(t, first[0]) and np.array_equal(i, first[1])


def test_trials_after_a_reset_equal_the_oracle(oracle_lib):
    """The same at the headline size against the oracle's raster, so that a loss that every trial has would show."""
    import oracle
    from neuronbridge_gb300 import workloads

    net, cfg = workloads.izhikevich_stdp(n=100_000, in_degree=100, steps=500, seed=6)
    ref = oracle.OracleNet(net.to_native().flat(cfg.timestep, seed=6)).set_threads(8)
    ref.run(500)
    ot, oi = ref.spikes()  # every layer of this network is an output layer
    order = np.lexsort((oi, ot))
    v, u = (ref.state(f).astype(np.float32) for f in (0, 1))
    sim = nb.Simulation(net, cfg, seed=6)
    for _ in range(3):
        sim.reset()
        sim.run(500)
        t, i = sim.spike_raster()
        assert len(t) > 0 and np.array_equal(t, ot[order]) and np.array_equal(i, oi[order])
        assert np.array_equal(sim.state_field(0), v) and np.array_equal(sim.state_field(1), u)


def test_event_log_of_many_short_calls(oracle_lib):
    """Each call's log is emptied before the next call writes its first entry: every delivered event is in it once."""
    import oracle
    from neuronbridge_gb300 import workloads

    net, cfg = workloads.plain_lif(steps=400)
    sim = nb.Simulation(net, cfg, event_log_capacity=2_000_000)
    for _ in range(100):
        sim.run(4)
    o = oracle.OracleNet(net.to_native().flat(cfg.timestep))
    o.set_event_log(True)
    o.run(400)
    gt, gc, gw = sim.logged_events()
    ot, oc, ow = o.events()
    g, k = np.lexsort((gc, gt)), np.lexsort((oc, ot))
    assert len(ot) > 0 and np.array_equal(gt[g], ot[k]) and np.array_equal(gc[g], oc[k])
    assert np.array_equal(gw[g], ow[k].astype(np.float32))
