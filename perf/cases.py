"""Workloads of the simulation core, through the entry points a program calls.

A case is one pass of a kind of work that users of this package run:

  frame       an editor-like frame: a small liquid advanced by a few steps,
              then its membrane potentials, traces and recent spike counts
              read back; the sim goes on from frame to frame
  trial       one network simulated from reset and read out: the random K-out
              networks (80/20 excitatory/inhibitory, distance delays) of 10k,
              100k and 1M neurons, Izhikevich or AdEx, quiet (Gaussian current
              noise alone) or active (Poisson kicks on top, ~22 Hz), with the
              fixed-point or the float ring
  driven      a trial of a network with synapses that have their own time
              constant, input streams and a spike record
  batch       many local 3-D liquids of uneven size stepped together, each
              with its input streams, read out as spike counts per window
  serve       a burst of trial requests through the server, host data in and
              window counts out
  build       a new network from a plain synapse list, and its first steps
  fit_multi   the multi-class ridge readout of window counts
  fit_binary  the binary ridge readout

Float-ring networks are quiet here: float additions arrive in any order, and
in a spiking network a last bit moves spikes after some tens of milliseconds,
so two runs of the same active float-ring trial are not comparable.
"""
import math

import numpy as np
import torch

import neuro_edit_v2_b200 as nb
from neuro_edit_v2_b200 import workloads as W

IZH_EXC, IZH_INH = (0.02, 0.2, -65.0, 8.0), (0.1, 0.2, -65.0, 2.0)
ADEX_EXC = (281.0, 30.0, -70.6, -50.4, 2.0, 4.0, 144.0, 80.5, -70.6, 20.0)
ADEX_INH = (281.0, 30.0, -70.6, -50.4, 2.0, 0.0, 144.0, 0.0, -70.6, 20.0)
ADEX_GAIN = 281.0  # weights of AdEx networks are currents in pA: scaled by C
FRAME_INPUTS = 8


def listed():
    return [
        # the smallest call: one 1 ms frame of a 1,000-neuron liquid
        dict(name="frame_1k", kind="frame", side=10, steps=10),
        # the 10,000-neuron network as configured, float ring: launch latency
        dict(name="trial_10k_f32_quiet", kind="trial", n=10000, k=100, model="izh", ring="f32", kick_hz=0.0,
             record=False, steps=2000),
        # the 100,000-neuron network as configured, fixed-point ring
        dict(name="trial_100k_quiet", kind="trial", n=100000, k=100, model="izh", ring="int", kick_hz=0.0,
             record=False, steps=2000),
        # the same size, active, with the spike record and a 50 ms readout window
        dict(name="trial_100k_active", kind="trial", n=100000, k=100, model="izh", ring="int", kick_hz=100.0,
             record=True, steps=1500),
        # the largest network, active: 1e8 synapses, a ring far larger than L2
        dict(name="trial_1m_active", kind="trial", n=1000000, k=100, model="izh", ring="int", kick_hz=100.0,
             record=False, steps=800),
        # the AdEx variant of the largest network, as configured
        dict(name="trial_1m_adex", kind="trial", n=1000000, k=100, model="adex", ring="int", kick_hz=0.0,
             record=False, steps=800),
        # a ragged size with custom synapse currents, input streams and a record
        dict(name="driven_20k", kind="driven", n=20011, k=40, tau_share=0.25, steps=1000),
        # uneven liquids in one batch: 150 ms trials, 50 ms windows, kicks 30 Hz
        dict(name="batch_48_liquids", kind="batch", count=48, kick_hz=30.0, steps=1500),
        # twelve requests of 2,000-50,000 neurons and 200-2000 ms at once
        dict(name="serve_12", kind="serve", count=12, longest=20000),
        # an unordered list of 2e7 synapses becomes a network and runs 10 ms
        dict(name="build_200k", kind="build", n=200000, k=100, shuffled=True, steps=100),
        # 1,000 trials of a 216-neuron liquid x 20 windows, four classes
        dict(name="fit_multi_1000x4320", kind="fit_multi", t=1000, f=4320, classes=4, on_device=True),
        # 1,200 trials x 5 windows of the same liquid, design in host memory
        dict(name="fit_binary_1200x1080", kind="fit_binary", t=1200, f=1080, on_device=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "trial", "trial", "trial", "driven", "batch", "serve", "build", "fit_multi",
                       "fit_binary"])
    if kind == "frame":
        return dict(kind=kind, side=rng.randint(5, 24), steps=_log_int(rng, 1, 100))
    if kind == "trial":
        n = _log_int(rng, 1000, 1000000)
        k = rng.randint(30, 100)
        ring = "f32" if rng.random() < 0.25 else "int"
        kick = 0.0 if ring == "f32" or rng.random() < 0.4 else 100.0
        steps = rng.randint(200, max(201, min(2000, 600000000 // n)))
        return dict(kind=kind, n=n, k=k, model=rng.choice(["izh", "izh", "adex"]), ring=ring, kick_hz=kick,
                    record=rng.random() < 0.5, steps=steps)
    if kind == "driven":
        return dict(kind=kind, n=_log_int(rng, 500, 30000), k=rng.randint(10, 50),
                    tau_share=round(rng.uniform(0.05, 0.5), 3), steps=rng.randint(200, 1000))
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 4, 64), kick_hz=rng.choice([0.0, 30.0]),
                    steps=rng.randint(500, 1500))
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(2, 12), longest=rng.randint(4000, 20000))
    if kind == "build":
        return dict(kind=kind, n=_log_int(rng, 2000, 300000), k=rng.randint(20, 100), shuffled=rng.random() < 0.7,
                    steps=rng.randint(20, 100))
    if kind == "fit_multi":
        return dict(kind=kind, t=_log_int(rng, 40, 1500), f=_log_int(rng, 100, 6000), classes=rng.randint(2, 6),
                    on_device=rng.random() < 0.7)
    return dict(kind=kind, t=_log_int(rng, 60, 1500), f=_log_int(rng, 30, 1300), on_device=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _neurons(n, model):
    """80/20 excitatory/inhibitory rows: (model ids, parameter rows, kinds)."""
    inh = np.arange(n) >= int(0.8 * n)
    exc_row, inh_row = (ADEX_EXC, ADEX_INH) if model == "adex" else (IZH_EXC, IZH_INH)
    rows = np.where(inh[:, None], np.float32(inh_row), np.float32(exc_row)).astype(np.float32)
    ids = np.full(n, nb.MODEL_ADEX if model == "adex" else nb.MODEL_IZH, np.uint8)
    return ids, rows, inh.astype(np.uint8)


def _synapse_list(n, k, seed, gain=1.0, shuffled=False):
    """Random K-out synapses on the device: targets uniform, positions uniform
    in a 1000 um cube, delay = distance / (100 um per ms) up to 20 ms,
    |w| uniform in [0, 0.5] (exc) or [0, 1] (inh) x 0.7."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    e = n * k
    pos = torch.rand((n, 3), device="cuda", generator=g) * 1000.0
    src = torch.arange(n, device="cuda").repeat_interleave(k)
    tgt = torch.randint(0, n, (e,), device="cuda", generator=g)
    w = torch.rand(e, device="cuda", generator=g)
    w *= torch.where(src < int(0.8 * n), 0.5, 1.0) * (0.7 * gain)
    d2 = torch.zeros(e, device="cuda")
    for axis in range(3):
        d2 += (pos[:, axis][src] - pos[:, axis][tgt]) ** 2
    delay = (d2.sqrt() / 100.0).clamp(0.1, 20.0)
    if shuffled:
        order = torch.randperm(e, device="cuda", generator=g)
        src, tgt, w, delay = src[order], tgt[order], w[order], delay[order]
    cols = (src.to(torch.int32).view(torch.uint32), tgt.to(torch.int32).view(torch.uint32), w.contiguous(),
            delay.contiguous())
    torch.cuda.synchronize()
    return cols


def _sim_from_list(case, cols, seed):
    ids, rows, kinds = _neurons(case["n"], case.get("model", "izh"))
    kick = case.get("kick_hz", 100.0)
    cfg = nb.default_config(int_weights=0 if case.get("ring") == "f32" else 1, gauss_sd=1.0, synapse_tau_ms=5.0,
                            noise_rate_hz=kick, noise_kick_mv=20.0 if kick else 0.0, seed=seed + 1,
                            record_spikes=1 if case.get("record") else 0, spike_record_steps=512)
    return nb.B200Sim.from_synapses(ids, rows, kinds, *cols, cfg)


def _design(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.poisson(1.5, (case["t"], case["f"])).astype(np.float32)
    y = rng.integers(0, case.get("classes", 2), case["t"])
    return x, y.astype(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "frame":
        net = nb.liquid(case["side"], seed=seed + 1)
        sim = nb.B200Sim(net, nb.default_config(int_weights=1, record_spikes=1, seed=seed + 1, noise_rate_hz=100.0,
                                                noise_kick_mv=20.0))
        rng = np.random.default_rng(seed)
        for j, s in enumerate(W.bit_streams(rng, 100, FRAME_INPUTS).T):
            sim.loop_input(j, s)
        sim.run_steps(200)  # a frame is taken from a running network
        sim.synchronize()
        st["sim"] = sim
    elif kind == "trial":
        gain = ADEX_GAIN if case["model"] == "adex" else 1.0
        st["sim"] = _sim_from_list(case, _synapse_list(case["n"], case["k"], seed, gain), seed)
    elif kind == "driven":
        n, k = case["n"], case["k"]
        rng = np.random.default_rng(seed)
        ids, rows, kinds = _neurons(n, "izh")
        e = n * k
        tau = np.where(rng.random(e) < case["tau_share"], rng.uniform(1.0, 30.0, e), 0.0)
        net = nb.from_synapses(ids, rows, kinds, np.repeat(np.arange(n), k), rng.integers(0, n, e),
                               rng.random(e) * 0.7, rng.uniform(0.1, 15.0, e), tau_ms=tau)
        flat = W.with_inputs(net, FRAME_INPUTS, 24, 12.0, rng)
        sim = nb.B200Sim(flat, nb.default_config(int_weights=1, record_spikes=1, synapse_tau_ms=5.0, seed=seed + 1,
                                                 noise_rate_hz=100.0, noise_kick_mv=20.0))
        for j, s in enumerate(W.bit_streams(rng, 200, FRAME_INPUTS).T):
            sim.loop_input(j, s)
        st["sim"] = sim
    elif kind == "batch":
        count = case["count"]
        rng = np.random.default_rng(seed)
        # the cube sides follow from the count alone, and so does a case's work
        sides = W.batched_liquid_sizes(count)
        nets = [nb.liquid(s, seed=1000 * (seed % 100000) + j)
                for j, s in enumerate(sides)]
        kick = case["kick_hz"]
        wins = max(1, case["steps"] // W.WINDOW_STEPS)
        b = nb.Batch(nets, [nb.default_config(int_weights=1, window_steps=W.WINDOW_STEPS, max_windows=wins,
                                              seed=seed + j, noise_rate_hz=kick, noise_kick_mv=20.0 if kick else 0.0)
                            for j in range(count)])
        st.update(batch=b, windows=wins,
                  inputs=[W.bit_streams(rng, -(-case["steps"] // W.SPB)) for _ in range(count)])
    elif kind == "serve":
        # sizes and durations follow from the count alone; nets, streams and noise from the seed
        specs = W.request_stream(case["count"], seed=7)
        st["requests"] = []
        for j, q in enumerate(specs):
            rng = np.random.default_rng([seed, j])
            gain = ADEX_GAIN if q.model == nb.MODEL_ADEX else 1.0
            if q.wiring == "local":
                net = nb.liquid(round(q.n ** (1.0 / 3.0)), seed=seed + j + 1, model=q.model)
            else:
                net = nb.random_kout(q.n, 100, seed + j + 1, w_scale=0.7 * gain)
                if q.model == nb.MODEL_ADEX:
                    nb.to_adex(net)
                net = W.with_inputs(net, 8, 24, 12.0 * gain, rng)
            q.steps = min(q.steps, case["longest"] // W.SPB * W.SPB)
            inputs, _ = W.coincident_streams(rng, q.steps // W.SPB)
            st["requests"].append((net, W.request_config(q, seed + j), inputs, q.steps))
        st["server"] = nb.Server(neuron_capacity=16 << 20, synapse_capacity=1 << 30, ring_capacity=6 << 30,
                                 max_requests=64, steps_per_launch=100, admission_threads=4)
    elif kind == "build":
        st["cols"] = _synapse_list(case["n"], case["k"], seed, shuffled=case["shuffled"])
        st["seed"] = seed
    else:
        x, y = _design(case, seed)
        st["x"] = torch.from_numpy(x).cuda() if case["on_device"] else x
        st["y"] = y if kind == "fit_multi" else y.astype(np.float32)
        torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------- pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        sim = state["sim"]
        sim.run_steps(case["steps"])
        return {"v": sim.v(), "trace": sim.trace(), "counts": sim.spike_counts(case["steps"])}
    if kind in ("trial", "driven"):
        sim = state["sim"]
        sim.reset_state()
        sim.run_steps(case["steps"])
        out = {"v": sim.v(), "u": sim.state(1), "s": sim.syn_current(), "spikes": sim.spikes_total()}
        if kind == "driven" or case["record"]:
            out["counts"] = sim.spike_counts(case["steps"])
            if case["steps"] > 500:
                out["window"] = sim.spike_counts(500)
        return out
    if kind == "batch":
        b = state["batch"]
        b.reset_state()
        for j, x in enumerate(state["inputs"]):
            b.set_input_matrix(j, x)
        b.run_steps(case["steps"])
        nets = range(case["count"])
        return {"counts": np.concatenate([b.window_counts(j, w) for j in nets for w in range(state["windows"])]),
                "v": np.concatenate([b.state(j, 0) for j in nets]),
                "spikes": np.array([b.spikes_total(j) for j in nets], np.int64)}
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(*q) for q in state["requests"]]
        while srv.stats()["active"]:
            srv.step()
        got = [srv.take(i) for i in ids]
        return {"counts": np.concatenate([c.reshape(-1) for c, _ in got]),
                "spikes": np.array([t for _, t in got], np.int64)}
    if kind == "build":
        with _sim_from_list(case, state["cols"], state["seed"]) as sim:
            sim.run_steps(case["steps"])
            return {"v": sim.v(), "u": sim.state(1), "s": sim.syn_current(), "spikes": sim.spikes_total(),
                    "synapses": sim.syn_count()}
    if kind == "fit_multi":
        return {"w": nb.fit_ridge_multi(state["x"], state["y"], case["classes"], 1.0)}
    return {"w": nb.fit_ridge(state["x"], state["y"], 1.0)}


# -------------------------------------------------------------------- work
def _steps_work(n, steps, events, adex=False):
    """v, u and s read and written and the due ring word read, per neuron and
    step; a synapse record and a ring word per synaptic event."""
    return {"bytes": float(steps) * n * 28 + float(events) * 12, "flops": float(steps) * n * (60 if adex else 25)}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        return _steps_work(case["side"] ** 3, case["steps"], 0)
    if kind == "trial":
        rate = 22.0 if case["kick_hz"] else 0.0  # Hz, as measured
        events = case["n"] * case["k"] * rate * case["steps"] * 1e-4
        return _steps_work(case["n"], case["steps"], events, case["model"] == "adex")
    if kind == "driven":
        return _steps_work(case["n"], case["steps"], case["n"] * case["k"] * 22.0 * case["steps"] * 1e-4)
    if kind == "batch":
        n = sum(s ** 3 for s in W.batched_liquid_sizes(case["count"]))
        return _steps_work(n, case["steps"], n * 37 * (20.0 if case["kick_hz"] else 0.0) * case["steps"] * 1e-4)
    if kind == "serve":  # 15,000 neurons x 11,000 steps on average, ~40 synapses per spike, 50 Hz
        n_steps = case["count"] * 15000.0 * min(11000.0, 0.7 * case["longest"])
        return _steps_work(1, n_steps, n_steps * 60 * 50 * 1e-4)
    if kind == "build":
        e = case["n"] * case["k"]
        w = _steps_work(case["n"], case["steps"], e * 22.0 * case["steps"] * 1e-4)
        return {"bytes": w["bytes"] + e * 24.0, "flops": w["flops"]}
    t, f = float(case["t"]), float(case["f"])
    if kind == "fit_multi":
        return {"bytes": 4 * t * f + 8 * case["classes"] * f,
                "flops": t * t * f + t ** 3 / 3 + 2 * case["classes"] * (t * t + t * f)}
    return {"bytes": 4 * t * f + 8 * f, "flops": t * f * f + f ** 3 / 3 + 2 * f * f}


# ------------------------------------------------------------------- exact
def _exact_quiet(case, seed):
    """A quiet trial in 64 bits: no neuron spikes, so each is alone with its
    Gaussian current, whose whole-number draws come from a counter hash of
    (neuron, step, seed).  None if a neuron does spike."""
    n, adex = case["n"], case["model"] == "adex"
    _, rows, _ = _neurons(n, case["model"])
    p = torch.from_numpy(rows).cuda().double().T.contiguous()
    dt = float(np.float32(0.1))
    amp = math.sqrt(3.0) / 256.0
    idx = torch.arange(n, device="cuda", dtype=torch.int64)
    v = p[2].clone() if adex else torch.full((n,), -65.0, device="cuda", dtype=torch.float64)
    u = torch.zeros_like(v) if adex else p[1] * v
    worst = torch.full((), -1e300, device="cuda", dtype=torch.float64)
    m32 = 0xFFFFFFFF
    for t in range(case["steps"]):
        step = (t * 0xBF58476D1CE4E5B9 + (seed + 1) * 0x94D049BB133111EB) & ((1 << 64) - 1)
        x = idx ^ (step & m32)
        x = x ^ (x >> 16)
        x = (x * 0x7FEB352D) & m32
        x = x ^ (x >> 15)
        x = (x * 0x846CA68B) & m32
        x = x ^ (x >> 16)
        x = x ^ (step >> 32)
        x = (x * 0x9E3779B1) & m32
        x = x ^ (x >> 16)
        draws = (x & 255) + ((x >> 8) & 255) + ((x >> 16) & 255) + (x >> 24) - 510
        cur = draws.double() * amp
        if adex:
            cur = cur * p[0]
            ex = torch.exp(torch.clamp((v - p[3]) / p[4], max=10.0))
            v = v + dt * (-p[1] * (v - p[2]) + p[1] * p[4] * ex - u + cur) / p[0]
            u = u + dt * (p[5] * (v - p[2]) - u) / p[6]
        else:
            v = v + dt * (0.04 * v * v + 5.0 * v + 140.0 - u + cur)
            u = u + dt * p[0] * (p[1] * v - u)
        worst = torch.maximum(worst, v.max())
    if float(worst) >= (20.0 if adex else 30.0):
        return None
    return {"v": v.cpu().numpy(), "u": u.cpu().numpy(), "s": np.zeros(n)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "trial" and not case["kick_hz"]:
        return _exact_quiet(case, seed)
    if kind in ("fit_multi", "fit_binary"):
        x, y = _design(case, seed)
        x = x.astype(np.float64)
        t, f = x.shape
        if kind == "fit_multi":
            mu = x.mean(axis=0)
            xc = x - mu
            k = case["classes"]
            one = (y[:, None] == np.arange(k)).astype(np.float64)
            ybar = one.mean(axis=0)
            a = np.linalg.solve(xc @ xc.T + np.eye(t), one - ybar)
            w = (xc.T @ a).T
            return {"w": np.concatenate([w, (ybar - w @ mu)[:, None]], axis=1)}
        x1 = np.concatenate([x, np.ones((t, 1))], axis=1)
        reg = np.eye(f + 1)
        reg[f, f] = 0.0
        return {"w": np.linalg.solve(x1.T @ x1 + reg, x1.T @ y.astype(np.float64))}
    return None  # a spiking network's state has no 64-bit counterpart: rounding moves spikes
