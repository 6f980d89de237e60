"""Cases whose speed is measured: what users of the simulator have it do.

A pass is one call of a user's main loop on a compiled network: give the
network this call's inputs (rate-coded networks), simulate a stretch of
model time, and fetch the results the program goes on with (rates, recorded
values, spikes, potentials, weights). Networks keep their state from pass to
pass, as a program that simulates in stretches does. Networks, sizes and
values are those of annarchy_b200.workloads and of the repository's tests,
smaller and larger.

Single-precision networks hand their values back as float64 arrays; the
program keeps them in the network's own float32.
"""
import math

import numpy as np

import annarchy_b200 as ann
from annarchy_b200 import workloads as wl
from annarchy_b200.core.batch import Batch


def listed():
    return [
        # a small rate-coded model inside a program's control loop (inputs in,
        # 10 ms, rates out): latency and launches are all there is
        dict(name="rate_loop_500", kind="rate", n_in=100, n_out=400, p_in=0.1, p_rec=0.05,
             precision="double", storage="csr", steps=10, record=0),
        # the 1000 -> 4000 rate-coded network with recordings, in the default
        # double precision and in single precision
        dict(name="rate_5000_double", kind="rate", n_in=1000, n_out=4000, p_in=0.1, p_rec=0.02,
             precision="double", storage="csr", steps=200, record=10),
        dict(name="rate_5000_float", kind="rate", n_in=1000, n_out=4000, p_in=0.1, p_rec=0.02,
             precision="float", storage="csr", steps=200, record=10),
        # a larger recurrent rate-coded network in single precision, storage
        # format left to the simulator
        dict(name="rate_40000_float", kind="rate", n_in=2000, n_out=38001, p_in=0.01, p_rec=0.0026,
             precision="float", storage="auto", steps=100, record=0),
        # an input sweep: 64 copies of one block-connected rate network
        dict(name="rate_batch_64", kind="rate_batch", copies=64, n_in=500, n_out=6000, density=0.08,
             steps=50),
        # the 4000-neuron conductance-based spiking network, 100 ms stretches
        # with spike recording: double precision (default) and single
        dict(name="coba_4000_double", kind="coba", n=4000, p=0.02, precision="double",
             delays="none", steps=1000),
        dict(name="coba_4000_float", kind="coba", n=4000, p=0.02, precision="float",
             delays="none", steps=400),
        # the same family with a delay per synapse (0.1 to 2 ms)
        dict(name="coba_3000_delays", kind="coba", n=3000, p=0.02, precision="double",
             delays="synapse", steps=200),
        # spike-timing dependent plasticity: simulate, then fetch the weights
        dict(name="stdp_10000_double", kind="stdp", n=10001, fan=100, precision="double", steps=500),
        dict(name="stdp_20000_float", kind="stdp", n=20000, fan=80, precision="float", steps=500),
        # a large static spiking network, connectivity generated on the device
        dict(name="large_100k_double", kind="large", n=100000, fan_e=400, fan_i=100,
             precision="double", weights="", steps=200),
        # a parameter sweep: spiking networks of uneven sizes in one batch
        dict(name="sweep_96_float", kind="sweep", count=96, n_min=400, n_max=2800,
             precision="float", steps=500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rate", "rate", "rate", "rate_batch", "coba", "coba", "coba", "stdp", "stdp",
                       "large", "sweep"])
    precision = rng.choice(["double", "float"])
    if kind == "rate":
        n = _log(rng, 100, 20000)
        fan = _log(rng, 10, 150)
        n_in = _log(rng, 50, 2000)
        storage = "auto" if precision == "float" and n > 8000 else rng.choice(["csr", "csr", "ell"])
        return dict(kind="rate", n_in=n_in, n_out=n, p_in=min(0.5, fan / n_in / 2),
                    p_rec=min(0.3, fan / n), precision=precision, storage=storage,
                    steps=_log(rng, 10, 200), record=rng.choice([0, 0, 10]))
    if kind == "rate_batch":
        return dict(kind="rate_batch", copies=rng.choice([16, 48, 64, 112, 128, 256]),
                    n_in=_log(rng, 64, 1000), n_out=_log(rng, 1000, 6000),
                    density=round(rng.uniform(0.02, 0.1), 4), steps=_log(rng, 10, 60))
    if kind == "coba":
        n = _log(rng, 300, 5000)
        delays = rng.choice(["none", "none", "uniform", "synapse"])
        return dict(kind="coba", n=n, p=min(0.1, 80.0 / n), precision=precision, delays=delays,
                    steps=_log(rng, 50, 400 if precision == "float" or delays != "none" else 1000))
    if kind == "stdp":
        return dict(kind="stdp", n=_log(rng, 400, 15000), fan=_log(rng, 20, 100), precision=precision,
                    steps=_log(rng, 50, 400))
    if kind == "large":
        n = _log(rng, 20000, 100000)
        return dict(kind="large", n=n, fan_e=4 * _log(rng, 25, 100), fan_i=_log(rng, 25, 100),
                    precision=precision,
                    weights=rng.choice(["float32", "bfloat16"]) if precision == "float" else "",
                    steps=_log(rng, 50, 200))
    n_min = _log(rng, 200, 800)
    return dict(kind="sweep", count=rng.randint(8, 48), n_min=n_min, n_max=3 * n_min,
                precision=precision, steps=_log(rng, 100, 400))


# -- inputs ------------------------------------------------------------------------

def _rate_inputs(c, seed):
    rng = np.random.default_rng(seed)
    n_in, n = c["n_in"], c["n_out"]
    w_in = wl.bernoulli_csr_skip(rng, n, n_in, c["p_in"], lambda k: rng.normal(0.02, 0.05, k))
    w_rec = wl.bernoulli_csr_skip(rng, n, n, c["p_rec"], lambda k: rng.normal(0.0, 0.02, k))
    return wl.RateNet(n_in, n, w_in, w_rec, rng.uniform(0.0, 1.0, n_in))


def _batch_inputs(c, seed):
    """Input weights on all pairs with probability 0.1; recurrent weights in
    dense 64 x 64 blocks; one input vector per copy."""
    rng = np.random.default_rng(seed)
    n_in, n = c["n_in"], c["n_out"]
    w_in = wl.bernoulli_csr_skip(rng, n, n_in, 0.1, lambda k: rng.normal(0.02, 0.05, k))
    nb = -(-n // 64)
    mask = rng.random((nb, nb)) < c["density"]
    mask[np.arange(nb), np.arange(nb)] = True
    indptr = np.zeros(n + 1, dtype=np.int64)
    cols = []
    for b in range(nb):
        k = (np.nonzero(mask[b])[0][:, None] * 64 + np.arange(64)).ravel()
        k = k[k < n]
        rows = min(64, n - 64 * b)
        indptr[64 * b + 1:64 * b + 1 + rows] = k.size
        cols.append(np.tile(k, rows))
    np.cumsum(indptr, out=indptr)
    cols = np.concatenate(cols)
    w_rec = type(w_in)((rng.normal(0.0, 0.01, cols.size), cols, indptr), shape=(n, n))
    return w_in, w_rec, rng.uniform(0.0, 1.0, (c["copies"], n_in))


def _coba_inputs(c, seed):
    cn = wl.coba_net(seed=seed, n=c["n"], p=c["p"], steps=c["steps"], skip=True)
    rng = np.random.default_rng(seed + 1)
    if c["delays"] == "uniform":
        d = (int(rng.integers(2, 20)), int(rng.integers(2, 20)))
    elif c["delays"] == "synapse":
        d = (rng.integers(1, 21, cn.w_exc.nnz), rng.integers(1, 21, cn.w_inh.nnz))
    else:
        d = (None, None)
    return cn, d


def _stdp_inputs(c, seed):
    n = c["n"]
    cn = wl.coba_net(seed=seed, n=n, p=c["fan"] / (0.8 * n), w_exc=0.6 * 64 / c["fan"],
                     w_inh=6.7 * 16 * 4 / c["fan"], steps=c["steps"], skip=True)
    rng = np.random.default_rng(seed + 1)
    # plastic synapses: `fan` per neuron, one from each of `fan` equal ranges
    ne, fan = cn.n_exc, c["fan"]
    lo = np.arange(fan + 1) * ne // fan
    cols = rng.integers(lo[:-1], lo[1:], (ne, fan))
    w_ee = type(cn.w_exc)((rng.uniform(0.0, 0.5, ne * fan), cols.ravel(), np.arange(ne + 1) * fan),
                          shape=(ne, ne))
    return cn, w_ee


def _sweep_inputs(c, seed):
    rng = np.random.default_rng(seed)
    nets = []
    for i, n in enumerate(np.linspace(c["n_min"], c["n_max"], c["count"]).astype(int).tolist()):
        nets.append(wl.coba_net(seed=seed + i, n=n, p=min(0.1, 60.0 / n),
                                w_exc=float(rng.uniform(0.3, 0.9)), w_inh=float(rng.uniform(3.0, 9.0)),
                                steps=c["steps"], skip=True))
    return nets


# -- what a program has in hand before the call ----------------------------------------

def prepare(case, seed):
    c = dict(case, seed=seed)
    k = c["kind"]
    if k == "rate":
        rn = _rate_inputs(c, seed)
        net = ann.Network(dt=1.0, seed=seed)
        net.config(precision=c["precision"])
        inp = net.create(rn.n_in, ann.Neuron(parameters="r = 0.0"))
        pop = net.create(rn.n_out, ann.Neuron(parameters=dict(tau=rn.tau),
                                              equations="tau*dr/dt + r = sum(exc) : min=0.0"))
        net.connect(inp, pop, "exc").from_sparse(wl.to_from_sparse(rn.w_in), storage_format="csr")
        net.connect(pop, pop, "exc").from_sparse(wl.to_from_sparse(rn.w_rec),
                                                 storage_format=c["storage"])
        mon = net.monitor(pop, "r", period=float(c["record"])) if c["record"] else None
        net.compile()
        return dict(c=c, net=net, inp=inp, pop=pop, mon=mon, x=rn.r_in)
    if k == "rate_batch":
        w_in, w_rec, x = _batch_inputs(c, seed)
        tpl = ann.Network(dt=1.0, seed=seed)
        inp = tpl.create(c["n_in"], ann.Neuron(parameters="r = 0.0"))
        pop = tpl.create(c["n_out"], ann.Neuron(parameters="tau = 10.0",
                                                equations="tau*dr/dt + r = sum(exc) : min=0.0"))
        tpl.connect(inp, pop, "exc").from_sparse(wl.to_from_sparse(w_in))
        tpl.connect(pop, pop, "exc").from_sparse(wl.to_from_sparse(w_rec))
        rb = ann.RateBatch(tpl, batch=c["copies"]).compile()
        return dict(c=c, net=rb, inp=inp, pop=pop, x=x)
    if k == "coba":
        cn, d = _coba_inputs(c, seed)
        net, pop, mon = wl.build_coba_network(cn, precision=c["precision"], delays=d)
        net.compile()
        return dict(c=c, net=net, pop=pop, mon=mon)
    if k == "stdp":
        cn, w_ee = _stdp_inputs(c, seed)
        net, pop, mon = wl.build_coba_network(cn, precision=c["precision"], stdp_w_ee=w_ee)
        net.compile()
        return dict(c=c, net=net, pop=pop, mon=mon, proj=net.projections[0])
    if k == "large":
        ln = wl.LargeNet(n=c["n"], fan_e=c["fan_e"], fan_i=c["fan_i"], w_exc=0.6 * 64 / c["fan_e"],
                         w_inh=6.7 * 16 / c["fan_i"], seed=seed)
        kw = {"weight_dtype": c["weights"]} if c["weights"] else {}
        net, pop, mon, _ = wl.build_large_network(ln, precision=c["precision"], stdp=False, **kw)
        net.compile()
        return dict(c=c, net=net, pop=pop, mon=mon)
    nets = _sweep_inputs(c, seed)
    members = [wl.build_coba_network(cn, "double", "grid") for cn in nets]
    batch = Batch([m[0] for m in members], precision=c["precision"])
    batch.compile()
    return dict(c=c, net=batch, members=members)


def _own(c, a):
    return np.asarray(a, dtype=np.float64 if c.get("precision") == "double" else np.float32)


def _counts(steps, ranks, first, nsteps, n):
    """Spikes per neuron and spikes per step."""
    return [np.bincount(ranks, minlength=n), np.bincount(steps - first, minlength=nsteps)]


def _spikes(mon, first, nsteps):
    """The recorded spikes, handed over and counted."""
    steps, ranks = mon.spike_arrays()
    mon.reset()
    return _counts(steps, ranks, first, nsteps, mon.population.size)


def run(state):
    c, net = state["c"], state["net"]
    k = c["kind"]
    if k == "rate":
        state["inp"].r = state["x"]
        net.simulate(float(c["steps"]))
        out = [_own(c, state["pop"].r)]
        if state["mon"] is not None:
            out.append(_own(c, state["mon"].get("r")))
        return out
    if k == "rate_batch":
        net.set(state["inp"], "r", state["x"])
        net.simulate(float(c["steps"]))
        return _own(c, net.get(state["pop"], "r"))
    first = net.current_step
    net.simulate_steps(c["steps"])
    if k == "sweep":
        got = [[_own(c, p.v), *_spikes(m, first, c["steps"])] for _, p, m in state["members"]]
        return [np.concatenate(a) for a in zip(*got)]
    pop = state["pop"]
    out = [_own(c, pop.v), _own(c, pop.g_exc), _own(c, pop.g_inh),
           *_spikes(state["mon"], first, c["steps"])]
    if k == "stdp":
        out.append(_own(c, state["proj"].get("w", flat=True)))
    return out


# -- the work of one pass -------------------------------------------------------------

def work(case):
    """Inputs (connectivity and state) read once, state and results written
    once; the additions and multiplications of every step. Spikes are taken
    at 20 per neuron and second (10 in the large networks)."""
    c = case
    k, steps = c["kind"], c["steps"]
    fb = 8 if c.get("precision", "float") == "double" else 4
    if k == "rate":
        nnz = c["p_in"] * c["n_in"] * c["n_out"] + c["p_rec"] * c["n_out"] ** 2
        rec = steps // c["record"] * c["n_out"] if c["record"] else 0
        return dict(bytes=nnz * (4 + fb) + c["n_in"] * fb + c["n_out"] * 2 * fb + rec * 8,
                    flops=steps * (2 * nnz + 4 * c["n_out"]))
    if k == "rate_batch":
        b, n = c["copies"], c["n_out"]
        w = 0.1 * c["n_in"] * n + (c["density"] + 64.0 / n) * n * n
        return dict(bytes=2 * w + 4 * b * (c["n_in"] + 2 * n), flops=steps * b * (2 * w + 4 * n))
    dt, rate = 1e-4, 20.0
    if k == "coba":
        n, fan = c["n"], c["p"] * c["n"]
    elif k == "stdp":
        n, fan = c["n"], 1.25 * c["fan"]
    elif k == "large":
        n, fan, rate = c["n"], c["fan_e"] + c["fan_i"], 10.0
    else:
        n, fan = c["count"] * 0.5 * (c["n_min"] + c["n_max"]), 60.0
    events = rate * dt * steps * n * fan
    wb = 2 if c.get("weights") == "bfloat16" else fb
    syn = min(events, n * fan) * (4 + wb)          # synapses no spike reaches are not read
    if k == "stdp":
        syn = n * fan * (4 + 4 * wb + wb)
    return dict(bytes=syn + n * (10 * fb + 8) + rate * dt * steps * n * 16,
                flops=events * (12 if k == "stdp" else 1) + steps * n * 20)


# -- the same in 64 bits, plain numpy ------------------------------------------------------

def _csc(m):
    """(pointers, post ranks, positions in the CSR arrays) by pre rank."""
    rows = np.repeat(np.arange(m.shape[0]), np.diff(m.indptr))
    order = np.argsort(m.indices, kind="stable")
    ptr = np.zeros(m.shape[1] + 1, dtype=np.int64)
    np.cumsum(np.bincount(m.indices, minlength=m.shape[1]), out=ptr[1:])
    return ptr, rows[order], order


def _ranges(ptr, idx):
    """Concatenated index ranges ptr[i]..ptr[i+1] of the given rows."""
    n = ptr[idx + 1] - ptr[idx]
    if n.sum() == 0:
        return np.zeros(0, dtype=np.int64)
    return np.repeat(ptr[idx] - np.concatenate(([0], np.cumsum(n)[:-1])), n) + np.arange(n.sum())


def _exact_rate(w_in, w_rec, x, steps, record, n):
    dense = x.ndim == 2
    x = x.T if dense else x
    r = np.zeros((n,) + x.shape[1:])
    drive = w_in @ x
    rec = []
    for t in range(steps):
        r = np.maximum(r + (drive + w_rec @ r - r) / 10.0, 0.0)
        if record and t % record == 0:
            rec.append(r.copy())
    return (r.T if dense else r), np.array(rec)


def _exact_spiking(cn, steps, delays=(None, None), w_ee=None):
    """Euler steps of the spiking network: transmissions, update, spikes;
    with w_ee the excitatory-excitatory synapses are plastic."""
    p, n, ne = cn.params, cn.n, cn.n_exc
    parts = [(cn.w_exc if w_ee is None else cn.w_exc[ne:], 0, 0, 0 if w_ee is None else ne, delays[0]),
             (cn.w_inh, ne, 1, 0, delays[1])]
    parts = [(_csc(m), m.data, lo, tgt, off, d) for m, lo, tgt, off, d in parts]
    v, g, ref = cn.v0.copy(), [np.zeros(n), np.zeros(n)], np.zeros(n, dtype=np.int64)
    slots = 32
    queue = [[np.zeros(n), np.zeros(n)] for _ in range(slots)]
    spiked = np.zeros(0, dtype=np.int64)
    st, sr = [], []
    s = dict(wl.STDP_PARAMS)
    if w_ee is not None:
        ptr, posts, pos = _csc(w_ee)
        row_ptr = w_ee.indptr.astype(np.int64)
        w = w_ee.data.copy()
        x, y, last = np.zeros(w.size), np.zeros(w.size), np.full(w.size, -10000)

        def decay(j, t):
            gap = (last[j] - t) * cn.dt
            x[j] *= np.exp(gap / s["tau_plus"])
            y[j] *= np.exp(gap / s["tau_minus"])

    for t in range(steps):
        now = queue[t % slots]
        for (cptr, cpost, cpos), data, lo, tgt, off, d in parts:
            mine = spiked[(spiked >= lo) & (spiked < lo + cptr.size - 1)] - lo
            q = _ranges(cptr, mine)
            if d is None or np.ndim(d) == 0:
                late = 0 if d is None else d - 1
                np.add.at(queue[(t + late) % slots][tgt], cpost[q] + off, data[cpos[q]])
            else:
                late = np.asarray(d)[cpos[q]] - 1
                for k in np.unique(late):
                    u = q[late == k]
                    np.add.at(queue[(t + k) % slots][tgt], cpost[u] + off, data[cpos[u]])
        if w_ee is not None:
            q = _ranges(ptr, spiked[spiked < ne])
            j = pos[q]
            np.add.at(now[0], posts[q], w[j])
            decay(j, t - 1)
            last[j] = t
            x[j] += s["A_plus"] * s["w_max"]
            w[j] = np.clip(w[j] + y[j], s["w_min"], s["w_max"])
        g[0] += now[0]
        g[1] += now[1]
        now[0][:] = 0.0
        now[1][:] = 0.0
        free = ref <= 0
        dv = ((p["El"] - v) + g[0] * (p["Erev_exc"] - v) + g[1] * (p["Erev_inh"] - v) + p["I"]) / p["tau"]
        dg = -g[0] / p["tau_exc"], -g[1] / p["tau_inh"]
        v = v + cn.dt * dv * free
        g = [g[0] + cn.dt * dg[0], g[1] + cn.dt * dg[1]]
        ref -= ~free
        spiked = np.nonzero(free & (v > p["Vt"]))[0]
        v[spiked] = p["Vr"]
        ref[spiked] = int(round(cn.refractory / cn.dt))
        st.append(np.full(spiked.size, t))
        sr.append(spiked)
        if w_ee is not None:
            j = _ranges(row_ptr, spiked[spiked < ne])
            decay(j, t)
            last[j] = t
            y[j] -= s["A_minus"] * s["w_max"]
            w[j] = np.clip(w[j] + x[j], s["w_min"], s["w_max"])
    out = [v, g[0], g[1], *_counts(np.concatenate(st), np.concatenate(sr), 0, steps, n)]
    return out + ([w] if w_ee is not None else [])


def exact(case, seed):
    c = dict(case)
    k = c["kind"]
    if k == "rate":
        rn = _rate_inputs(c, seed)
        r, rec = _exact_rate(rn.w_in, rn.w_rec, rn.r_in, c["steps"], c["record"], c["n_out"])
        return [r, rec] if c["record"] else [r]
    if k == "rate_batch":
        w_in, w_rec, x = _batch_inputs(c, seed)
        if w_rec.nnz * c["copies"] * c["steps"] > 1.2e10:
            return None                    # the products would take over 20 seconds
        return _exact_rate(w_in, w_rec, x, c["steps"], 0, c["n_out"])[0]
    if k == "coba":
        cn, d = _coba_inputs(c, seed)
        return _exact_spiking(cn, c["steps"], d)
    if k == "stdp":
        cn, w_ee = _stdp_inputs(c, seed)
        return _exact_spiking(cn, c["steps"], w_ee=w_ee)
    if k == "large":
        return None                        # connectivity generated on the device
    nets = _sweep_inputs(c, seed)
    got = [_exact_spiking(cn, c["steps"]) for cn in nets]
    return [np.concatenate([o[i] for o in got]) for i in (0, 3, 4)]
