"""The work a user of the simulator has it do, as cases with sizes, inputs and results.

Every case goes through the package's public classes (Simulation, Ensemble, Server)
and returns what such a program reads back: spike counts, state arrays, rasters,
calcium samples, connectivity, summaries.  Five kinds of work:

  step      a network in hand is advanced by `ms` of biological time and read
  delays    the same with unequal synaptic delays (the per-step engine)
  job       one whole run: build the network, pre-run and recorded run, read, free
  ensemble  one whole batch of networks of uneven size, built, run and summarised
  serve     a request loop that is handed a burst of runs and works it off

`exact` restates the model in NumPy (FP64) for the networks small enough for it.
"""
import math
import random

import numpy as np

import astrosimgpu_cuda_b200 as asg
from astrosimgpu_cuda_b200 import abi


def listed():
    return [
        # The smallest network in real use (500 cells, the plain method): each millisecond
        # is a launch or two, so latency decides.
        dict(name="step_500_fp64", kind="step", n=500, precision="fp64", ms=100, dt=0.1, substeps=1, drive=1.0),
        # A parameter-study network, ragged size, background drive off its default.
        dict(name="step_5003_fp32", kind="step", n=5003, precision="fp32", ms=100, dt=0.1, substeps=1, drive=1.2),
        # Middle size: enough cells to fill part of the chip.
        dict(name="step_100k_fp32", kind="step", n=100003, precision="fp32", ms=100, dt=0.1, substeps=1, drive=1.0),
        # The one-million-cell configuration in the default precision.
        dict(name="step_1m_fp64", kind="step", n=1_000_000, precision="fp64", ms=50, dt=0.1, substeps=1, drive=1.0),
        # The headline size, FP32 stages: throughput of the resident network.
        dict(name="step_10m_fp32", kind="step", n=10_000_000, precision="fp32", ms=100, dt=0.1, substeps=1,
             drive=1.0),
        # Two RK4 substeps with calcium recorded every millisecond.
        dict(name="record_50k_fp64", kind="step", n=50_000, precision="fp64", ms=100, dt=0.1, substeps=2, drive=1.0,
             record=True),
        # Unequal delays, which the windowed engine does not take.
        dict(name="delays_20k_fp64", kind="delays", n=20_011, precision="fp64", ms=50, dt=0.1, substeps=1,
             drive=1.0),
        # A small run from configuration to result, with raster and connectivity read back
        # (the command-line default size).
        dict(name="job_1000_fp64", kind="job", n=1000, precision="fp64", pre_ms=20, ms=80, dt=0.1, raster=True),
        # A middle-sized run, ragged size.
        dict(name="job_300k_fp32", kind="job", n=300_007, precision="fp32", pre_ms=10, ms=90, dt=0.1, raster=False),
        # The headline network from configuration to result: the build dominates.
        dict(name="job_10m_fp32", kind="job", n=10_000_000, precision="fp32", pre_ms=10, ms=40, dt=0.1,
             raster=False),
        # A batch: sizes spread log-uniformly, as in a parameter sweep.
        dict(name="ensemble_48_fp32", kind="ensemble", networks=48, lo=500, hi=50_000, precision="fp32", ms=300),
        # Served requests of the served distribution's sizes, in one burst.
        dict(name="serve_24_fp32", kind="serve", requests=24, lo=1000, hi=200_000, precision="fp32", ms=100),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "delays", "job", "job", "ensemble", "serve"])
    precision = rng.choice(["fp32", "fp64"])
    drive = rng.uniform(0.8, 1.2)
    dt = rng.choice([0.1, 0.1, 0.1, 0.2])
    if kind == "step":
        n = _log_size(rng, 300, 5_000_000)
        return dict(kind="step", n=n, precision=precision, ms=100 if n < 500_000 else 50, dt=dt,
                    substeps=rng.choice([1, 1, 2]), drive=drive, record=rng.random() < 0.25)
    if kind == "delays":
        return dict(kind="delays", n=_log_size(rng, 300, 200_000), precision=precision, ms=30, dt=dt, substeps=1,
                    drive=drive)
    if kind == "job":
        n = _log_size(rng, 300, 5_000_000)
        return dict(kind="job", n=n, precision=precision, pre_ms=rng.choice([0, 10, 20]),
                    ms=80 if n < 500_000 else 30, dt=dt, raster=n < 20_000)
    if kind == "ensemble":
        return dict(kind="ensemble", networks=rng.randrange(3, 48), lo=500, hi=_log_size(rng, 2000, 50_000),
                    precision=precision, ms=rng.randrange(50, 250))
    return dict(kind="serve", requests=rng.randrange(2, 24), lo=1000, hi=_log_size(rng, 5000, 200_000),
                precision=precision, ms=rng.randrange(30, 100))


# ------------------------------------------------------------------ configurations

def _spread(case, count):
    """`count` sizes spread evenly in the logarithm over [lo, hi], odd ones among them."""
    r = math.log(case["hi"] / case["lo"]) / max(1, count - 1)
    return [int(round(case["lo"] * math.exp(r * i))) for i in range(count)]


def _configs(case, seed):
    """The runs of a batch: distinct seeds, drive and a2n weight within 20 % of the defaults."""
    rng = random.Random(seed)
    count = case["networks"] if case["kind"] == "ensemble" else case["requests"]
    out = []
    for i, n in enumerate(_spread(case, count)):
        ms = case["ms"]
        if case["kind"] == "serve":
            ms = case["ms"] * (1 + i % 3)  # requests of uneven length leave the batch at different times
        kw = dict(n_total=n, seed=rng.getrandbits(40) + 1, pre_ms=0.0, sim_ms=float(ms), precision=case["precision"],
                  neuron_drive_scale=rng.uniform(0.8, 1.2))
        if case["kind"] == "ensemble":
            kw["w_a2n"] = rng.uniform(0.8, 1.2)
        out.append(kw)
    rng.shuffle(out)
    return out


def _single(case, seed):
    """Configuration and biology of a case with one network."""
    rng = random.Random(seed)
    pre = float(case.get("pre_ms", 0))
    kw = dict(n_total=case["n"], seed=rng.getrandbits(40) + 1, pre_ms=pre, sim_ms=float(case["ms"]), dt=case["dt"],
              substeps=case.get("substeps", 1), precision=case["precision"],
              neuron_drive_scale=case.get("drive", 1.0))
    if case.get("raster"):
        kw["raster_steps"] = _steps(case)
    biology = {"d_e": 1.0, "d_i": 0.6, "d_a2n": 1.4} if case["kind"] == "delays" else None
    return kw, biology


def _steps(case):
    return int(round((case.get("pre_ms", 0) + case["ms"]) / case.get("dt", 0.1)))


# ------------------------------------------------------------------ one pass

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "delays"):
        kw, biology = _single(case, seed)
        return dict(kind=kind, sim=asg.Simulation(biology=biology, **kw), steps=_steps(case), done=0,
                    record=bool(case.get("record")), every=max(1, int(round(1.0 / case["dt"]))))
    if kind == "job":
        kw, _ = _single(case, seed)
        return dict(kind=kind, cfg=kw, steps=_steps(case), raster=bool(case.get("raster")))
    cfgs = _configs(case, seed)
    if kind == "ensemble":
        return dict(kind=kind, cfgs=cfgs, steps=_steps(case))
    return dict(kind=kind, cfgs=cfgs, server=asg.Server(precision=case["precision"]))


_COUNTED = ("n_exc_edges", "n_inh_edges", "n_e2a_edges", "n_sic_edges", "spikes_total", "spikes_measured",
            "active_astro", "engaged_astro")
_MEASURED = ("mean_rate_hz", "mean_ca")


def _table(summaries):
    return {"counted": np.array([[s[k] for k in _COUNTED] for s in summaries], dtype=np.int64),
            "measured": np.array([[s[k] for k in _MEASURED] for s in summaries], dtype=np.float64)}


def run(state):
    kind = state["kind"]
    if kind in ("step", "delays"):
        sim, n = state["sim"], state["steps"]
        if state["record"]:
            sim.record_calcium(state["every"], max_samples=n // state["every"])
        sim.step(n)
        out = {"counts": sim.spike_counts(state["done"], n), "V": sim.state("V"), "Ca": sim.state("Ca")}
        if state["record"]:
            out["recorded"] = sim.calcium()
        state["done"] += n
        return out
    if kind == "job":
        with asg.Simulation(**state["cfg"]) as sim:
            sim.step(state["steps"])
            out = {"summary": _table([sim.summary()]), "counts": sim.spike_counts(0, state["steps"]),
                   "V": sim.state("V"), "Ca": sim.state("Ca")}
            if state["raster"]:
                out["raster"] = sim.raster()
                out["exc_rows"] = sim.csr("exc")[0]
        return out
    if kind == "ensemble":
        with asg.Ensemble([abi.default_config(**kw) for kw in state["cfgs"]]) as ens:
            ens.step(state["steps"])
            return _table([ens.summary(i) for i in range(len(ens))])
    server = state["server"]
    ids = [server.submit(**kw) for kw in _request_fields(state["cfgs"])]
    results = [None] * len(ids)
    while any(r is None for r in results):
        server.pump(10)
        results = [r if r is not None else server.result(i) for i, r in zip(ids, results)]
    return _table(results)


def _request_fields(cfgs):
    """A request takes its precision from the server."""
    return [{k: v for k, v in kw.items() if k != "precision"} for kw in cfgs]


# ------------------------------------------------------------------ what a pass cannot do without

# Arithmetic of one cell and time step, counted from the model: an AdEx neuron's four
# right-hand sides, its conductance cascade and its Poisson draw; an astrocyte's four
# Li-Rinzel right-hand sides, its Poisson draw and its Gaussian draw.
_NEURON_FLOPS, _ASTRO_FLOPS = 130.0, 220.0


def _cells(n):
    n_exc, n_inh, n_astro, _ = asg.scaling(n)
    return n_exc + n_inh, n_astro


def _network_work(n, steps, substeps, precision, built):
    """One network over `steps` steps: its state read and written once, its flops, and
    its connectivity written once when it is built (about 132 edges a neuron)."""
    r = 8 if precision == "fp64" else 4
    neurons, astros = _cells(n)
    # V, w, stp time, refractory count and two parameters; seven values in the stage type
    state = neurons * (2 * (8 + 8 + 8 + 4 + 7 * r) + 16) + astros * (2 * (16 + r) + 32)
    flops = steps * substeps * (neurons * _NEURON_FLOPS + astros * _ASTRO_FLOPS)
    return state + (132.0 * neurons * 4 if built else 0.0), flops


def work(case):
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        count = case["networks"] if kind == "ensemble" else case["requests"]
        nets = [(n, int(case["ms"] * 10 * (1 + (i % 3 if kind == "serve" else 0))))
                for i, n in enumerate(_spread(case, count))]
        parts = [_network_work(n, s, 1, case["precision"], True) for n, s in nets]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    steps = _steps(case)
    b, f = _network_work(case["n"], steps, case.get("substeps", 1), case["precision"], kind == "job")
    neurons, astros = _cells(case["n"])
    b += 8.0 * (neurons + astros) + 4 * steps
    if case.get("record"):
        b += 8.0 * astros * case["ms"]
    if case.get("raster"):
        b += neurons / 8 * steps + 4 * 80.0 * neurons
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ the model in FP64 NumPy

_EXACT_CELL_STEPS = 6e6  # about ten seconds


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        cfgs = _configs(case, seed)
        if sum(kw["n_total"] * kw["sim_ms"] * 10 for kw in cfgs) > _EXACT_CELL_STEPS:
            return None
        return _table([_Model(kw, None).run(int(round(kw["sim_ms"] * 10))).summary() for kw in cfgs])
    if case["n"] * _steps(case) * case.get("substeps", 1) > _EXACT_CELL_STEPS:
        return None
    kw, biology = _single(case, seed)
    m = _Model(kw, biology)
    every = max(1, int(round(1.0 / case["dt"]))) if case.get("record") else 0
    m.run(_steps(case), every, bool(case.get("raster")))
    out = {"counts": np.array(m.counts, dtype=np.uint32), "V": m.V, "Ca": m.Ca}
    if case.get("record"):
        out["recorded"] = np.array(m.recorded)
    if kind == "job":
        out["summary"] = _table([m.summary()])
        if case.get("raster"):
            out["raster"] = np.array(m.raster, dtype=np.uint32)
            out["exc_rows"] = m.exc[0]
    return out


_M64 = (1 << 64) - 1


def _mix(z):
    with np.errstate(over="ignore"):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _uniform(seed, stream, counter):
    """53-bit uniform of (seed, stream, counter); stream or counter is an array."""
    with np.errstate(over="ignore"):
        z = (np.uint64(seed & _M64) + np.asarray(stream, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
             + np.asarray(counter, dtype=np.uint64) * np.uint64(0xBF58476D1CE4E5B9))
    return (_mix(z) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _normal(seed, stream):
    u1 = np.maximum(_uniform(seed, stream, 0), 1e-300)
    return np.sqrt(-2.0 * np.log(u1)) * np.cos(2.0 * np.pi * _uniform(seed, stream, 1))


def _poisson(seed, stream, lam):
    limit = math.exp(-lam)
    count = np.zeros(stream.shape, dtype=np.float64)
    product = _uniform(seed, stream, 0)
    live = np.flatnonzero(product > limit)
    c = 1
    while live.size:
        count[live] += 1
        product[live] *= _uniform(seed, stream[live], c)
        live = live[product[live] > limit]
        c += 1
    return count


class _Stream:
    """The set-up stream (seed, 0x5EED) read in order."""

    def __init__(self, seed):
        self.seed, self.at, self.block = seed, 0, np.empty(0)
        self.first = 0
        self.spare = None

    def _fill(self):
        self.first = self.at
        self.block = _uniform(self.seed, 0x5EED, np.arange(self.at, self.at + (1 << 16), dtype=np.uint64)).tolist()

    def uniform(self):
        k = self.at - self.first
        if k >= len(self.block):
            self._fill()
            k = 0
        self.at += 1
        return self.block[k]

    def normal(self):
        if self.spare is not None:
            v, self.spare = self.spare, None
            return v
        u1 = self.uniform()
        while u1 <= 1e-300:
            u1 = self.uniform()
        th, r = 2.0 * math.pi * self.uniform(), math.sqrt(-2.0 * math.log(u1))
        self.spare = r * math.sin(th)
        return r * math.cos(th)

    def scaled(self, mean, lower, upper, var):
        lo, hi = sorted((mean * lower, mean * upper))
        for _ in range(1000):
            v = mean + var * abs(mean) * self.normal()
            if lo <= v <= hi:
                return v
        return min(max(mean, lo), hi)


def _rows(edges, n_targets):
    """Target-keyed rows of (source, target) pairs, sources in emission order."""
    e = np.array(edges, dtype=np.int64).reshape(-1, 2)
    order = np.argsort(e[:, 1], kind="stable")
    start = np.zeros(n_targets + 1, dtype=np.uint32)
    start[1:] = np.cumsum(np.bincount(e[:, 1], minlength=n_targets))
    return start, e[order, 0].astype(np.uint32)


class _Population:
    def __init__(self, exc):
        (self.a, self.tau_w, self.V_reset, self.b, self.V0, self.C, self.gL, self.EL, self.Vth) = (
            (4.0, 450.0, -50.0, 300.0, -50.0, 130.0, 18.0, -58.0, -50.0) if exc else
            (-0.8, 264.0, -60.0, 130.0, -60.0, 104.0, 4.3, -65.0, -52.0))
        self.rate = 2700.0 if exc else 2500.0


class _Model:
    """Tripartite AdEx and Li-Rinzel network with its default biology, one step at a time."""

    def __init__(self, kw, biology):
        self.seed, self.dt = kw["seed"], kw.get("dt", 0.1)
        self.sub, self.sim_ms = kw.get("substeps", 1), kw["sim_ms"]
        self.pre = int(kw["pre_ms"] / self.dt + 0.5)
        self.w_a2n = kw.get("w_a2n", 1.0)
        n = kw["n_total"]
        self.nE, self.nI, self.nA, p = asg.scaling(n)
        self.nN = self.nE + self.nI
        delay = {"d_e": 1.0, "d_i": 1.0, "d_a2n": 1.0, **(biology or {})}
        self.d_e, self.d_i, self.d_a = (max(1, int(delay[k] / self.dt + 0.5)) for k in ("d_e", "d_i", "d_a2n"))
        pops = (_Population(True), _Population(False))
        nE, nN, nA = self.nE, self.nN, self.nA
        is_exc = np.arange(nN) < nE
        for name in ("a", "tau_w", "C", "gL", "EL", "Vth", "V0"):
            setattr(self, name, np.where(is_exc, getattr(pops[0], name), getattr(pops[1], name)))
        self.lam = [pp.rate * kw["neuron_drive_scale"] * self.dt * 1e-3 for pp in pops]
        self._connect(p)
        rs = _Stream(self.seed)
        means = (1.8958264782990153, 0.010925583871830699, 1058.7589568400845, 0.04911592657233997)
        self.Ct, self.I0, self.tau, self.dI = np.array(
            [[rs.scaled(m, 0.9, 1.05, 0.1) for m in means] for _ in range(nA)]).T
        self.V_reset, self.b = np.array(
            [[rs.scaled(m, 0.9, 1.1, 0.05) for m in (q.V_reset, q.b)]
             for q in (pops[0 if j < nE else 1] for j in range(nN))]).T
        self.V = self.V0.copy()
        self.w, self.gx, self.dgx, self.gi, self.dgi, self.sic = (np.zeros(nN) for _ in range(6))
        self.x, self.t_last = np.ones(nN), np.full(nN, -1e12)
        self.Ca, self.IP3, self.h = np.full(nA, 0.073), np.full(nA, 0.010925583871830699), np.full(nA, 0.793)
        self.slots = max(self.d_e, self.d_i, self.d_a) + 1
        self.ring, self.ring_s = np.zeros((self.slots, nN)), np.zeros((self.slots, nA))
        self.engaged = np.zeros(nA, dtype=bool)
        self.counts, self.raster, self.recorded, self.t = [], [], [], 0

    def _connect(self, p):
        nE, nN, nA, nI = self.nE, self.nN, self.nA, self.nI
        rs = _Stream(self.seed)
        for _ in range(4 * nA + 2 * nN):
            rs.normal()
        rs.spare = None
        take = min(5, nA)
        pools = []
        for _ in range(nN):
            if take * 4 >= nA:
                cand = list(range(nA))
                for k in range(take):
                    i = min(int(rs.uniform() * (nA - k)) + k, nA - 1)
                    cand[k], cand[i] = cand[i], cand[k]
                pools.append(cand[:take])
            else:
                pool = []
                while len(pool) < take:
                    c = int(rs.uniform() * nA) % nA
                    if c not in pool:
                        pool.append(c)
                pools.append(pool)
        log1mp = math.log1p(-p) if p < 1.0 else 0.0

        def landing(pos, end):
            if p >= 1.0:
                return pos
            return pos + min(math.floor(math.log1p(-rs.uniform()) / log1mp), end - pos)

        exc, inh, e2a, a2n, degree = [], [], [], [], [0] * nA
        for lo, hi in ((0, nE), (nE, nN)):
            for pre in range(nE):
                pos = landing(lo, hi)
                while pos < hi:
                    if pre != pos:
                        exc.append((pre, pos))
                        if rs.uniform() < 0.2:
                            a = pools[pos][int(rs.uniform() * take) % take]
                            if degree[a] < 10000:
                                e2a.append((pre, a))
                                a2n.append((a, pos))
                                degree[a] += 1
                    pos += 1
                    if pos < hi:
                        pos = landing(pos, hi)
        for pre in range(nI):
            pos = landing(0, nN)
            while pos < nN:
                if pre + nE != pos:
                    inh.append((pre, pos))
                pos += 1
                if pos < nN:
                    pos = landing(pos, nN)
        self.exc, self.inh = _rows(exc, nN), _rows(inh, nN)
        self.a2n, self.e2a = _rows(a2n, nN), _rows(e2a, nA)

    @staticmethod
    def _gather(rows, values):
        start, src = rows
        target = np.repeat(np.arange(start.size - 1), np.diff(start.astype(np.int64)))
        return np.bincount(target, weights=values[src], minlength=start.size - 1)

    def _neuron_rhs(self, V, w, gx, gi, ext):
        Vc = np.minimum(V, 0.0)
        dV = (-self.gL * (Vc - self.EL) + self.gL * 2.0 * np.exp((Vc - self.Vth) / 2.0) - gx * Vc - gi * (Vc + 85.0)
              - w + ext) / self.C
        return dV, (self.a * (Vc - self.EL) - w) / self.tau_w

    def _astro_rhs(self, Ca, IP3, h, noise):
        ratio = 0.185
        d = (self.Ct - Ca) / ratio - Ca
        m, n = IP3 / (IP3 + 0.13), Ca / (Ca + 0.08234)
        pump = 0.0009 * Ca * Ca / (0.1 * 0.1 + Ca * Ca)
        alpha = 0.0002 * 1.049 * (IP3 + 0.13) / (IP3 + 0.9434)
        return (ratio * 0.006 * (m * n * h) ** 3 * d - pump + ratio * 0.00011 * d + noise, (self.I0 - IP3) / self.tau,
                alpha * (1.0 - h) - 0.0002 * Ca * h)

    @staticmethod
    def _rk4(f, hs, y):
        k1 = f(*y)
        k2 = f(*(v + 0.5 * hs * k for v, k in zip(y, k1)))
        k3 = f(*(v + 0.5 * hs * k for v, k in zip(y, k2)))
        k4 = f(*(v + hs * k for v, k in zip(y, k3)))
        return [v + hs / 6.0 * (a + 2.0 * b + 2.0 * c + d) for v, a, b, c, d in zip(y, k1, k2, k3, k4)]

    def _astro_step(self):
        t, hs = self.t, self.dt / self.sub
        stream = np.uint64(t * 1000003) + np.arange(self.nA, dtype=np.uint64)
        kick = 0.2 * self._gather(self.e2a, self.ring[(t - self.d_e) % self.slots])
        kick += _poisson(self.seed ^ 0xC2B2AE3D27D4EB4F, stream, 3.029715502945856 * self.dt * 1e-3)
        noise = 0.0003 * _normal(self.seed ^ 0x9E3779B97F4A7C15, stream)
        self.IP3 = self.IP3 + self.dI * kick
        for _ in range(self.sub):
            Ca, IP3, h = self._rk4(lambda c, i, g: self._astro_rhs(c, i, g, noise), hs, (self.Ca, self.IP3, self.h))
            self.Ca, self.h, self.IP3 = np.clip(Ca, 0.0, self.Ct), np.clip(h, 0.0, 1.0), np.maximum(IP3, 0.0)
        y = (self.Ca - 0.19669) * 1000.0
        return np.where(y <= 1.0, 0.0, np.log(np.maximum(y, 1.0)))

    def _neuron_step(self):
        t, hs, nE = self.t, self.dt / self.sub, self.nE
        cell = np.arange(self.nN, dtype=np.uint64)
        stream = np.uint64(t * 1000003) + cell
        x_in = 5.0 * self._gather(self.exc, self.ring[(t - self.d_e) % self.slots])
        i_in = 5.0 * self._gather(self.inh, self.ring[(t - self.d_i) % self.slots])
        key = self.seed ^ 0x2545F4914F6CDD1D
        x_in[:nE] += _poisson(key, stream[:nE], self.lam[0])
        x_in[nE:] += _poisson(key, stream[nE:], self.lam[1])
        if t >= self.d_a:
            self.sic = self.w_a2n * self._gather(self.a2n, self.ring_s[(t - self.d_a) % self.slots])
        ext = self.sic + 100.0 * _normal(self.seed ^ 0x9E3779B185EBCA87, np.uint64(t // 10 * 1000033) + cell)
        ex, ix = math.exp(-hs / 0.2), math.exp(-hs / 2.0)
        gx, gi = self.gx, self.gi
        dgx, dgi = self.dgx + x_in * (math.e / 0.2), self.dgi + i_in * (math.e / 2.0)
        spiked = np.zeros(self.nN, dtype=bool)
        for _ in range(self.sub):
            gx1, gi1 = ex * (gx + hs * dgx), ix * (gi + hs * dgi)
            stages = iter(((gx, gi), (0.5 * (gx + gx1), 0.5 * (gi + gi1)), (0.5 * (gx + gx1), 0.5 * (gi + gi1)),
                           (gx1, gi1)))
            self.V, self.w = self._rk4(lambda V, w: self._neuron_rhs(V, w, *next(stages), ext), hs, (self.V, self.w))
            gx, gi, dgx, dgi = gx1, gi1, ex * dgx, ix * dgi
            over = self.V >= 0.0
            self.V, self.w = np.where(over, self.V_reset, self.V), np.where(over, self.w + self.b, self.w)
            spiked |= over
        self.gx, self.dgx, self.gi, self.dgi = gx, dgx, gi, dgi
        out, j = np.zeros(self.nN), np.flatnonzero(spiked)
        decay = np.exp(-(t * self.dt - self.t_last[j]) / 800.0)
        self.x[j] = 1.0 + (self.x[j] - self.x[j] * 0.5 - 1.0) * decay
        self.t_last[j] = t * self.dt
        out[j] = self.x[j] * 0.5
        return spiked, out

    def run(self, steps, record_every=0, raster=False):
        mark = max(self.pre, 1) - 1
        for _ in range(steps):
            with np.errstate(over="ignore"):
                factor = self._astro_step()
                spiked, out = self._neuron_step()
            slot = self.t % self.slots
            self.ring[slot], self.ring_s[slot] = out, factor
            self.engaged |= factor > 0.0
            if self.t == mark:
                self.engaged[:] = False
            self.counts.append(int(spiked.sum()))
            if raster:
                padded = np.zeros((self.nN + 31) // 32 * 32, dtype=np.uint8)
                padded[: self.nN] = spiked
                self.raster.append(np.packbits(padded, bitorder="little").view(np.uint32))
            self.t += 1
            if record_every and self.t % record_every == 0:
                self.recorded.append(self.Ca.copy())
        return self

    def summary(self):
        mark = max(self.pre, 1) - 1
        measured = sum(self.counts[mark + 1:])
        return {"n_exc_edges": self.exc[1].size, "n_inh_edges": self.inh[1].size, "n_e2a_edges": self.e2a[1].size,
                "n_sic_edges": self.a2n[1].size, "spikes_total": sum(self.counts), "spikes_measured": measured,
                "active_astro": int(np.sum((self.Ca - 0.19669) * 1000.0 > 1.0)),
                "engaged_astro": int(self.engaged.sum()),
                "mean_rate_hz": measured / (self.nN * self.sim_ms * 1e-3), "mean_ca": float(np.mean(self.Ca))}
