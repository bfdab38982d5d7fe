"""The work that users of this framework have it do, as cases that can be
timed: whole simulations, hours stepped one by one, steps on caller-owned
device memory, ensembles and served requests, from a thousand eggs to 5e7.

Every pass starts from the case's initial population and is a whole call
sequence of a user's program, so passes on one state repeat each other. A
pass returns what such a program keeps: the statistics of every hour, the age
histogram and (where a program would read it back) the final pool. A
simulation's numbers are whole or decided bit for bit by the model's binary32
definitions; only the single step on device memory returns computed columns
that a 64-bit evaluation can stand beside (exact())."""
import ctypes as C
import os

import numpy as np
import torch

from sampo_gb300 import _lib, inputs
from sampo_gb300.batch import Batch, ReplicateSpec
from sampo_gb300.population import make_pool
from sampo_gb300.serve import Request, Server
from sampo_gb300.sim import Simulation, pop_from_ranges, rand_state, seed_stream
from sampo_gb300.species import Species

HOT_SPECIES = os.path.join("tests", "golden", "species", "hot_species.h")


def listed():
    return [
        # src/abms.c's own loop: the host hands over each hour's inputs and
        # reads its statistics back before the next; one day of 10,000 eggs
        dict(name="hourly_1e4", kind="hourly", initial=10_000, hours=24, interventions=True),
        # the smallest useful simulation: a month of a thousand eggs
        dict(name="plain_1e3_month", kind="plain", initial=1_000, days=30, age_days=3, interventions=False, pool=True),
        # the CPU-runnable configuration: 10,000 eggs for a year
        dict(name="plain_1e4_year", kind="plain", initial=10_000, days=365, age_days=3, interventions=False, pool=True),
        # the reference's default start (32,000 age-0 eggs) with all four
        # interventions switched on and off, for two months
        dict(name="plain_default_2months", kind="plain", initial=32_000, days=60, age_days=-1, interventions=True, pool=True),
        # a large plain run while it grows: 1e6 eggs, two months, up to 3e7 agents
        dict(name="plain_1e6_2months", kind="plain", initial=1_000_000, days=60, age_days=3, interventions=False, pool=False),
        # the size of the bandwidth-roofline configuration: 5e7 eggs in 1e8 slots, twelve days
        dict(name="plain_5e7_12days", kind="plain", initial=50_000_000, days=12, age_days=3, interventions=False, pool=False),
        # a study that starts from a population in progress: 1e6 mixed-stage
        # agents (40/30/10/20) loaded from the host, ten days
        dict(name="mixed_1e6_10days", kind="mixed", eggs=400_000, larvae=300_000, pupae=100_000, adults=200_000, days=10),
        # another species' header, compiled at run time: 20,000 eggs, a month
        dict(name="species_2e4_month", kind="species", initial=20_000, days=30, interventions=True),
        # one hour on pools that live in another framework's device memory:
        # a small odd one by day, and 5e6 agents uniform over the stages at night
        dict(name="device_step_5e3", kind="device_step", eggs=2_003, larvae=1_499, pupae=501, adults=1_001, hour=12, interventions=True),
        dict(name="device_step_5e6", kind="device_step", eggs=1_250_000, larvae=1_250_000, pupae=1_250_000, adults=1_250_000, hour=20,
             interventions=False),
        # a batched ensemble: replicates log-uniform in [1e3, 1e6] eggs, each with its own weather
        dict(name="ensemble_96", kind="ensemble", replicates=96, low=1_000, high=1_000_000, days=20),
        # requests served with continuous batching: all there at once, one to two months each
        dict(name="served_24", kind="served", requests=24, low=100, high=200_000, min_days=30, max_days=60),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["hourly", "plain", "plain", "plain", "mixed", "species", "device_step", "device_step", "ensemble", "served"])
    on = rng.random() < 0.4
    if kind == "hourly":
        return dict(kind=kind, initial=_log(rng, 500, 200_000), hours=rng.randint(6, 48), interventions=on)
    if kind == "plain":
        days = rng.randint(5, 120)
        most = 1.4e10 / (24 * days * max(1.0, _growth(days)))  # fewer agent-hours than the largest listed case
        return dict(kind=kind, initial=_log(rng, 500, min(5e7, most)), days=days, age_days=rng.choice([-1, 3]), interventions=on,
                    pool=False)
    if kind == "mixed":
        n = _log(rng, 3_000, 1_000_000)
        return dict(kind=kind, days=rng.randint(2, 10), **_stages(rng, n))
    if kind == "species":
        return dict(kind=kind, initial=_log(rng, 500, 100_000), days=rng.randint(10, 40), interventions=on)
    if kind == "device_step":
        return dict(kind=kind, hour=rng.randint(0, 23), interventions=on, **_stages(rng, _log(rng, 500, 5_000_000)))
    if kind == "ensemble":
        return dict(kind=kind, replicates=rng.randint(3, 96), low=_log(rng, 200, 5_000), high=_log(rng, 20_000, 1_000_000),
                    days=rng.randint(5, 20))
    lo = rng.randint(30, 40)
    return dict(kind=kind, requests=rng.randint(4, 24), low=100, high=_log(rng, 5_000, 200_000), min_days=lo, max_days=lo + rng.randint(1, 20))


def _stages(rng, n):
    w = [rng.uniform(0.2, 1.0), rng.uniform(0.2, 1.0), rng.uniform(0.02, 0.4), rng.uniform(0.05, 0.5)]
    c = [int(n * x / sum(w)) for x in w]
    return dict(eggs=c[0], larvae=c[1], pupae=c[2], adults=c[3])


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _weather(days, seed, on, cc):
    """Hourly temperatures and environment rows, as readSingleValFile and
    readEnvironment would return them."""
    w = inputs.seasonal_weather(days, seed, mean=26.0, amplitude=4.0, noise_sd=0.5)
    T = np.repeat(w.temperature_c.astype(np.float32), 24)
    env = np.zeros(len(T), dtype=inputs.ENV_DTYPE)
    env["bloodmealSuccess"] = 0.25
    env["carryingCapacity"] = np.float32(cc)
    if on:
        row = inputs.alternating_interventions()
        r = np.array([row(i) for i in range(len(T))], dtype=np.float32)
        for k, name in enumerate(("IRSValue", "ITNValue", "larvacideValue", "oviTrapValue")):
            env[name] = r[:, 2 * k] * r[:, 2 * k + 1]
        env["bloodmealSuccess"] = r[:, 8]
    return T, env


def _capacity(initial, days):
    """Slots for `days` of growth (populations reach about 35 x their start after two to four months)."""
    most = 2 if days <= 12 else 12 if days <= 20 else 30 if days <= 40 else 48
    return int(most * initial) + 65_536


_species = []


def _hot_species():
    """Compiled once per process, as a program that runs several simulations keeps it."""
    if not _species:
        _species.append(Species(header_path=HOT_SPECIES))
    return _species[0]


def _simulation(case, seed, initial, steps, capacity):
    cc = 5.0 * initial
    sim = Simulation(capacity=capacity, carrying_capacity=cc, max_steps=steps + 1)
    if case["kind"] == "species":
        sim.set_species(_hot_species())
    T, env = _weather(-(-steps // 24), seed, case.get("interventions", False), cc)
    init, seeds = seed_stream(seed, steps)
    sim.set_inputs(T[:steps], env[:steps])
    sim.set_seeds(0, seeds)
    return dict(case=case, seed=seed, sim=sim, T=T, env=env, init=init, seeds=seeds, steps=steps)


def prepare(case, seed):
    kind = case["kind"]
    s = 1 + (seed * 7919 + 17) % 1_000_003
    if kind == "hourly":
        return _simulation(case, s, case["initial"], case["hours"], 3 * case["initial"] + 65_536)
    if kind in ("plain", "species"):
        n, days = case["initial"], case["days"]
        return _simulation(case, s, n, 24 * days, _capacity(n, days))
    if kind == "mixed":
        counts = (case["eggs"], case["larvae"], case["pupae"], case["adults"])
        st = _simulation(case, s, sum(counts), 24 * case["days"], 24 * sum(counts) + 65_536)
        st["pool"] = make_pool(counts, st["T"][0], seed=s)
        return st
    if kind == "device_step":
        return _device_step_state(case, s)
    if kind == "ensemble":
        return _ensemble_state(case, s)
    rng = np.random.default_rng(s)
    lo, hi = np.log(case["low"]), np.log(case["high"])
    reqs = []
    for i in range(case["requests"]):
        n = int(round(float(np.exp(rng.uniform(lo, hi)))))
        reqs.append(Request(i, _spec(rng, n, int(rng.integers(case["min_days"], case["max_days"] + 1)), 2 * n + 65_536), 0.0))
    return dict(case=case, server=Server(budget_bytes=150_000_000_000, max_days=case["max_days"]), requests=reqs)


def _spec(rng, n, days, capacity):
    return ReplicateSpec(initial=n, seed=int(rng.integers(1, 2**31 - 1)), mean_t=float(rng.uniform(20.0, 30.0)),
                         amplitude=float(rng.uniform(2.0, 8.0)), rain_mean=float(rng.uniform(2.0, 8.0)), days=days, capacity=capacity)


def _ensemble_state(case, s):
    rng = np.random.default_rng(s)
    lo, hi, days = np.log(case["low"]), np.log(case["high"]), case["days"]
    batch = Batch(case["replicates"], 24 * days + 1)
    reps = []
    for _ in range(case["replicates"]):
        n = int(round(float(np.exp(rng.uniform(lo, hi)))))
        spec = _spec(rng, n, days, 20 * n + 65_536)
        slot = batch.add(spec.capacity, spec.cc, stop_step=spec.steps)
        T, env = spec.inputs()
        batch.set_inputs(slot, T, env)
        reps.append((slot, spec, *rand_state(spec.seed)))
    return dict(case=case, batch=batch, reps=reps)


COLUMNS = [("ageInHours", torch.float32), ("hoursInState", torch.float32), ("delay", torch.float32),
           ("cumulativeSporogonicDevelopment", torch.float32), ("larvalDelayOrOviAttempts", torch.int32),
           ("availableEggs", torch.int32), ("cycleLength", torch.int32), ("humanBloodmealCount", torch.int32),
           ("numEggBatches", torch.int32)]


def _device_columns(capacity):
    t = {name: torch.zeros(capacity + 4, dtype=dt, device="cuda") for name, dt in COLUMNS}
    t["flags"] = torch.zeros(capacity + 16, dtype=torch.uint8, device="cuda")
    return t, _lib.DevicePool(**{k: v.data_ptr() for k, v in t.items()})


def _step_inputs(case, s):
    """What one step reads, on the host: the pool, the temperature, the environment and the generator's seeds."""
    counts = (case["eggs"], case["larvae"], case["pupae"], case["adults"])
    T, env = _weather(21, s, case["interventions"], 5.0 * sum(counts))
    i = 480 - 24 + case["hour"] if case["interventions"] else case["hour"]  # the interventions' second block of ten days is on
    ranges, arrays = make_pool(counts, T[0], seed=s)
    _, seeds = seed_stream(s, 1)
    return ranges, arrays, float(T[i]), env[i], seeds[0]


def _step_capacities(case):
    n = case["eggs"] + case["larvae"] + case["pupae"] + case["adults"] + 512  # the ranges start on multiples of 64
    return n, 3 * n + 65_536


def _device_step_state(case, s):
    ranges, arrays, T, env, seeds = _step_inputs(case, s)
    n, (cap, cap_out) = int(ranges[7][1]), _step_capacities(case)
    tin, din = _device_columns(cap)
    for name, dt in COLUMNS:
        tin[name][:n].copy_(torch.from_numpy(arrays[name].view(np.int32 if dt == torch.int32 else np.float32)))
    tin["flags"][:n].copy_(torch.from_numpy((arrays["state"] & 7) | (arrays["isFemale"] << 3)))
    tout, dout = _device_columns(cap_out)
    return dict(case=case, tin=tin, din=din, cap=cap, tout=tout, dout=dout, cap_out=cap_out, pop=pop_from_ranges(ranges),
                env=_lib.Environment(*[float(env[k]) for k in inputs.ENV_DTYPE.names]), T=T,
                cc=float(env["carryingCapacity"]), seeds=np.ascontiguousarray(seeds, dtype=np.uint32))


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _rows(rows):
    return np.ascontiguousarray(rows).view(np.int32).reshape(-1, 23)


def _padded(a, n):
    """Outputs of one size whatever the seed: `a`, then zeros up to n rows."""
    out = np.zeros((n,) + a.shape[1:], dtype=a.dtype)
    out[:len(a)] = a
    return out


def _pool(sim):
    pop, a = sim.read_pool()
    gap = np.ones(len(a["state"]), dtype=bool)  # slots between the ranges hold nothing
    for start, end in pop["ranges"]:
        gap[start:end] = False
    for v in a.values():
        v[gap] = 0
    a = {k: v if v.dtype != np.uint32 else v.view(np.int32) for k, v in a.items()}
    return {"ranges": pop["ranges"].astype(np.int32), **{k: _padded(v, sim.capacity) for k, v in a.items()}}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("plain", "species"):
        sim = state["sim"]
        sim.init_population(case["initial"], state["init"], age_days_max=case.get("age_days", 3), age_seed=state["seed"])
        out = {"rows": _rows(sim.run(state["steps"])), "histogram": sim.histogram().view(np.int32)}
        if kind == "species" or case["pool"]:
            out["pool"] = _pool(sim)
        return out
    if kind == "mixed":
        sim = state["sim"]
        sim.load_pool(*state["pool"])
        return {"rows": _rows(sim.run(state["steps"])), "histogram": sim.histogram().view(np.int32)}
    if kind == "hourly":
        sim = state["sim"]
        sim.init_population(case["initial"], state["init"], age_days_max=3, age_seed=state["seed"])
        rows = [sim.step(state["env"][h], state["T"][h], h % 24, state["seeds"][h]) for h in range(state["steps"])]
        return {"rows": _rows(np.stack(rows)), "histogram": sim.histogram().view(np.int32), "pool": _pool(sim)}
    if kind == "device_step":
        row, pop, bnc = _lib.StatsRow(), _lib.Population(), _lib.BitesCycles()
        rc = _lib.load().sampo_step_noalloc(
            C.byref(state["din"]), state["cap"], C.byref(state["dout"]), state["cap_out"], C.byref(state["pop"]), C.byref(state["env"]),
            state["T"], case["hour"], state["seeds"].ctypes.data, state["cc"], C.byref(row), C.byref(pop), C.byref(bnc), 0, None)
        if rc != 0:
            raise RuntimeError("sampo_step_noalloc returned %d" % rc)
        whole = [np.frombuffer(bytes(x), dtype=np.int32) for x in (row, pop, bnc)]
        return {"row": whole[0], "next": whole[1], "counters": whole[2], **state["tout"]}
    if kind == "ensemble":
        batch, steps = state["batch"], 24 * case["days"]
        for slot, spec, init, stream in state["reps"]:
            batch.init_population(slot, spec.initial, init, age_days_max=spec.age_days_max, age_seed=spec.seed)
            batch.seed_stream(slot, stream)
        batch.run(steps)
        return {"rows": _rows(np.concatenate([batch.rows(r[0], 0, steps + 1) for r in state["reps"]])),
                "histograms": np.stack([batch.histogram(r[0]) for r in state["reps"]]).view(np.int32)}
    done = state["server"].serve(state["requests"])
    most = 24 * case["max_days"] + 1
    return {"rows": _rows(np.concatenate([_padded(r.rows, most) for r in done])), "histograms": np.stack([r.histogram for r in done]).view(np.int32),
            "status": np.array([r.status for r in done], dtype=np.int32)}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
# Live agents per initial egg, averaged over the first `days` of a run under
# this weather (26 +- 4 C, carrying capacity 5 x initial).
GROWTH = ((0, 1.0), (2, 0.9), (5, 0.76), (10, 0.59), (15, 0.49), (20, 1.55), (30, 2.7), (40, 5.7), (60, 11.4), (90, 18.0), (120, 22.0),
          (180, 24.5), (365, 18.3))


def _growth(days):
    return float(np.interp(days, *zip(*GROWTH)))


# An agent that lives through an hour is read and written. What it carries
# depends on its stage: age, delay and sex (9 bytes) as an egg, its development
# too (13) as a larva, 17 as a pupa or an unbitten adult, 37 as a biting female.
# Populations in progress are about 70 % eggs, 24 % larvae, 2 % pupae, 4 % adults.
AGENT_BYTES = 2 * (0.70 * 9 + 0.24 * 13 + 0.02 * 17 + 0.04 * 25)
HOUR_BYTES = 4 + 24 + 64 + 92  # the hour's inputs and its row


def work(case):
    kind = case["kind"]
    if kind == "device_step":  # whole records, read and written, in the caller's columns
        n = case["eggs"] + case["larvae"] + case["pupae"] + case["adults"]
        return {"bytes": 74.0 * n, "flops": 10.0 * n}
    if kind == "ensemble":
        lo, hi, days = case["low"], case["high"], case["days"]
        agents, hours = case["replicates"] * (hi - lo) / np.log(hi / lo) * _growth(days), 24 * days * case["replicates"]
        agents *= 24 * days
    elif kind == "served":
        lo, hi, days = case["low"], case["high"], (case["min_days"] + case["max_days"]) / 2
        agents, hours = case["requests"] * (hi - lo) / np.log(hi / lo) * _growth(days) * 24 * days, 24 * days * case["requests"]
    elif kind == "mixed":
        hours = 24 * case["days"]
        agents = (case["eggs"] + case["larvae"] + case["pupae"] + case["adults"]) * 6.4 * hours
    elif kind == "hourly":
        hours = case["hours"]
        agents = case["initial"] * hours
    else:
        hours = 24 * case["days"]
        agents = case["initial"] * _growth(case["days"]) * hours
    if case.get("interventions"):
        agents *= 0.35  # interventions on every other ten days hold the population down
    return {"bytes": float(AGENT_BYTES * agents + HOUR_BYTES * hours), "flops": float(10.0 * agents)}


# ---------------------------------------------------------------------------
# A step's computed columns in 64 bits
# ---------------------------------------------------------------------------
F, U = np.float32, np.uint32
DEV_RATES = (0.000175044, 0.000549094, 0.00109031, 0.001494158, 0.001752487, 0.001962866, 0.002171238, 0.002392989, 0.002633689, 0.00289619,
             0.003182685, 0.003495287, 0.003836204, 0.004207789, 0.004612566, 0.005053243, 0.005532729, 0.006054144, 0.006620836, 0.007236393,
             0.007904657, 0.008629745, 0.009416051, 0.010267388, 0.011113704, 0.011960019, 0.012806335, 0.010401163, 0.007995991, 0.00033845,
             0.00000533086, 0.0000000840986)


def _taus(z, a, b, c, m):
    return ((z & U(m)) << U(c)) ^ (((z << U(a)) ^ z) >> U(b))


def _uniform(seed, gid):
    """HybridTaus of one seed slot (include/gpuRand.h:33-50): a binary32 uniform number per slot index."""
    z1, z2, z3, z4 = (np.array([x], dtype=U) for x in seed)
    v = _taus(z1 + U(128), 13, 19, 12, 4294967294) ^ _taus(z2 + U(128) + gid, 2, 25, 4, 4294967288)
    v = v ^ _taus(z3 + U(128), 3, 11, 17, 4294967280) ^ (U(1664525) * (z4 * gid) + U(1013904223))
    return F(2.3283064365387e-10) * v.astype(F)


def _mortality(dmr):
    dsr = (F(1) - dmr).astype(F)
    return (F(1) - np.power(dsr.astype(np.float64), np.float64(F(1) / F(24))).astype(F)).astype(F)


def exact(case, seed):
    """The columns of the one step whose values are computed: decisions by the
    model's binary32 definitions, every value that is stored in 64 bits."""
    if case["kind"] != "device_step" or case["eggs"] + case["larvae"] + case["pupae"] + case["adults"] > 6_000_000:
        return None
    with np.errstate(all="ignore"):
        return _exact_step(case, 1 + (seed * 7919 + 17) % 1_000_003)


def _exact_step(case, s):
    ranges, arrays, T, env, seeds = _step_inputs(case, s)
    T, cc, wt = F(T), F(env["carryingCapacity"]), case["hour"]
    rg = [slice(int(a), int(b)) for a, b in ranges]
    night = wt <= 6 or wt >= 18
    days = lambda age: np.minimum(age / F(24), F(99)).astype(np.int64)  # noqa: E731
    larvae = arrays["ageInHours"][rg[1]]
    l1 = int((larvae / F(24)).astype(np.int64).sum())
    biomass = F(l1 + int(ranges[0][1]) + int(ranges[2][1] - ranges[2][0]))
    d = np.arange(100, dtype=F)
    e = np.exp((d / F(25)).astype(np.float64)).astype(F)
    adult_hmr = _mortality(((F(0.1) * e) / (F(1) + (F(0.1) * F(25) * F(0.1) * (e - F(1))))).astype(F))
    larva_hmr = _mortality(np.minimum(F(0.1) * np.exp((F(l1) / (d * cc * F(1))).astype(np.float64)).astype(F), F(0.8)))
    aquatic = _mortality(np.array([0.1], dtype=F))[0]
    inc = 1.0 / (np.float64(F(111) / (T - F(16))) * 14.0) if T > 16 else 0.0
    pupa_delay, immature_delay, bmd_delay = (-0.923 * np.float64(T) + 60.923, -2.667 * np.float64(T) + 120.0, -1.231 * np.float64(T) + 77.231)
    to, cols, new_eggs = [[] for _ in range(8)], ("age", "his", "delay", "sporo"), 0
    for k in range(8):
        a = {n: arrays[c][rg[k]] for n, c in (("age", "ageInHours"), ("his", "hoursInState"), ("delay", "delay"), ("uni", "larvalDelayOrOviAttempts"),
                                             ("sporo", "cumulativeSporogonicDevelopment"), ("avail", "availableEggs"),
                                             ("hbc", "humanBloodmealCount"), ("female", "isFemale"))}
        gid = np.arange(rg[k].start, rg[k].stop, dtype=U)
        u = lambda slot: _uniform(seeds[slot], gid)  # noqa: E731,B023
        hmr = adult_hmr[days(a["age"])] if k >= 3 else larva_hmr[days(a["age"])] if k == 1 else aquatic
        alive = u(0) > hmr
        age, his = a["age"].astype(np.float64) + 1, a["his"].astype(np.float64) + 1
        sporo = a["sporo"].astype(np.float64) + np.where((a["hbc"] > 0) & bool(T > 16), inc, 0.0)
        delay, ns = a["delay"].astype(np.float64), np.full(len(gid), k)
        due = his >= a["delay"]
        if k == 0:
            r = np.sqrt(-2 * np.log(u(1).astype(np.float64))) * np.sin(np.float64(F(2) * F(3.14159274101257)) * u(2))
            go, nxt, nd, na = due, 1, r * 0.1 + 1, 24.0
        elif k == 1:
            if env["larvacideValue"] > 0:
                alive &= ~((his == 1) & (u(2) <= env["larvacideValue"]))
            dev = F(DEV_RATES[int(min(max(T, F(12)), F(48))) - 12])
            go, nxt, nd, na = (a["uni"].view(F) + dev >= a["delay"]) & night, 2, pupa_delay, None
        elif k == 2:
            go, nxt, nd, na = due & night, 3, immature_delay, 0.0
        elif k == 3:
            go, nxt, nd, na = due, 4, 1.0, None
        elif k == 4:
            go, nxt, nd, na = due & (a["female"] > 0) & (wt == 18), 5, 0.0, None
        elif k == 5:
            go, nxt, nd, na = due & night & (u(1) <= env["bloodmealSuccess"]), 6, bmd_delay, None
            if env["ITNValue"] > 0:
                alive &= ~(go & (u(2) <= env["ITNValue"]))
        elif k == 6:
            if env["IRSValue"] > 0:
                alive &= ~(u(2) <= env["IRSValue"])
            go, nxt, nd, na = due, 7, delay, None
        else:
            lays = (u(1) < F(0.25)) & night & alive
            trapped = lays & (u(2) <= env["oviTrapValue"]) & bool(env["oviTrapValue"] > 0)
            left = np.maximum(F(0), F(1) - biomass / ((a["uni"].astype(F) + F(1)) * cc))
            laid = np.where(lays & ~trapped, np.ceil(a["avail"].astype(F) * left), 0).astype(np.int64)
            new_eggs += int(laid.sum())
            alive &= ~trapped
            go, nxt, nd, na = lays & (a["avail"] == laid), 5, 0.0, None
        ns[go], his, delay = nxt, np.where(go, 0.0, his), np.where(go, nd, delay)
        age = age if na is None else np.where(go, na, age)
        for j in sorted({k, nxt}):
            m = alive & (ns == j)
            to[j].append([x[m] for x in (age, his, delay, sporo)])
    out, start = {c: np.zeros(_step_capacities(case)[1] + 4) for c in cols}, 0
    gid = np.arange(new_eggs, dtype=U)
    p = _uniform(seeds[2], gid)
    m, b = (np.select([p < F(x) for x in (0.5, 0.85, 0.90, 0.94)], [F(y) for y in v[:4]], F(v[4])).astype(F)
            for v in ((48.0, 68.5714, 480.0, 600.0, 2400.0), (0.0, -10.2857, -360.0, -468.0, -2160.0)))
    hatch = np.trunc((m * p + b + F(0.5)).astype(F)).astype(np.float64)
    to[0].insert(0, [np.zeros(new_eggs), np.zeros(new_eggs), -0.923 * np.float64(T) + 60.923 + hatch, np.zeros(new_eggs)])
    for j in range(8):
        parts = [np.concatenate(x) for x in zip(*to[j])] if to[j] else [np.zeros(0)] * 4
        for c, x in zip(cols, parts):
            out[c][start:start + len(x)] = x
        start = ((start + len(parts[0]) + 64) // 64) * 64
    names = dict(zip(cols, ("ageInHours", "hoursInState", "delay", "cumulativeSporogonicDevelopment")))
    whole = ("row", "next", "counters", "larvalDelayOrOviAttempts", "availableEggs", "cycleLength", "humanBloodmealCount", "numEggBatches", "flags")
    return {**{k: None for k in whole}, **{names[c]: out[c] for c in cols}}
