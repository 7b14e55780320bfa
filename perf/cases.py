"""Performance cases: the simulations that a program runs with this package,
from a 10,000-agent town to the 20-million-agent population, each through the
entry points that such a program calls.

A pass is one scenario: the simulation goes back to its saved initial state,
runs its days, and the program reads the daily statistics rows and the whole
end state.
"""
import functools
import math

import numpy as np
import torch

from pansim_gb300 import adjoint, cabi, closures, immunization, native, snapshot, synth
from pansim_gb300.interface import SimulatorInterface
from pansim_gb300.snapshot import AGENT_DTYPES, AGENT_MUTABLE, LOC_DTYPES, LOC_MUTABLE

START = 0  # checkpoint slot of a scenario's initial state

# the health columns of a snapshot: moved together, they are another set of
# initially infected agents
HEALTH = ["state", "days", "variant", "infectious", "st_infected_ts", "st_infected_count", "st_worst_state",
          "st_variant_mask"]

# the day flags of the runForDay binding: opening day, tightening in two
# steps, a day without changes, reopening
FLAGS = [["TPdef", "PLNONE", "CFNONE", "SONONE", "QU0", "MA1.0"],
         ["TP015", "PL0", "CF2000-0500", "SO12", "QU2", "MA0.8"],
         [],
         ["TP035", "QU3"],
         ["TPdef", "PLNONE", "CFNONE", "SONONE", "QU0", "MA1.0"]]


def listed():
    return [
        # a town, the size of the statistical tests: each timestep is a few
        # microseconds of latency
        dict(name="town_10k", kind="city", agents=10_000, locations=2_000, days=7, infected=0.001, variants=1,
             quarantine=0, testing=False, dwell=0),
        # the smallest of the benchmark populations, its week
        dict(name="city_100k", kind="city", agents=100_000, locations=20_000, days=7, infected=0.001, variants=1,
             quarantine=0, testing=False, dwell=0),
        # the benchmark's main population, its week
        dict(name="city_2m", kind="city", agents=2_000_000, locations=500_000, days=7, infected=0.001, variants=1,
             quarantine=0, testing=False, dwell=0),
        # an odd-sized city well into an epidemic: two variants, states that
        # last several days, testing and quarantine
        dict(name="outbreak_777k", kind="city", agents=777_777, locations=190_001, days=7, infected=0.03, variants=2,
             quarantine=3, testing=True, dwell=3),
        # the largest population, with every policy on: testing, quarantine,
        # a closure rule and immunization
        dict(name="policy_20m", kind="policy", agents=20_000_000, locations=5_000_000, days=2, infected=0.001),
        # an ensemble of small runs in one context (32 seeds of one town)
        dict(name="ensemble_32x10k", kind="replicas", replicas=32, smallest=10_000, largest=10_000, days=7),
        # 64 uneven replicas, a tenth of the batch benchmark's sizes
        dict(name="ensemble_64_uneven", kind="replicas", replicas=64, smallest=25_000, largest=200_000, days=5),
        # the day-at-a-time binding with changing policy flags and non-COVID
        # disease
        dict(name="flags_300k", kind="flags", agents=300_000, locations=75_000, days=5, infected=0.005),
        # a host program that calls the phases one by one, as the policy
        # adapters do: one day
        dict(name="phases_100k", kind="phases", agents=100_000, locations=20_000, steps=144, infected=0.001),
        dict(name="phases_2m", kind="phases", agents=2_000_000, locations=500_000, steps=144, infected=0.001),
        # one gradient of a calibration (expected curve forward and backward)
        dict(name="calibration_4x250k", kind="calibration", replicas=4, agents=250_000, days=7),
        # host containers regrouped by location: state in, agent list and
        # infection ratios out
        dict(name="regroup_500k", kind="regroup", agents=500_000, locations=125_000, infected=0.02),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["city", "city", "city", "policy", "replicas", "flags", "phases", "calibration", "regroup"])
    infected = math.exp(rng.uniform(math.log(0.001), math.log(0.03)))
    if kind == "city":
        n = _log(rng, 3_000, 2_500_000)
        return dict(kind=kind, agents=n, locations=n // rng.choice([3, 4, 5, 6]), days=rng.randint(2, 7),
                    infected=infected, variants=rng.choice([1, 1, 2]), quarantine=rng.choice([0, 0, 2, 3]),
                    testing=rng.random() < 0.5, dwell=rng.choice([0, 0, 3]))
    if kind == "policy":
        n = _log(rng, 100_000, 3_000_000)
        return dict(kind=kind, agents=n, locations=n // rng.choice([4, 5]), days=rng.randint(2, 4), infected=infected)
    if kind == "replicas":
        lo = _log(rng, 3_000, 50_000)
        return dict(kind=kind, replicas=rng.randint(2, 48), smallest=lo, largest=int(lo * rng.uniform(1.0, 3.0)),
                    days=rng.randint(2, 7))
    if kind == "flags":
        n = _log(rng, 20_000, 600_000)
        return dict(kind=kind, agents=n, locations=n // 4, days=rng.randint(3, 5), infected=infected)
    if kind == "phases":
        n = _log(rng, 10_000, 2_000_000)
        return dict(kind=kind, agents=n, locations=n // rng.choice([4, 5]), steps=rng.randint(60, 144),
                    infected=infected)
    if kind == "calibration":
        return dict(kind=kind, replicas=rng.randint(1, 6), agents=_log(rng, 10_000, 250_000), days=rng.randint(2, 7))
    n = _log(rng, 20_000, 2_000_000)
    return dict(kind=kind, agents=n, locations=n // 4, infected=infected)


@functools.lru_cache(maxsize=1)
def _population(agents, locations, infected, quarantine, testing, variants, dwell):
    s = synth.make_snapshot(agents, locations, pop_seed=1, initial_infected_frac=infected,
                            quarantine_policy=quarantine, testing=testing, n_variants=variants,
                            avg_len=float(dwell) if dwell else 1.0, max_len=2.0 * dwell)
    if variants > 1:
        ill = np.nonzero(s.agents["st_infected_count"])[0]
        s.agents["variant"][ill] = np.arange(len(ill)) % variants
        s.agents["st_variant_mask"][ill] = 1 << s.agents["variant"][ill].astype(np.uint32)
    return s


def _snapshot(seed, agents, locations, infected, quarantine=0, testing=False, variants=1, dwell=0):
    """The population of that size (a program has its city on file) with the
    seed's initially infected agents and the seed's draws."""
    base = _population(agents, locations, infected, quarantine, testing, variants, dwell)
    cols, shift = dict(base.agents), 1 + seed * 7919 % (agents - 1)
    for k in HEALTH:
        cols[k] = np.roll(cols[k], shift)
    cols["susceptible"] = np.roll(cols["susceptible"].reshape(variants, -1), shift, axis=1).reshape(-1)
    reps = dict(base.reps, seed=np.array([seed + 1], np.uint64))
    return snapshot.Snapshot(base.model, cols, dict(base.locs), dict(base.params, seed=seed + 1), reps)


def _pinned(snap):
    """The mutable arrays moved into one block of pinned memory in the
    library's layout: an upload or a download is one copy."""
    fields = [(snap.agents, k) for k in AGENT_MUTABLE] + [(snap.locs, k) for k in LOC_MUTABLE]
    off = native.state_layout(snap.n_agents, snap.n_locations, int(snap.model["n_variants"]))
    block = torch.empty(int(off[-1]), dtype=torch.uint8, pin_memory=True)
    buf = block.numpy()
    for j, (part, k) in enumerate(fields):
        view = buf[int(off[j]): int(off[j]) + part[k].nbytes].view(part[k].dtype)
        view[...] = part[k]
        part[k] = view
    return block


def _batch(case, seed):
    n, ks, seeds = synth.batch_sizes(case["replicas"], case["smallest"], case["largest"])
    seeds = seeds + np.uint64(seed)
    parts = [synth.make_snapshot(int(a), int(a) // 4, seed=int(seeds[r]), pop_seed=1 + r, k=float(ks[r]))
             for r, a in enumerate(n)]
    return snapshot.concat(parts, seeds, ks)


def _places(seed, snap):
    """Every agent at one of its own locations (midday, not all at home)."""
    rng = np.random.default_rng(seed)
    off = snap.agents["loc_offset"].astype(np.int64)
    pick = off[:-1] + (rng.random(snap.n_agents) * np.diff(off)).astype(np.int64)
    snap.agents["location"] = snap.agents["poss_loc"][pick]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "calibration":
        parts = [synth.make_snapshot(case["agents"], case["agents"] // 4, seed=seed + r, pop_seed=1 + r)
                 for r in range(case["replicas"])]
        batch = snapshot.concat(parts, [seed + 1 + r for r in range(len(parts))], [3.74e-4] * len(parts))
        runner = adjoint.CalibrationRunner(batch, case["days"])
        rng = np.random.default_rng(seed)
        theta = adjoint.theta_of(batch) * rng.uniform(0.9, 1.1, adjoint.N_THETA)
        target = torch.from_numpy(rng.uniform(50.0, 150.0, (len(parts), case["days"])))
        return dict(kind=kind, runner=runner, theta=torch.from_numpy(theta), target=target,
                    curve=adjoint.expected_curve_function())
    if kind == "replicas":
        snap = _batch(case, seed)
    elif kind == "city":
        snap = _snapshot(seed, case["agents"], case["locations"], case["infected"], case["quarantine"],
                         case["testing"], case["variants"], case["dwell"])
    else:
        policies = kind in ("policy", "flags")
        snap = _snapshot(seed, case["agents"], case["locations"], case["infected"],
                         quarantine=3 if kind in ("policy", "phases") else 0, testing=policies)
    if kind == "regroup":
        _places(seed, snap)
    state = dict(kind=kind, snap=snap, block=_pinned(snap), days=case.get("days"), steps=case.get("steps"))
    if kind == "flags":
        state["interface"] = SimulatorInterface()
        state["interface"].initSimulation(snap, other_disease=cabi.other_disease_options())
        state["sim"] = state["interface"].sim
    else:
        state["sim"] = native.GpuSim(snap)
    if kind == "policy":
        state["rules"] = [dict(name="lockdown", conditionType="newCasesFraction", threshold=0.0005,
                               threshold2=0.00025, closeAfter=1, openAfter=7, parameter=0,
                               locationTypesToClose=[synth.WORK, synth.SCHOOL, synth.SHOP])]
        state["header"] = closures.stats_header(synth.STATE_NAMES)
        state["immunization"] = immunization.options(
            immunizations_per_week=snap.n_agents * 7 // 400, immunizationStart=0,
            immunizationOrder="1,2,3,4,5,6,0,0,0,0", boosterStart="1000", boosters_per_week=[([0], [1.0] * 10)])
    if kind != "regroup":
        state["sim"].checkpoint_save(START)
    return state


def _row(stats):
    """The statistics rows of all replicas, as the library returns them."""
    words = np.frombuffer(stats, np.uint32).reshape(len(stats), -1)
    return _signed(words[:, : 2 + cabi.PSIM_STATS_MAX + cabi.PSIM_MAX_STRAINS])


def _signed(a):
    """32-bit words as torch indexes them."""
    return a.view(np.int32) if a.dtype == np.uint32 else a


def _outputs(state, rows):
    state["sim"].download()
    snap = state["snap"]
    return dict(rows=np.stack([np.asarray(r) for r in rows]),
                agents={k: _signed(snap.agents[k]) for k in AGENT_MUTABLE},
                locations={k: _signed(snap.locs[k]) for k in LOC_MUTABLE})


def run(state):
    kind = state["kind"]
    if kind == "calibration":
        theta = state["theta"].clone().requires_grad_(True)
        expected = state["curve"].apply(theta, state["runner"])
        ((expected - state["target"]) ** 2).sum().backward()
        return dict(expected=expected.detach(), gradient=theta.grad)
    sim = state["sim"]
    if kind == "regroup":
        sim.upload()
        sim.regroup()
        offsets, agents = sim.csr()
        return dict(offsets=_signed(offsets), agents=_signed(agents), ratios=sim.hazard())
    sim.checkpoint_restore(START)
    if kind == "flags":
        ui = state["interface"]
        ui.day, ui.mask = 0, 1.0
        return _outputs(state, [ui.runForDay(FLAGS[d]) for d in range(state["days"])])
    if kind == "phases":
        row = _row(sim.midnight(0))
        for t in range(state["steps"]):
            sim.movement(t)
            sim.regroup()
            sim.infect(t)
        return _outputs(state, [row])
    if kind == "policy":
        sim.closures_init(state["rules"], state["header"])
        sim.immunization_init(state["immunization"])
    return _outputs(state, [_row(sim.run_day(d)) for d in range(state["days"])])


def _sizes(case):
    if case["kind"] == "calibration":
        n = case["replicas"] * case["agents"]
        return n, n // 4
    if case["kind"] == "replicas":
        n = case["replicas"] * (case["smallest"] + case["largest"]) // 2
        return n, n // 4
    return case["agents"], case["locations"]


def work(case):
    """The population read once, its mutable state written once; the homes
    (two agents and a half each) are locations too."""
    agents, others = _sizes(case)
    locations = others + agents * 2 // 5
    if case["kind"] == "regroup":
        # the positions and infectiousness in; the agent list, the offsets
        # and the ratios out, from the locations' weights
        return dict(bytes=12 * agents + 12 * locations, flops=0)
    variants = case.get("variants", 1)
    state = sum(np.dtype(AGENT_DTYPES[k]).itemsize * (variants if k in ("susceptible", "symptom_scaling_v") else 1)
                for k in AGENT_MUTABLE)
    loc_state = sum(np.dtype(LOC_DTYPES[k]).itemsize for k in LOC_MUTABLE)
    # type, age, band, progression id, symptom scaling, list offset and five
    # list entries per agent; type and essential flag per location
    fixed = 1 + 1 + 1 + 2 + 4 + 4 + 5 * 5
    return dict(bytes=agents * (fixed + 2 * state) + locations * (2 + 2 * loc_state), flops=0)


def exact(case, seed):
    """The infection ratios in 64 bits.  The other cases are whole
    simulations of a sampled trajectory, which plain numpy does not follow."""
    if case["kind"] != "regroup":
        return None
    snap = _snapshot(seed, case["agents"], case["locations"], case["infected"])
    _places(seed, snap)
    p, loc, n_loc = snap.params, snap.agents["location"], snap.n_locations
    count = np.bincount(loc, minlength=n_loc)
    total = np.bincount(loc, weights=snap.agents["infectious"].astype(np.float64), minlength=n_loc)
    # the seasonal factor of day 0 (a cosine over the year around day 81)
    peak, day = 81, (int(p["start_date"]) + 6) % 366
    day = 366 - day if day > 183 else day
    wave = [0.5 * 3.08 * math.cos(2.0 * math.pi * (d - peak) / 366.0) + 1.0 - 0.5 * 3.08 for d in (day, peak)]
    season = 1.0 if day < peak else min(1.0, max(0.5, wave[0] / wave[1]))
    x = (float(p["k"]) * total / np.maximum(count, 1) * snap.locs["infectiousness"].astype(np.float64) * season
         * float(p["time_step"]))
    return dict(offsets=None, agents=None, ratios=-np.expm1(-x))
