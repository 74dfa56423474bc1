"""Performance cases of the stepping loop.

Each case is a whole transport as a program of this package makes it: primaries
in hand, a ``Stepper`` with its parameters, then reseed for the event, insert
the primaries, step until no track is alive or queued, and read the results
(the served cases instead let events join the running loop). The listed cases
are the package's own workloads (``celeritas_gb300.workloads``) at the sizes
that a pass of at most about a second allows, from one shower in a few
thousand track slots, where a pass is all launches and latency, to a batch of
events in 2^21 slots: both precisions, both geometries, no field, a uniform
field and a field map, multiple scattering on and off, sorted and unsorted
track orders, detector hits, and events served from one pool.

Outputs are the step counters of every step, the energy deposited in every
detector volume and, where the case asks for them, the events' depositions or
the detector hits, in arrays of a length that the case fixes (a caller's
buffers). A shower has no closed form, so ``exact`` has no value for
them: they are a function of the primaries and the seed alone, and a run of
the same inputs gives the same counters.
"""

import math

import numpy as np

import celeritas_gb300 as gb
from celeritas_gb300.primaries import eta_beam, pencil_beam, spread_beam

PDGS = {"electron": (11,), "positron": (-11,), "photon": (22,), "mixed": (11, 22)}

# Defaults of a case: a transport in the calorimeter, nothing optional
BASE = dict(precision="double", geometry="calo", field="none", msc=False, order=0,
            tuned=False, hits=False, served=False, beam="electron", primaries=1, events=1,
            emin=1000.0, emax=1000.0, slots=4096)
MAX_STEPS = 20_000


def case(name=None, **settings):
    c = dict(BASE, **settings)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # One electron shower in a small state: the smallest call, all
        # launches and latency (unit tests, step-by-step debugging, the
        # reference's own stepper tests)
        case("fp64_calo_single", emin=100.0, emax=100.0, slots=4096),
        # One two-particle event in the CMS-like detector, as an interactive
        # user or a low-rate server has it
        case("mixed_cms_single", precision="mixed", geometry="cms", field="uniform", msc=True,
             order=7, beam="mixed", primaries=2, slots=1 << 14),
        # The c1 workload: 100 electrons of 1 GeV, no field, no multiple
        # scattering, the bit-exact build
        case("fp64_calo_c1", primaries=100, slots=1 << 16),
        # c2's physics (multiple scattering, 1 T) in the bit-exact build, a
        # slot count that is no multiple of any block
        case("fp64_calo_c2", field="uniform", msc=True, order=7, primaries=300, events=300,
             emin=100.0, emax=1e4, slots=200_001),
        # One c3-like event in the bit-exact build, plain order
        case("fp64_cms_event", geometry="cms", field="uniform", msc=True, beam="mixed",
             primaries=20, emin=1000.0, emax=1e4, slots=1 << 17),
        # The same physics with detector hits collected (StepCollector)
        case("fp64_cms_hits", geometry="cms", field="uniform", msc=True, beam="mixed",
             hits=True, primaries=7, emin=500.0, emax=5000.0, slots=50_000),
        # Photons, no field, no multiple scattering: straight lines only
        case("mixed_calo_photons", precision="mixed", beam="photon", order=5,
             primaries=2000, events=2000, slots=1 << 18),
        # The c2 workload in the mixed build, default launch settings
        case("mixed_calo_c2", precision="mixed", field="uniform", msc=True, order=7,
             primaries=3000, events=3000, emin=100.0, emax=1e4, slots=1 << 20),
        # A batch of c3 events with the launch settings the tuner finds: the
        # largest case
        case("mixed_cms_c3", precision="mixed", geometry="cms", field="uniform", msc=True,
             order=7, tuned=True, beam="mixed", primaries=650, events=13, emin=1000.0,
             emax=1e5, slots=1 << 21),
        # Events in the R-Z field map, sorted by particle type
        case("mixed_cms_map", precision="mixed", geometry="cms", field="map", msc=True, order=4,
             beam="mixed", primaries=120, events=4, emin=1000.0, emax=2e4, slots=300_000),
        # Events of uneven size served from one pool: they join the running
        # loop in three waves, per-event results (continuous batching)
        case("mixed_cms_served", precision="mixed", geometry="cms", field="uniform", msc=True,
             order=7, tuned=True, served=True, beam="mixed", primaries=200, events=24,
             emin=100.0, emax=2e4, slots=1 << 19),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["fp64_calo", "fp64_cms", "mixed_calo", "mixed_cms", "served"])
    mixed = not kind.startswith("fp64")
    cms = kind.endswith("cms") or kind == "served"
    served = kind == "served"
    # Transported energy, of which the work is a nearly fixed multiple
    top = {"fp64_calo": 6e5, "fp64_cms": 6e3, "mixed_calo": 6e6, "mixed_cms": 6e6,
           "served": 8e5}[kind]
    energy = _log_uniform(rng, 1e4 if served else 200.0, top)
    mean = _log_uniform(rng, 100.0, min(2e4, energy / 4 if served else energy))
    spread = rng.choice([1.0, 1.5, 4.0])
    primaries = max(4 if served else 1, int(energy / mean))
    field = rng.choice(["uniform", "uniform", "map"] if cms and mixed else
                       ["uniform"] if cms else ["none", "uniform"])
    # At least as many slots as primaries, at most what the listed cases have
    cap = (1 << 21) if mixed else (1 << 18)
    slots = int(_log_uniform(rng, max(4000, 2 * primaries, energy / 50), cap))
    order = rng.choice([0, 4, 5, 7])
    return case(precision="mixed" if mixed else "double",
                geometry="cms" if cms else "calo", field=field,
                msc=cms or field != "none" or rng.random() < 0.3, order=order,
                tuned=mixed and order == 7 and rng.random() < 0.5,
                hits=not mixed and energy < 2e4 and rng.random() < 0.4, served=served,
                beam=rng.choice(["mixed"] if cms else ["electron", "positron", "photon"]),
                primaries=primaries,
                events=min(primaries, rng.randint(4, 24)) if served else
                rng.choice([1, primaries]),
                emin=round(mean / spread, 3), emax=round(mean * spread, 3), slots=slots)


def _mean_energy(c):
    lo, hi = c["emin"], c["emax"]
    return lo if hi <= lo else (hi - lo) / math.log(hi / lo)


def _primaries(c, seed):
    n, events = c["primaries"], c["events"]
    if c["geometry"] == "cms":
        p = eta_beam(n, emin=c["emin"], emax=c["emax"], pdgs=PDGS[c["beam"]], seed=seed,
                     num_events=events)
        if c["served"]:
            # Uneven events: cut the primaries at random places
            rng = np.random.default_rng(seed + 1)
            cuts = np.sort(rng.choice(np.arange(1, n), size=events - 1, replace=False))
            p["event"] = np.searchsorted(cuts, np.arange(n), side="right")
        return p
    if c["emax"] > c["emin"]:
        return spread_beam(n, emin=c["emin"], emax=c["emax"], pdg=PDGS[c["beam"]][0], seed=seed,
                           num_events=events)
    p = pencil_beam(n, energy=c["emin"], pdg=PDGS[c["beam"]][0], num_events=events)
    return p


def prepare(case, seed):
    c = dict(BASE, **case)
    uniform = (0.0, 0.0, 3.8) if c["geometry"] == "cms" else (1.0, 0.0, 0.0)
    params = gb.Params(gb.physics_file(c["geometry"]), c["geometry"],
                       field_tesla=uniform if c["field"] == "uniform" else (0.0, 0.0, 0.0),
                       rz_field=gb.field_map_file("cms") if c["field"] == "map" else None,
                       msc=c["msc"], track_order=c["order"], precision=c["precision"],
                       rng_per_track=c["served"], event_tallies=c["served"],
                       reentrant_looping=c["field"] != "none")
    stepper = gb.Stepper(params, c["slots"], seed=seed % 1_000_003)
    if c["tuned"]:
        stepper.set_tuning(along_block_size=128, along_persistent=0, sort_threshold=1 << 17,
                           sort_material=1)
    if c["hits"]:
        # Hits of the whole transport: fewer than its track-steps
        capacity = 1 << int(10 * c["primaries"] * c["emax"]).bit_length()
        stepper.set_step_output(capacity=capacity)
        c["capacity"] = capacity
    stepper.warm_up()
    return {"case": c, "stepper": stepper, "primaries": _primaries(c, seed % 2_000_003)}


def _filled(values, size):
    """'values' in an array of 'size' rows, the rest zero."""
    out = np.zeros((size,) + values.shape[1:], dtype=values.dtype)
    out[:len(values)] = values
    return out


def _counters(results):
    return _filled(np.array([(r.generated, r.queued, r.active, r.alive) for r in results],
                            dtype=np.int64), MAX_STEPS)


def run(state):
    c, st, prim = state["case"], state["stepper"], state["primaries"]
    st.clear_energy_deposition()
    out = {}
    if c["served"]:
        # Three waves of events join the loop, which runs until it is empty
        results = []
        wave = -(-c["events"] // 3)
        for first in range(0, c["events"], wave):
            here = (prim["event"] >= first) & (prim["event"] < first + wave)
            results.append(st.step(prim[here]))
            results += st.run(max_steps=64, batch=16)
            st.event_live(c["events"])
        while results[-1]:
            results += st.run(max_steps=64, batch=16)
            live = st.event_live(c["events"])
        out["live"] = live.astype(np.int64)
        out["events"] = st.event_energy_deposition(c["events"], clear=True)
        out["event_detectors"] = st.event_detector_energy_deposition(0, c["events"], clear=True)
    else:
        st.reseed(0)
        results = [st.step(prim)]
        results += st.run(max_steps=MAX_STEPS - 1)
    out["steps"] = _counters(results)
    out["deposition"] = st.energy_deposition()
    if c["hits"]:
        hits = st.read_step_output(copy=False)
        # Track IDs are handed out by an atomic counter in thread order, the
        # step is counted from the stepper's first pass
        for k, v in hits.items():
            if k not in ("track_id", "parent_id", "step"):
                v = v.astype(np.int64) if v.dtype.kind == "u" else v
                out[k] = _filled(v, c["capacity"])
    return out


def work(case):
    """Track-steps of the showers, each of which reads and writes its track's
    state once, and the arithmetic of one track-step."""
    c = dict(BASE, **case)
    # Track-steps per MeV of the calorimeter and of the CMS-like detector
    per_mev = 3.2 if c["geometry"] == "cms" else 7.0
    steps = c["primaries"] * _mean_energy(c) * per_mev
    state = 215 + 18 * (8 if c["precision"] == "double" else 4)
    flops = 300 + (700 if c["field"] != "none" else 0) + (300 if c["msc"] else 0)
    return {"bytes": 2.0 * steps * state, "flops": steps * flops}


def exact(case, seed):
    return None
