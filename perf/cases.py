"""The performance cases of the transport library: what a detector-simulation program asks of it.

Each case is one call of a public entry point (`SimulationEngine.run_packed`,
`HistogramAdjoint.loss_and_grad`, `partition_deposits_on_device`) on inputs that the program has
on the host before the call, as the API takes them. The engine (lattice tables, detector, field
mesh) is what such a program builds once and keeps; the inputs are another batch each time.

Kinds:
  pool       batched_fp32, phonon events: the form a production run uses
  published  batched_fp32, the published phonon benchmark (polynomial surfaces, 100 bounces)
  charges    batched_fp32, an electron-hole pair per event drifting at 4 V, Luke phonons counted
  recoil     batched_fp32, electron recoils in a field mesh, 5 % of the Luke phonons tracked
  inline     batched_fp32_inline, phonon events: hits in a fixed order, as the adjoint replays them
  plain      plain_fp64 (the default form), the reference's event streams bit for bit
  adjoint    loss and gradient of an arrival-time histogram (two transports)
  partition  recoil deposits split into carriers and phonons on the device

The batched forms return the hits of an event as a set in no fixed order; a case that keeps them
orders them by time, as a program that builds pulses does, and every case copies the records it
keeps into the program's own buffers (sized once for the batch; unused entries are zero). Large
production batches ask for the per-event record only (keep_hits False).

No case has values that plain numpy could give: every output is the end of a Monte Carlo history
of thousands of dependent steps, so `exact` answers None.
"""
import functools
import math

import numpy as np

import cmpmc_b200 as cm
from cmpmc_b200 import _ffi

_ADJOINT_BINS, _ADJOINT_RANGE = 64, (0.0, 1e-3)
# the sampling caps of a fast deposit simulation (records carry the weights)
_MAX_PAIRS, _MAX_PHONONS = 64, 50


def listed():
    return [
        # one recoil-sized group of phonons, its pulse wanted at once: launch and chain latency
        {"name": "pool_one_event", "kind": "pool", "events": 1, "mask": False, "surrogate": False, "hits": True},
        # a short batch with the SuperCDMS electrode layout on both faces (an odd count)
        {"name": "pool_masked_203", "kind": "pool", "events": 203, "mask": True, "surrogate": False, "hits": False},
        # the benchmark's batch: 1,000,000 primary phonons of 1-30 meV
        {"name": "pool_10000", "kind": "pool", "events": 10000, "mask": False, "surrogate": False, "hits": False},
        # the published phonon benchmark, one 7.5 meV phonon per event
        {"name": "published_100000", "kind": "published", "events": 100000},
        # a calibration run of pairs that does not fill the card, and one that does
        {"name": "charges_2000", "kind": "charges", "events": 2000},
        {"name": "charges_50000", "kind": "charges", "events": 50000},
        # low-energy recoils in the 3D field mesh: carriers, prompt and Luke phonons in turns
        {"name": "recoil_light_64", "kind": "recoil", "events": 64},
        # hits in a fixed order for a replayable forward pass
        {"name": "inline_500", "kind": "inline", "events": 500},
        # event-by-event validation against the reference: phonons in the volume, and the
        # mixed phonon / pair events with 2 % of the Luke phonons tracked
        {"name": "plain_phonon_2000", "kind": "plain", "events": 2000, "charges": False},
        {"name": "plain_mixed_203", "kind": "plain", "events": 203, "charges": True},
        # one optimisation step of the four transport parameters
        {"name": "adjoint_200", "kind": "adjoint", "events": 200},
        # the deposits of one exposure, 10 eV - 10 keV, electron and nuclear recoils
        {"name": "partition_1024", "kind": "partition", "events": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pool", "pool", "pool", "published", "charges", "charges", "recoil", "inline", "plain", "plain",
                       "adjoint", "partition"])
    if kind == "pool":
        n = _log_int(rng, 1, 10000)
        return {"kind": kind, "events": n, "mask": rng.random() < 0.3, "surrogate": rng.random() < 0.2,
                "hits": n <= 4}
    if kind == "plain":
        return {"kind": kind, "events": _log_int(rng, 1, 10000), "charges": rng.random() < 0.3}
    lo, hi = {"published": (1, 200000), "charges": (1, 50000), "recoil": (4, 128), "inline": (1, 1000),
              "adjoint": (1, 500), "partition": (1, 4096)}[kind]
    return {"kind": kind, "events": _log_int(rng, lo, hi)}


@functools.lru_cache(maxsize=None)
def _lattice():
    return cm.CrystalLattice(cm.materials.Germanium())


@functools.lru_cache(maxsize=None)
def _recoil_mesh():
    return cm.TriLinearMesh3D.recoil_mesh(cm.DetectorModel())


@functools.lru_cache(maxsize=1)
def _engine(setup):
    """The engine a program keeps for its detector; one at a time, so that its device buffers go
    with it."""
    det = cm.DetectorModel()
    if setup == "published":
        det = cm.DetectorModel.published_benchmark()
    elif setup == "masked":
        for face in (0, 1):
            det.surfaces[face].electrode_mask = cm.ElectrodePatternMask.supercdms_qet_mask(det.solid.radius, 0.8)
    elif setup == "drift":
        det.e_field = cm.UniformElectricField.from_bias(4.0, 2.54 * cm.units.cm)
        det.luke_sample_fraction = 0.0
    elif setup == "recoil":
        det.mesh_field_3d = _recoil_mesh()
        det.luke_sample_fraction = 0.05
    elif setup == "mixed":
        det.e_field = cm.UniformElectricField.from_bias(2.0, 2.54 * cm.units.cm)
        det.luke_sample_fraction = 0.02
    return cm.SimulationEngine(_lattice(), det)


def prepare(case, seed):
    kind, n = case["kind"], case["events"]
    if kind == "partition":
        return _prepare_deposits(n, seed)
    w = cm.workloads
    setup, workload, form = {
        "pool": ("masked" if case.get("mask") else "default", w.mixed_energy, "batched_fp32"),
        "published": ("published", w.published_phonon, "batched_fp32"),
        "charges": ("drift", w.pair_drift, "batched_fp32"),
        "recoil": ("recoil", w.recoil_light, "batched_fp32"),
        "inline": ("default", w.mixed_energy, "batched_fp32_inline"),
        "plain": ("mixed", w.test_parallel, "plain_fp64") if case.get("charges") else
                 ("default", w.single_l_volume, "plain_fp64"),
        "adjoint": ("default", w.mixed_energy, None),
    }[kind]
    engine = _engine(setup)
    packed = engine.generate(workload, n, seed)
    if kind == "adjoint":
        adjoint = cm.HistogramAdjoint(engine, packed, seed, n_bins=_ADJOINT_BINS, t_range=_ADJOINT_RANGE)
        theta = cm.default_theta(engine)
        rng = np.random.default_rng(seed)
        # a measured pulse: the exponential arrival-time shape at the batch's size, with noise
        t = np.linspace(*_ADJOINT_RANGE, _ADJOINT_BINS, endpoint=False)
        target = 27.0 * 100 * n * np.exp(-t / 2.5e-4) * rng.uniform(0.9, 1.1, _ADJOINT_BINS) / 16.0
        return {"kind": kind, "adjoint": adjoint, "theta": theta, "target": np.round(target)}
    hits = {"pool": case.get("hits", False), "published": False, "recoil": False, "charges": n <= 2000}.get(kind, True)
    options = cm.RunOptions(seed=seed, form=form, keep_hits=hits, want_event_stats=True,
                            kaplan_surrogate=bool(case.get("surrogate")))
    buffer = np.zeros(_hit_room(case) if hits else 0, dtype=_ffi.HIT_DTYPE)
    return {"kind": kind, "engine": engine, "packed": packed, "options": options, "hits": buffer,
            "order": kind in ("pool", "charges")}


def _hit_room(case):
    """Hits that a batch of this size may bring, with room for its fluctuations."""
    kind, n = case["kind"], case["events"]
    if kind == "charges":
        return 2 * n
    if kind == "plain" and case["charges"]:
        return 2000 * n + 20000
    primaries = n if kind == "plain" else 100 * n
    return int(30 * primaries + 400 * math.sqrt(primaries))


def _prepare_deposits(n, seed):
    rng = np.random.default_rng(seed)
    engine = _engine("default")
    deposits = np.zeros(n, dtype=_ffi.DEPOSIT_DTYPE)
    solid = engine.detector.solid
    r, phi = solid.radius * np.sqrt(rng.uniform(size=n)), 2.0 * np.pi * rng.uniform(size=n)
    deposits["pos"] = np.stack([r * np.cos(phi), r * np.sin(phi), solid.half_z * rng.uniform(-1.0, 1.0, n)], axis=1)
    deposits["time_s"] = 1e-9 * np.arange(n)
    deposits["edep_eV"] = 10.0 * 10.0 ** (3.0 * rng.uniform(size=n))
    deposits["is_nuclear_recoil"] = np.arange(n) % 3 == 2
    states = rng.integers(1, 1 << 63, size=(n, 4), dtype=np.uint64)
    options = cm.PartitionOptions(max_sampled_pairs=_MAX_PAIRS, max_sampled_phonons=_MAX_PHONONS)
    return {"kind": "partition", "engine": engine, "deposits": deposits, "states": states, "options": options,
            "charges": np.zeros(2 * _MAX_PAIRS * n, dtype=_ffi.CHARGE_DTYPE),
            "phonons": np.zeros(_MAX_PHONONS * n, dtype=_ffi.PHONON_DTYPE)}


def _columns(records, prefix):
    return {f"{prefix}_{name}": records[name] for name in records.dtype.names if not name.startswith("_pad")}


def _keep(buffer, records):
    buffer[:len(records)].view(np.uint8)[:] = records.view(np.uint8)


def run(state):
    if state["kind"] == "adjoint":
        loss, grad, res = state["adjoint"].loss_and_grad(state["theta"], state["target"])
        return {"loss": loss, "grad": grad, "grad_var": res.grad_var, "value": res.value, "hist": res.hist,
                **res.stats.as_dict()}
    if state["kind"] == "partition":
        ch_off, ch, ph_off, ph, rng_state = cm.partition_deposits_on_device(
            state["engine"], state["deposits"], state["states"], state["options"])
        _keep(state["charges"], ch)
        _keep(state["phonons"], ph)
        return {"charge_offsets": ch_off, "phonon_offsets": ph_off, "rng_state": rng_state,
                **_columns(state["charges"], "charge"), **_columns(state["phonons"], "phonon")}
    res = state["engine"].run_packed(state["packed"], state["options"])
    out = _columns(res.event_stats, "event")
    if state["options"].keep_hits:
        hits = res.hits
        if state["order"]:  # the hits of each event by arrival time
            event = np.repeat(np.arange(len(res.hit_offsets) - 1), np.diff(res.hit_offsets.astype(np.int64)))
            hits = hits[np.lexsort((hits["time"], event))]
        _keep(state["hits"], hits)
        out.update(_columns(state["hits"], "hit"), hit_offsets=res.hit_offsets)
    return out


# Mean steps of a history (a primary with everything it leaves behind), measured, and the
# arithmetic a step cannot do without: free flight, exit test, move, new direction and the
# blended group-velocity lookup of a phonon; rates, mid-point velocity and exit test of a carrier.
_PHONON_STEP, _CARRIER_STEP = 120.0, 150.0


def work(case):
    kind, n = case["kind"], case["events"]
    track, record, hit = 128.0, 208.0, 56.0
    if kind == "partition":
        pairs, phonons = 46.0, 49.0  # sampled records of a deposit, mean over the energies
        return {"bytes": n * (48 + 64 + (2 * pairs + phonons) * track), "flops": n * (2 * pairs + phonons) * 100.0}
    if kind in ("pool", "inline", "adjoint"):
        steps = 4230.0 * 100 * n
        passes = 2 if kind == "adjoint" else 1
        kept = 2743.0 * hit if (kind == "inline" or case.get("hits")) else 0.0
        return {"bytes": passes * n * (100 * track + record + kept), "flops": passes * steps * _PHONON_STEP}
    if kind == "published":
        return {"bytes": n * (track + record), "flops": n * 3480.0 * _PHONON_STEP}
    if kind == "charges":
        return {"bytes": n * 2 * (track + hit) + n * record, "flops": n * 2 * 19100.0 * _CARRIER_STEP}
    if kind == "recoil":
        return {"bytes": n * (46 * track + record), "flops": n * (26 * 19100.0 * _CARRIER_STEP + 5e6 * _PHONON_STEP)}
    if case["charges"]:
        return {"bytes": n * (2 * track + record), "flops": n * (19100.0 * _CARRIER_STEP + 1e6 * _PHONON_STEP)}
    return {"bytes": n * (track + record + 27 * hit), "flops": n * 4070.0 * _PHONON_STEP}


def exact(case, seed):
    return None
