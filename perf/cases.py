"""The work a program built on this package has it do, as cases to be timed.

Five kinds, one for each way a program drives the package:

* ``fused``    one beam through ``FusedTracker.track`` (engine.py), the path of
               a long tracking run, in each of its precision forms;
* ``batch``    many beams with their own machine settings through
               ``BatchTracker.track`` (batch.py), the path of a parameter scan;
* ``adjoint``  a gradient through ``AdjointTracker`` (adjoint.py), forward and
               backward, the path of an optimisation of the RF programme;
* ``objects``  the reference's main loop, call by call: the induced voltage,
               the RF kick and drift, the slicing and the bunch statistics
               (impedances, trackers, beam, monitors);
* ``wake``     the multi-turn wake of long-range resonators, evaluated turn by
               turn by ``InducedVoltageResonator``.

The machine is the one of bench.py: 26 GeV/c protons, C = 6911.5 m, gamma_t =
18, h = 4620, 4.5 MV, one or two RF systems, a bi-Gaussian bunch in a window
of 2.5 ns.  Bunches are drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from blond_b200 import bmath as bm
from blond_b200.adjoint import AdjointTracker, bunch_loss, gaussian_target
from blond_b200.batch import BatchTracker
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.profile import CutOptions, OtherSlicesOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import (InducedVoltageFreq, InducedVoltageResonator,
                                             InductiveImpedance, TotalInducedVoltage)
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.llrf.beam_feedback import BeamFeedback
from blond_b200.toolbox.next_regular import next_regular
from blond_b200.trackers.tracker import RingAndRFTracker

CLIGHT, E_CHARGE = 299792458.0, 1.602176634e-19
MASS = 1.67262192595e-27 * CLIGHT**2 / E_CHARGE  # proton, eV
LENGTH, ALPHA, MOMENTUM, HARMONIC, VOLTAGE = 6911.5, 1 / 18**2, 26e9, 4620, 4.5e6
WINDOW, SIGMA_DT = 2.5e-9, 0.4e-9
RAMP = 1e4  # eV/c per turn of an accelerating programme
LOOP_GAIN, LOOP_GAIN2 = 1000.0, 0.05

# shunt impedance, frequency and quality factor of the resonators
SOURCES = {
    "broadband": ([5e6], [1e9], [1.0]),
    "modes": ([2e5, 1e5, 5e4, 3e4], [200e6, 800e6, 1.4e9, 2.0e9],
              [100.0, 1000.0, 3000.0, 30000.0]),
    "long": ([1e6, 5e5, 2e5, 1e9], [200e6, 630e6, 915e6, 1.4e9], [150.0, 500.0, 3e4, 5e7]),
    "optimised": ([1e6], [1e9], [1.0]),
}
Z_OVER_N = 0.1  # Ohm, of the constant inductive impedance

FUSED = {"kind": "fused", "precision": "f64", "particles": 1_000_000, "slices": 100, "turns": 50,
         "n_rf": 1, "solver": "simple", "sources": "none", "inductive": False, "ramp": False,
         "smooth": False, "interpolation": False, "loop": False, "intensity": 1e10}


def listed():
    """The cases, in the order of their kinds."""
    return [
        # a program that looks at the profile after every turn: a small
        # bunch, odd sizes, one turn per call -- launches and latency
        {**FUSED, "name": "fused_one_turn_small", "particles": 20_001, "slices": 201, "turns": 1,
         "sources": "broadband"},
        # the reference's own single-bunch benchmark: no collective effects
        {**FUSED, "name": "fused_1e6_100_slices", "turns": 100},
        # the headline single-bunch run: 2^14 slices, broadband impedance
        {**FUSED, "name": "fused_1e7_f64", "particles": 10_000_000, "slices": 16384,
         "sources": "broadband"},
        # the same in the mixed form (float32 energies)
        {**FUSED, "name": "fused_1e7_f32p64", "precision": "f32p64", "particles": 10_000_000,
         "slices": 16384, "sources": "broadband"},
        # the largest single bunch: double RF, a long profile, four
        # resonators, fixed-point energies
        {**FUSED, "name": "fused_1e8_q32p64", "precision": "q32p64", "particles": 100_000_000,
         "slices": 65536, "n_rf": 2, "sources": "modes"},
        # a run with a beam-phase loop closed every turn, legacy drift, Z/n
        # and a profile length that is no power of two
        {**FUSED, "name": "fused_phase_loop", "particles": 2_000_001, "slices": 2000,
         "solver": "legacy", "sources": "modes", "inductive": True, "loop": True},
        # smooth slicing and the interpolated kick on an accelerating ramp,
        # double RF, exact drift
        {**FUSED, "name": "fused_smooth_interpolated", "particles": 1_000_003, "slices": 600,
         "n_rf": 2, "solver": "exact", "sources": "modes", "ramp": True, "smooth": True,
         "interpolation": True},
        # the parameter scan: 256 ragged beams of 1e5 to 4e6 particles in
        # the batched engine's default form
        {"name": "batch_256_beams", "kind": "batch", "precision": "f32p64", "beams": 256,
         "smallest": 100_000, "largest": 4_000_000, "slices": 512, "turns": 50, "n_rf": 2,
         "solver": "simple", "sources": "modes", "intensity": 1e10},
        # one gradient of the RF programme and of the resonator
        {"name": "adjoint_2e6", "kind": "adjoint", "precision": "f32p64", "particles": 2_000_000,
         "slices": 1024, "turns": 100, "checkpoint_every": 50, "intensity": 3e9},
        # the reference's main loop on a large bunch: HBM-bound kernels
        {"name": "objects_1e7_f64", "kind": "objects", "dtype": "float64",
         "particles": 10_000_000, "slices": 16384, "turns": 5, "n_rf": 1, "solver": "simple",
         "sources": "broadband", "smooth": False, "interpolation": False, "statistics": False,
         "intensity": 1e10},
        # the same in single precision on a small odd bunch, with the bunch
        # statistics of every turn: launches and host work
        {"name": "objects_small_f32", "kind": "objects", "dtype": "float32",
         "particles": 300_001, "slices": 1000, "turns": 5, "n_rf": 2, "solver": "exact",
         "sources": "modes", "smooth": False, "interpolation": False, "statistics": True,
         "intensity": 1e10},
        # one turn of a multi-turn wake with 53 turns of memory
        {"name": "wake_4_modes", "kind": "wake", "particles": 1_000_000, "slices": 1024,
         "sources": "long", "intensity": 1e11},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _slices(rng, lo, hi):
    """A profile length: a power of two, a round number or any number."""
    s = _log_size(rng, lo, hi)
    return rng.choice([1 << (s.bit_length() - 1), max(lo, s // 100 * 100), s, s | 1])


def draw(rng):
    """One more case of the ranges above."""
    kind = rng.choice(["fused", "fused", "fused", "batch", "adjoint", "objects", "wake"])
    if kind == "fused":
        n = _log_size(rng, 2e4, 3e7)
        sources = rng.choice(["none", "broadband", "modes", "modes"])
        loop = sources != "none" and rng.random() < 0.15
        smooth = not loop and rng.random() < 0.15
        slices = _slices(rng, 64, 65536 if n > 1e6 else 8192)
        # the gradient of a profile much finer than that is its shot noise
        inductive = sources == "modes" and not smooth and slices <= 4096 and rng.random() < 0.5
        return {**FUSED, "precision": rng.choice(["f64", "f64", "f32p64", "q32p64"]),
                "particles": n, "slices": slices,
                "turns": rng.choice([1, 50, rng.randint(2, 100)]), "n_rf": rng.choice([1, 1, 2]),
                "solver": rng.choice(["simple", "simple", "legacy", "exact"]), "sources": sources,
                "inductive": inductive,
                "ramp": not loop and rng.random() < 0.25, "smooth": smooth,
                "interpolation": not loop and rng.random() < 0.15, "loop": loop}
    if kind == "batch":
        small = _log_size(rng, 1e3, 1e5)
        return {"kind": "batch", "precision": rng.choice(["f64", "f32p64", "f32p64", "q32p64"]),
                "beams": _log_size(rng, 4, 64), "smallest": small,
                "largest": _log_size(rng, 2 * small, 1_000_000), "slices": _slices(rng, 100, 2048),
                "turns": rng.randint(5, 60), "n_rf": rng.choice([1, 2]),
                "solver": rng.choice(["simple", "simple", "legacy", "exact"]),
                "sources": rng.choice(["none", "broadband", "modes"]), "intensity": 1e10}
    if kind == "adjoint":
        return {"kind": "adjoint", "precision": rng.choice(["f64", "f32p64"]),
                "particles": _log_size(rng, 2e4, 2e6), "slices": 2 * _slices(rng, 100, 2048),
                "turns": rng.randint(10, 100), "checkpoint_every": rng.choice([10, 50]),
                "intensity": 3e9}
    if kind == "objects":
        return {"kind": "objects", "dtype": rng.choice(["float64", "float64", "float32"]),
                "particles": _log_size(rng, 2e4, 2e7), "slices": _slices(rng, 64, 16384),
                "turns": rng.randint(1, 8), "n_rf": rng.choice([1, 2]),
                "solver": rng.choice(["simple", "legacy", "exact"]),
                "sources": rng.choice(["none", "broadband", "modes"]),
                "smooth": rng.random() < 0.2, "interpolation": rng.random() < 0.2,
                "statistics": rng.random() < 0.5, "intensity": 1e10}
    return {"kind": "wake", "particles": _log_size(rng, 5e4, 4e6),
            "slices": _slices(rng, 100, 2048), "sources": rng.choice(["long", "modes"]),
            "intensity": 1e11}


# ---------------------------------------------------------------- the machine
def _momentum(case, n_turns):
    return MOMENTUM + (RAMP if case.get("ramp") else 0.0) * np.arange(n_turns + 1)


def _rf_systems(n_rf, voltage=VOLTAGE):
    """Harmonics, voltages and phases: a second system at four times the
    frequency and a tenth of the voltage in the double-RF cases."""
    if n_rf == 1:
        return [HARMONIC], [voltage], [0.0]
    return [HARMONIC, 4 * HARMONIC], [voltage, 0.1 * voltage], [0.0, math.pi]


def _machine(case, n_turns, voltage=VOLTAGE):
    n_rf = case.get("n_rf", 1)
    h, v, p = _rf_systems(n_rf, voltage)
    ring = Ring(LENGTH, ALPHA, _momentum(case, n_turns), Proton(), n_turns)
    return ring, RFStation(ring, h, v, p, n_rf=n_rf)


def _programme(case, n_turns, voltage=VOLTAGE):
    """The same machine's programme from its formulas, for exact()."""
    p = _momentum(case, n_turns)
    gamma = np.sqrt(1 + (p / MASS) ** 2)
    beta, energy = np.sqrt(1 - 1 / gamma**2), np.sqrt(p**2 + MASS**2)
    h, v, ph = _rf_systems(case.get("n_rf", 1), voltage)
    d_e = np.diff(energy)
    phi_s = (math.pi - np.arcsin(np.append(d_e, d_e[-1]) / voltage)) % (2 * math.pi)
    omega = np.array([2 * math.pi * beta * CLIGHT * x / LENGTH for x in h])
    return {"beta": beta, "energy": energy, "t_rev": LENGTH / (beta * CLIGHT),
            "eta0": ALPHA - gamma**-2.0, "omega": omega, "phi": np.array(ph)[:, None] + 0 * omega,
            "harmonic": h, "voltage": v, "acc": -d_e, "phi_s": phi_s}


def _bunch(case, seed, n, sigma_dt=SIGMA_DT, voltage=VOLTAGE):
    """(dt, dE, bunch centre) of a bi-Gaussian bunch matched to the main RF
    system, drawn on the GPU."""
    m = _programme(case, 1, voltage)
    w, e, b = m["omega"][0, 0], m["energy"][0], m["beta"][0]
    phi_s = m["phi_s"][0]
    phi_b = w * sigma_dt + phi_s
    sigma_dE = math.sqrt(voltage * e * b**2
                         * (math.cos(phi_b) - math.cos(phi_s) + (phi_b - phi_s) * math.sin(phi_s))
                         / (math.pi * HARMONIC * abs(m["eta0"][0])))
    centre = phi_s / w
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    dt = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * sigma_dt + centre
    dE = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * sigma_dE
    return dt, dE, centre


def _beam_list(case, seed):
    """Per beam of a batch: particles (the scan's own, whatever the seed),
    voltage, bunch length, resonator quality factors."""
    sizes = np.random.default_rng(case["beams"]).uniform(
        np.log(case["smallest"]), np.log(case["largest"]), case["beams"])
    rng = np.random.default_rng(int(seed))
    return [(int(round(np.exp(x))), rng.uniform(2e6, 7e6), rng.uniform(0.2e-9, 0.5e-9),
             np.exp(rng.uniform(np.log(100), np.log(30000), 4))) for x in sizes]


def _sources(case, q_scan=None):
    R, f, Q = SOURCES[case["sources"]]
    return R, f, (list(q_scan[: len(R)]) if q_scan is not None and len(R) > 1 else Q)


def _programme_turns(case, bytes_per_turn):
    """Turns of a programme that outlasts some seconds of tracking."""
    if case["kind"] == "batch":
        seconds, shortest = 1.2, 10e-6
    else:
        seconds, shortest = 2.5, 6e-6
        if case["sources"] == "none" and case["turns"] > 1:
            shortest, bytes_per_turn = 1.5e-6, 0
    return int(seconds / max(shortest, bytes_per_turn / 6.5e12)) + 4 * case["turns"] + 200


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    bm.use_precision("single" if case.get("dtype") == "float32" else "double")
    state = {"fused": _prepare_fused, "batch": _prepare_batch, "adjoint": _prepare_adjoint,
             "objects": _prepare_objects, "wake": _prepare_wake}[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


def _energy_bytes(case):
    return 8 if case["precision"] == "f64" else 4


def _induced_voltage(case, beam, profile, rf, n_turns, q_scan=None):
    if case["sources"] == "none":
        return None
    R, f, Q = _sources(case, q_scan)
    parts = [InducedVoltageFreq(beam, profile, [Resonators(R, f, Q)])]
    if case.get("inductive"):
        parts.append(InductiveImpedance(beam, profile, [Z_OVER_N] * (n_turns + 1), rf))
    return TotalInducedVoltage(beam, profile, parts)


def _one_beam(case, seed, n_turns, dtype=torch.float64):
    n = case["particles"]
    ring, rf = _machine(case, n_turns)
    dt, dE, centre = _bunch(case, seed, n)
    beam = Beam(ring, n, case["intensity"], dt=dt, dE=dE, dtype=dtype)
    profile = Profile(beam, CutOptions(cut_left=centre - WINDOW / 2, cut_right=centre + WINDOW / 2,
                                       n_slices=case["slices"]),
                      other_slices_options=OtherSlicesOptions(smooth=case.get("smooth", False)))
    return ring, rf, beam, profile


def _prepare_fused(case, seed):
    n_turns = _programme_turns(case, case["particles"] * 2 * (8 + _energy_bytes(case)))
    ring, rf, beam, profile = _one_beam(case, seed, n_turns)
    tiv = _induced_voltage(case, beam, profile, rf, n_turns)
    loop = None
    if case["loop"]:
        loop = BeamFeedback(ring, rf, profile, {"machine": "LHC_F", "PL_gain": LOOP_GAIN,
                                                "FL_gain": LOOP_GAIN2})
    tracker = RingAndRFTracker(rf, beam, solver=case["solver"], beam_feedback=loop,
                               interpolation=case["interpolation"], profile=profile,
                               total_induced_voltage=tiv)
    fused = FusedTracker(tracker, profile, tiv, precision=case["precision"])
    fused.prepare()
    return {"fused": fused, "beam": beam, "turns": case["turns"], "voltage": tiv is not None}


def _prepare_batch(case, seed):
    beams = _beam_list(case, seed)
    n_turns = _programme_turns(case, sum(b[0] for b in beams) * 2 * (8 + _energy_bytes(case)))
    items = []
    for k, (n, voltage, sigma_dt, q_scan) in enumerate(beams):
        ring, rf = _machine(case, n_turns, voltage)
        dt, dE, centre = _bunch(case, 1000 * seed + k, n, sigma_dt, voltage)
        beam = Beam(ring, n, case["intensity"], dt=dt, dE=dE, dtype=torch.float64)
        profile = Profile(beam, CutOptions(cut_left=centre - WINDOW / 2,
                                           cut_right=centre + WINDOW / 2,
                                           n_slices=case["slices"]))
        tiv = _induced_voltage(case, beam, profile, rf, n_turns, q_scan)
        items.append((RingAndRFTracker(rf, beam, solver=case["solver"]), profile, tiv))
    batch = BatchTracker(items, precision=case["precision"])
    batch.autotune()
    batch.prepare()
    return {"batch": batch, "turns": case["turns"], "voltage": case["sources"] != "none"}


def _prepare_adjoint(case, seed):
    n, S, T = case["particles"], case["slices"], case["turns"]
    ring, rf = _machine(case, T)
    dt, dE, centre = _bunch(case, seed, n)
    cl, cr = centre - WINDOW / 2, centre + WINDOW / 2
    tracker = AdjointTracker(ring, rf, n, case["intensity"], cl, cr, S, T, n_fft=next_regular(S),
                             precision=case["precision"],
                             checkpoint_every=case["checkpoint_every"])
    R, f, Q = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in SOURCES["optimised"])
    return {"tracker": tracker, "dt": dt, "dE": dE, "resonator": (R, f, Q),
            "V": torch.full((T, 1), VOLTAGE, dtype=torch.float64, device="cuda"),
            "P": torch.zeros(T, 1, dtype=torch.float64, device="cuda"),
            "target": gaussian_target(S, cl, cr, centre, 0.35e-9),
            "bin_centers": tracker.bin_centers()}


def _prepare_objects(case, seed):
    n_turns = 40_000
    dtype = getattr(torch, case["dtype"])
    ring, rf, beam, profile = _one_beam(case, seed, n_turns, dtype)
    tiv = _induced_voltage(case, beam, profile, rf, n_turns)
    tracker = RingAndRFTracker(rf, beam, solver=case["solver"],
                               interpolation=case["interpolation"], profile=profile,
                               total_induced_voltage=tiv)
    return {"beam": beam, "profile": profile, "tiv": tiv, "tracker": tracker, "rf": rf,
            "turns": case["turns"], "statistics": case["statistics"],
            "interpolation": case["interpolation"]}


def _prepare_wake(case, seed):
    ring, rf, beam, profile = _one_beam(case, seed, 2000)
    R, f, Q = _sources(case)
    wake = InducedVoltageResonator(beam, profile, Resonators(R, f, Q), multi_turn_wake=True,
                                   rf_station=rf, time_decay_factor=0.01)
    return {"beam": beam, "profile": profile, "wake": wake,
            "tiv": TotalInducedVoltage(beam, profile, [wake])}


# ----------------------------------------------------------------------- run
def run(state):
    return {"fused": _run_fused, "batch": _run_batch, "adjoint": _run_adjoint,
            "objects": _run_objects, "wake": _run_wake}[state["kind"]](state)


def _run_fused(state):
    """Track, then take what a program looks at: coordinates (energies in
    eV), the profile and the induced voltage."""
    fused = state["fused"]
    fused.track(state["turns"])
    out = {"dt": fused.dt, "dE": fused.energies() if fused.precision == "q32p64" else fused.dE,
           "profile": fused.profile_tensor()}
    if state["voltage"]:
        out["voltage"] = fused.induced_voltage_tensor()
    return out


def _run_batch(state):
    batch = state["batch"]
    batch.track(state["turns"])
    dE = batch.dE
    if batch.precision == "q32p64":
        dE = torch.cat([batch.energies(b) for b in range(batch.B)])
    out = {"dt": batch.dt, "dE": dE, "profiles": batch.profiles_tensor()}
    if state["voltage"]:
        out["voltages"] = batch.induced_voltages_tensor()
    return out


def _run_adjoint(state):
    """One step's gradient: the RF programme's, the resonator's and the
    initial coordinates'."""
    tracker = state["tracker"]
    leaves = [x.detach().requires_grad_(True)
              for x in (state["dt"], state["dE"], state["V"], state["P"], *state["resonator"])]
    dt, dE, V, P, R, f, Q = leaves
    dt1, dE1, profile = tracker(dt, dE, V, P, tracker.impedance(R, f, Q))
    loss = bunch_loss(profile, state["target"], state["bin_centers"])
    grads = torch.autograd.grad(loss, leaves)
    return {"loss": loss.detach(), "dt": dt1.detach(), "dE": dE1.detach(),
            "profile": profile.detach(),
            **dict(zip(("g_dt", "g_dE", "g_V", "g_phi", "g_R", "g_f", "g_Q"), grads))}


def _run_objects(state):
    """The reference's main loop (with interpolation the RF tracker applies
    the induced voltage itself)."""
    beam, profile, tiv, tracker = (state[k] for k in ("beam", "profile", "tiv", "tracker"))
    for _ in range(state["turns"]):
        if tiv is not None:
            if state["interpolation"]:
                tiv.induced_voltage_sum()
            else:
                tiv.track()
        tracker.track()
        profile.track()
        if state["statistics"]:
            beam.statistics()
    out = {"dt": beam.dt, "dE": beam.dE, "profile": profile.n_macroparticles}
    if tiv is not None:
        out["voltage"] = tiv.induced_voltage
    if state["statistics"]:
        out["statistics"] = beam.stats_tensor()
    return out


def _run_wake(state):
    state["tiv"].induced_voltage_sum()
    return {"voltage": state["tiv"].induced_voltage, "memory": state["wake"].induced_voltage}


# ---------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass.  A bunch in a run with induced
    voltage passes through the chip once per turn (every particle's kick
    needs the whole bunch's profile); without it, once per call."""
    kind = case["kind"]
    n_rf = case.get("n_rf", 1)
    # per particle and turn: a sine and its kick for each RF system, drift,
    # slice, interpolated kick
    ops = 30 * n_rf + 12
    if kind == "fused":
        n, S, T = case["particles"], case["slices"], case["turns"]
        passes = T if case["sources"] != "none" else 1
        fft = 5 * S * math.log2(S) + 20 * S if case["sources"] != "none" else 0
        return {"bytes": passes * 2 * n * (8 + _energy_bytes(case)) + 16 * S,
                "flops": T * (n * ops + fft)}
    if kind == "batch":
        mean = (case["largest"] - case["smallest"]) / math.log(case["largest"] / case["smallest"])
        n, S, T = case["beams"] * mean, case["slices"] * case["beams"], case["turns"]
        passes = T if case["sources"] != "none" else 1
        return {"bytes": passes * 2 * n * (8 + _energy_bytes(case)) + 16 * S,
                "flops": T * (n * ops + 5 * S * math.log2(case["slices"]) + 20 * S)}
    if kind == "adjoint":
        # forward: coordinates in and out per turn; backward: both adjoints
        # in and out and the turn's times
        n, T = case["particles"], case["turns"]
        return {"bytes": T * n * (2 * (8 + _energy_bytes(case)) + 32 + 8), "flops": T * n * 130}
    if kind == "objects":
        n, S, T = case["particles"], case["slices"], case["turns"]
        size = 8 if case["dtype"] == "float64" else 4
        # interpolated kick and RF kick 3 n, drift 3 n, slicing n, statistics 2 n
        arrays = (3 * (case["sources"] != "none" or case["interpolation"])
                  + 3 * (not case["interpolation"]) + 3 + 1 + 2 * case["statistics"])
        return {"bytes": T * (arrays * size * n + 16 * S), "flops": T * n * ops}
    t = len(_wake_times(case)[0])
    modes = len(SOURCES[case["sources"]][0])
    return {"bytes": 8 * t * 3 + 16 * case["slices"], "flops": 60 * (t + case["slices"]) * modes}


# --------------------------------------------------------------------- exact
def exact(case, seed):
    """The same results from the formulas, in float64 torch."""
    return {"fused": _exact_fused, "batch": _exact_batch, "adjoint": _exact_adjoint,
            "objects": _exact_objects, "wake": _exact_wake}[case["kind"]](case, seed)


def _centres(cl, cr, S):
    edges = np.linspace(cl, cr, S + 1)
    return torch.as_tensor((edges[:-1] + edges[1:]) / 2, device="cuda")


def _impedance(R, f_r, Q, n_fft, bin_size):
    f = torch.arange(1, n_fft // 2 + 1, dtype=torch.float64, device="cuda") / (n_fft * bin_size)
    z = torch.zeros(n_fft // 2 + 1, dtype=torch.complex128, device="cuda")
    for r, fr, q in zip(R, f_r, Q):
        z[1:] += r / torch.complex(torch.ones_like(f), q * (f / fr - fr / f))
    return z / bin_size


def _counts(dt, cl, cr, S):
    k = torch.floor((dt - cl) * (S / (cr - cl)))
    k = k[(k >= 0) & (k < S)].long()
    return torch.bincount(k, minlength=S).double()


def _smooth_counts(dt, cl, cr, S):
    """Half of each particle's weight about its slice, moved linearly to the
    neighbour (histogram.cpp:75-132)."""
    w = (cr - cl) / S
    x = dt[(dt >= cl + w / 2) & (dt <= cr - w / 2)]
    f = (x - cl) * (S / (cr - cl))
    k = f.long()
    d = f - k
    out = torch.zeros(S, dtype=torch.float64, device="cuda")
    out.index_add_(0, k, 0.5 - d)
    other = torch.where(d > 0.5, (f + 1).long(), (f - 1).long())
    inside = (other >= 0) & (other < S)
    out.index_add_(0, other[inside], (0.5 + d)[inside])
    return out


def _interpolated_kick(dt, dE, v, bc, acc):
    S = len(bc)
    bc0, inv = float(bc[0]), (S - 1) / float(bc[-1] - bc[0])
    k = torch.floor((dt - bc0) * inv)
    inside = (k >= 0) & (k < S - 1)
    k = k.clamp(0, S - 2).long()
    slope = (v[1:] - v[:-1]) * inv
    return torch.where(inside, dE + (dt - bc[:-1][k]) * slope[k] + v[:-1][k] + acc, dE)


def _drift(dt, dE, solver, m, t):
    T, b, e, eta = m["t_rev"][t], m["beta"][t], m["energy"][t], m["eta0"][t]
    if solver == "simple":
        return dt + T * eta / (b * b * e) * dE
    if solver == "legacy":
        return dt + T * (1.0 / (1.0 - eta / (b * b * e) * dE) - 1.0)
    inner = (dE / e) ** 2 + 2.0 * dE / e
    delta = torch.sqrt(1.0 + inner / (b * b)) - 1.0
    return dt + T * ((1.0 + ALPHA * delta) * (1.0 + dE / e) / (1.0 + delta) - 1.0)


def _track_exact(case, m, dt, dE, window, Z, n_fft, ratio):
    """case["turns"] turns of the map; returns dt, dE, profile, voltage."""
    S, (cl, cr) = case["slices"], window
    bc = _centres(cl, cr, S)
    bin_size = (cr - cl) / S
    slicing = _smooth_counts if case.get("smooth") else _counts
    profile, voltage = slicing(dt, cl, cr, S), None
    omega, phi = m["omega"].copy(), m["phi"].copy()
    dphi_rf = np.zeros(len(omega))
    for t in range(case["turns"]):
        if Z is not None:
            voltage = -E_CHARGE * ratio * torch.fft.irfft(
                Z * torch.fft.rfft(profile, n_fft), n_fft)[:S]
            if case.get("inductive"):
                voltage = voltage - (E_CHARGE / (2 * math.pi) * ratio * Z_OVER_N * m["t_rev"][t]
                                     / bin_size) * torch.gradient(
                    profile, spacing=float(bc[1] - bc[0]))[0]
        if case.get("loop"):
            arg = omega[0, t] * bc + phi[0, t]
            tan = (torch.trapezoid(profile * torch.sin(arg), dx=bin_size)
                   / torch.trapezoid(profile * torch.cos(arg), dx=bin_size))
            error = math.atan(float(tan)) + math.pi - m["phi_s"][t]
            change = -LOOP_GAIN * error - LOOP_GAIN2 * (omega[0, t] - m["omega"][0, t])
            for j, h in enumerate(m["harmonic"]):
                omega[j, t + 1] += change * h / m["harmonic"][0]
                dphi_rf[j] += 2 * math.pi * h * (omega[j, t + 1] - m["omega"][j, t + 1]) \
                    / m["omega"][j, t + 1]
                phi[j, t + 1] += dphi_rf[j]
        at = bc if case.get("interpolation") else dt
        rf = torch.zeros_like(at)
        for j, v in enumerate(m["voltage"]):
            rf = rf + v * torch.sin(omega[j, t] * at + phi[j, t])
        if case.get("interpolation"):
            dE = _interpolated_kick(dt, dE, rf if voltage is None else rf + voltage, bc,
                                    m["acc"][t])
        else:
            if voltage is not None:
                dE = _interpolated_kick(dt, dE, voltage, bc, 0.0)
            dE = dE + rf + m["acc"][t]
        dt = _drift(dt, dE, case["solver"], m, t + 1)
        profile = slicing(dt, cl, cr, S)
    return dt, dE, profile, voltage


def _exact_beam(case, seed, n, voltage=VOLTAGE, sigma_dt=SIGMA_DT, q_scan=None, dtype=None):
    m = _programme(case, case["turns"] + 1, voltage)
    dt, dE, centre = _bunch(case, seed, n, sigma_dt, voltage)
    if dtype == torch.float32:  # the single-precision beam's own starting point
        dt, dE = dt.float().double(), dE.float().double()
    window = (centre - WINDOW / 2, centre + WINDOW / 2)
    Z, n_fft = None, next_regular(case["slices"])
    if case["sources"] != "none":
        Z = _impedance(*_sources(case, q_scan), n_fft, WINDOW / case["slices"])
    return _track_exact(case, m, dt, dE, window, Z, n_fft, case["intensity"] / n)


def _exact_fused(case, seed):
    dt, dE, profile, voltage = _exact_beam(case, seed, case["particles"])
    out = {"dt": dt, "dE": dE, "profile": profile}
    if voltage is not None:
        out["voltage"] = voltage
    return out


def _exact_batch(case, seed):
    got = [_exact_beam(case, 1000 * seed + k, n, voltage, sigma_dt, q_scan)
           for k, (n, voltage, sigma_dt, q_scan) in enumerate(_beam_list(case, seed))]
    out = {"dt": torch.cat([g[0] for g in got]), "dE": torch.cat([g[1] for g in got]),
           "profiles": torch.stack([g[2] for g in got])}
    if case["sources"] != "none":
        out["voltages"] = torch.stack([g[3] for g in got])
    return out


def _exact_objects(case, seed):
    dt, dE, profile, voltage = _exact_beam(case, seed, case["particles"],
                                           dtype=getattr(torch, case["dtype"]))
    out = {"dt": dt, "dE": dE, "profile": profile}
    if voltage is not None:
        out["voltage"] = voltage
    if case["statistics"]:
        s_t, s_e = dt.std(unbiased=False), dE.std(unbiased=False)
        out["statistics"] = torch.stack([
            torch.tensor(float(len(dt)), dtype=torch.float64, device="cuda"), dt.mean(), s_t,
            dE.mean(), s_e, math.pi * s_e * s_t, dt.square().sum(), dE.square().sum()])
    return out


def _exact_adjoint(case, seed):
    """Autograd through the map, the profile a cloud-in-cell deposit on the
    bin centres."""
    n, S, T = case["particles"], case["slices"], case["turns"]
    m = _programme(case, T + 1)
    dt0, dE0, centre = _bunch(case, seed, n)
    cl = centre - WINDOW / 2
    w, n_fft = WINDOW / S, next_regular(S)
    bc0 = cl + w / 2
    bc = bc0 + w * torch.arange(S, dtype=torch.float64, device="cuda")
    scale = E_CHARGE * case["intensity"] / n

    def cell(dt):
        f = (dt - bc0) / w
        k = torch.floor(f.detach())
        return f - k, k.long(), k

    def deposit(dt):
        u, k, kf = cell(dt)
        near = (kf >= -1) & (kf < S)
        u, k = u[near], k[near]
        out = torch.zeros(S + 2, dtype=torch.float64, device="cuda")
        return out.index_add(0, k + 1, 1 - u).index_add(0, k + 2, u)[1:S + 1]

    leaves = [x.requires_grad_(True) for x in (
        dt0, dE0, torch.full((T, 1), VOLTAGE, dtype=torch.float64, device="cuda"),
        torch.zeros(T, 1, dtype=torch.float64, device="cuda"),
        *(torch.tensor(x, dtype=torch.float64, device="cuda") for x in SOURCES["optimised"]))]
    dt, dE, V, P, R, fr, Q = leaves
    f = torch.arange(1, n_fft // 2 + 1, dtype=torch.float64, device="cuda") / (n_fft * w)
    x = f / fr - fr / f
    Z = torch.cat([torch.zeros(1, dtype=torch.complex128, device="cuda"),
                   R / torch.complex(torch.ones_like(x), Q * x) / w])
    profile = deposit(dt)
    for t in range(T):
        v = -scale * torch.fft.irfft(Z * torch.fft.rfft(profile, n_fft), n_fft)[:S]
        u, k, kf = cell(dt)
        inside = (kf >= 0) & (kf < S - 1)
        k = k.clamp(0, S - 2)
        kick = torch.where(inside, v[k] * (1 - u) + v[k + 1] * u, torch.zeros_like(dt))
        dE = dE + kick + V[t, 0] * torch.sin(m["omega"][0, t] * dt + P[t, 0]) + m["acc"][t]
        dt = _drift(dt, dE, "simple", m, t + 1)
        profile = deposit(dt)
    y = torch.exp(-0.5 * ((bc - centre) / 0.35e-9) ** 2)
    ends = torch.ones_like(profile)
    ends[0] = ends[-1] = 0.5
    norm = (ends * profile).sum()
    mean = (ends * profile * bc).sum() / norm
    loss = ((ends * profile * (bc - mean) ** 2).sum() / norm / 1e-18
            + ((profile / profile.sum() - y / y.sum()) ** 2).sum())
    grads = torch.autograd.grad(loss, leaves)
    return {"loss": loss.detach(), "dt": dt.detach(), "dE": dE.detach(),
            "profile": profile.detach(),
            **dict(zip(("g_dt", "g_dE", "g_V", "g_phi", "g_R", "g_f", "g_Q"), grads))}


def _wake_times(case):
    """Times of a multi-turn wake (one slicing window per turn over which the
    slowest mode decays to 1 %, counted as the reference counts it) and the
    window's slice centres."""
    m = _programme(case, 2000)
    _, f, Q = SOURCES[case["sources"]]
    decay = 2 * max(q / (2 * math.pi * x) for q, x in zip(Q, f))
    turns = min(int(math.ceil(math.log(0.01) / math.log(E_CHARGE) * decay / m["t_rev"].min())),
                2000)
    centre = m["phi_s"][0] / m["omega"][0, 0]
    edges = np.linspace(centre - WINDOW / 2, centre + WINDOW / 2, case["slices"] + 1)
    bc = (edges[:-1] + edges[1:]) / 2
    window = np.linspace(bc[0], bc[-1], len(bc))
    return np.concatenate([m["t_rev"][k] * k + window for k in range(turns)]), bc


def _exact_wake(case, seed):
    n, S = case["particles"], case["slices"]
    times, centres = _wake_times(case)
    t, bc = torch.as_tensor(times, device="cuda"), torch.as_tensor(centres, device="cuda")
    dt, _, centre = _bunch(case, seed, n)
    profile = _counts(dt, centre - WINDOW / 2, centre + WINDOW / 2, S)
    kappa = torch.diff(profile) / torch.diff(bc) / (n * (WINDOW / S))
    v = torch.zeros_like(t)
    for R, f, Q in zip(*SOURCES[case["sources"]]):
        w, qt = 2 * math.pi * f, Q * math.sqrt(1 - 1 / (4 * Q * Q))
        a, b = w * qt / Q, w / (2 * Q)
        for part in range(0, len(t), 8192):
            D = t[part:part + 8192, None] - bc
            F = torch.where(D > 0, (2 * torch.cos(a * D) + torch.sin(a * D) / qt)
                            * torch.exp(-b * D.clamp_min(0)) - 1, torch.ones_like(D))
            v[part:part + 8192] += R / (2 * w * Q) * (torch.diff(F) @ kappa)
    v = v * (-E_CHARGE * case["intensity"])
    return {"voltage": v[:S], "memory": v}
