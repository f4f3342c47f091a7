"""Performance cases: the work that a program built on this package has it do.

``listed()`` names fixed cases and ``draw(rng)`` gives more of the same ranges;
``prepare``, ``run`` and ``work`` make, run and count one, and ``exact`` is what
it computes in 64 bits. Three kinds of work:

``propagate``  one split-step propagation of a wave field (``Plan.propagate``):
               the call that big-wave's own drivers make, on fields from a few
               hundred samples to the sizes that need three FFT levels, with and
               without the returned spectrum and the frequency cutoff;
``fft``        the natural-order transforms (``Plan.fft`` / ``Plan.ifft``);
``sim``        whole simulations (``Simulation.run_source`` / ``run_sources``):
               gratings with phase stepping, a sample, plane and point sources,
               one source or a spectrum of energies. Complex128 runs return the
               detector; complex64 runs return the field at the detector, which
               holds everything that the detector's sums are taken from.

Field lengths are powers of two in the large runs and any number otherwise (the
reference takes any N); both dtypes are in use, complex128 being the
reference's default.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from rave_sim_b200.engine import Plan, Simulation

H_C = 6.62607004 * 10 ** (-34) * 299792458
EV = 1.602176634 * 10 ** (-19)
E_REF = 46000.0
PITCH = 4.2e-6
Z0 = 2.1  # first grating; point sources stand at z = 0, plane waves start here
# delta, beta at 46 keV: gold (absorption gratings), silicon (phase grating), aluminium (sample)
MATERIALS = {"Au": (19.32, 1.44e-6, 8e-9), "Si": (2.34, 2.27e-7, 1e-10), "Al": (2.70, 2.53e-7, 2e-10)}


def wavelength(energy):
    return H_C / (energy * EV)


def listed():
    return [
        # the smallest call: one propagation of a short field, where latency is everything
        {"name": "propagate_1k_c16", "kind": "propagate", "n": 1 << 10, "dtype": "c16", "spectrum": False, "cut": False},
        # a short complex64 field with the cutoff of a finite beam
        {"name": "propagate_16k_c8", "kind": "propagate", "n": 1 << 14, "dtype": "c8", "spectrum": False, "cut": True},
        # a length that is not a power of two, called as big-wave does: the spectrum comes back too
        {"name": "propagate_12000_c16", "kind": "propagate", "n": 12000, "dtype": "c16", "spectrum": True, "cut": True},
        # the single-grating setup's field length, big-wave's call
        {"name": "propagate_1m_c16", "kind": "propagate", "n": 1 << 20, "dtype": "c16", "spectrum": True, "cut": True},
        # a long ragged length in complex64
        {"name": "propagate_1594323_c8", "kind": "propagate", "n": 3 ** 13, "dtype": "c8", "spectrum": False, "cut": False},
        # the thick-sample field length in complex64
        {"name": "propagate_64m_c8", "kind": "propagate", "n": 1 << 26, "dtype": "c8", "spectrum": False, "cut": False},
        # transforms on their own, one in each direction
        {"name": "fft_4m_c16", "kind": "fft", "n": 1 << 22, "dtype": "c16", "inverse": False},
        {"name": "ifft_16m_c8", "kind": "fft", "n": 1 << 24, "dtype": "c8", "inverse": True},
        # a small interferometer, one energy: short launches one after the other
        {"name": "interferometer_64k_c16", "kind": "sim", "n": 1 << 16, "dtype": "c16", "source": "point", "steps": 3,
         "phases": 4, "rows": 0, "energies": 1},
        # a sample between the gratings, complex64
        {"name": "sample_4m_c8", "kind": "sim", "n": 1 << 22, "dtype": "c8", "source": "plane", "steps": 4, "phases": 2,
         "rows": 24, "energies": 1},
        # a spectrum on short fields: the energies run as one batch
        {"name": "spectrum_1m_c16", "kind": "sim", "n": 1 << 20, "dtype": "c16", "source": "plane", "steps": 5,
         "phases": 4, "rows": 0, "energies": 8},
        # the interferometer at its full field length, some of its energies
        {"name": "spectrum_16m_c16", "kind": "sim", "n": 1 << 24, "dtype": "c16", "source": "plane", "steps": 5,
         "phases": 2, "rows": 0, "energies": 4},
    ]


def _length(rng, lo, hi, any_n):
    """Log-uniform field length: a power of two, or any number."""
    e = rng.uniform(lo, hi)
    return int(2 ** e) if any_n else 1 << int(round(e))


def draw(rng):
    kind = rng.choice(["propagate", "propagate", "fft", "sim", "sim"])
    dtype = rng.choice(["c16", "c8"])
    if kind == "sim":
        sample = rng.random() < 0.4
        n = 1 << rng.randint(13, 23)
        return {"kind": "sim", "n": n, "dtype": dtype, "source": rng.choice(["plane", "plane", "point"]),
                "steps": rng.randint(2, 10), "phases": rng.choice([1, 2, 4, 5, 8]),
                "rows": rng.randint(5, 40) if sample else 0,
                "energies": 1 if dtype == "c8" else rng.choice([1, 1, 2, 3, 6, 8])}
    any_n = rng.random() < 0.3
    n = _length(rng, 8, 21, True) if any_n else _length(rng, 8, 26, False)
    if kind == "fft":
        return {"kind": "fft", "n": n, "dtype": dtype, "inverse": rng.random() < 0.5}
    return {"kind": "propagate", "n": n, "dtype": dtype, "spectrum": rng.random() < 0.4, "cut": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs
def _field(case, seed):
    """A wave field: amplitudes in [0.5, 1], random phases."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    a = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.5 + 0.5
    p = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    u = torch.polar(a, p)
    return u if case["dtype"] == "c16" else u.to(torch.complex64)


def _propagation(case, seed):
    rng = np.random.default_rng(seed)
    dx = 2e-9
    p = {"dx": dx, "wl": wavelength(rng.uniform(20e3, 70e3)), "dz": rng.uniform(1e-6, 1e-1), "cutoff_freq": 1e300}
    if case["cut"]:
        p["cutoff_freq"] = rng.uniform(0.1, 0.45) / dx
    return p


def _energies(case, seed):
    return sorted(np.random.default_rng(seed).uniform(20e3, 70e3, case["energies"]).tolist())


def _table(energy):
    r = E_REF / energy
    return [[[m, rho], [d * r * r, b * r ** 4]] for m, (rho, d, b) in MATERIALS.items()]


def _material(name):
    return [name, MATERIALS[name][0]]


def _sim_config(case, seed):
    """A Talbot-Lau interferometer (absorption, phase and analyser grating,
    the analyser stepped), with a sample behind the phase grating if it has
    ``rows``; returns (config, sample grids)."""
    rng = np.random.default_rng(seed)
    n, phases, dx = case["n"], case["phases"], 2e-9
    x0 = rng.uniform(0.0, PITCH)

    def grating(z, h, mat, xs):
        return {"type": "grating", "pitch": PITCH, "dc": [0.5, 0.5], "z_start": z, "thickness": h,
                "nr_steps": case["steps"], "x_positions": xs, "substrate_thickness": 0.0,
                "mat_a": _material(mat), "mat_b": None, "mat_substrate": None}

    els = [grating(Z0, 100e-6, "Au", [x0]), grating(Z0 + 0.8, 59.37e-6, "Si", [0.0])]
    grids = {}
    if case["rows"]:
        psx = max(0.1e-6, n * dx / 400)
        els.append({"type": "sample", "z_start": Z0 + 0.801, "pixel_size_x": psx, "pixel_size_z": 10e-6,
                    "grid_path": "sample.npy", "materials": [_material("Al")], "x_positions": [0.0]})
        # solid material with cracks: runs of a few pixels, so that most samples lie inside a pixel run
        grids[2] = np.repeat(rng.random((case["rows"], 50)) < 0.8, 6, axis=1).astype(np.int8)
    els.append(grating(Z0 + 0.882, 100e-6, "Au", [k * PITCH / phases for k in range(phases)]))
    detector = min(2.048e-3, 0.8 * n * dx)
    config = {
        "sim_params": {"N": n, "dx": dx, "z_detector": Z0 + 0.882 + 100e-6, "detector_size": detector,
                       "detector_pixel_size_x": max(1e-6, detector / 2048), "detector_pixel_size_y": 1.0,
                       "chunk_size": n},
        "elements": els,
        "cutoff_angles": [math.pi / 2] * (len(els) + 1),
    }
    return config, grids


def prepare(case, seed):
    if case["kind"] == "sim":
        config, grids = _sim_config(case, seed)
        sim = Simulation(config, grids=grids, dtype=case["dtype"])
        runs = [{"energy": e, "db_table": _table(e), "weight": 1.0 / (1 + k)}
                for k, e in enumerate(_energies(case, seed))]
        source = {"type": "point", "x": 1e-6, "z": 0.0} if case["source"] == "point" else {"type": "plane", "z": Z0}
        return {"case": case, "sim": sim, "runs": runs, "source": source}
    state = {"case": case, "plan": Plan(case["n"], case["dtype"]), "u": _field(case, seed)}
    if case["kind"] == "fft":
        state["out"] = torch.empty_like(state["u"])
    else:
        state["args"] = _propagation(case, seed)
        state["U"] = torch.empty_like(state["u"]) if case["spectrum"] else None
    return state


# -------------------------------------------------------------------- runs
def run(state):
    case = state["case"]
    if case["kind"] == "sim":
        sim, runs = state["sim"], state["runs"]
        sim.reset()
        if len(runs) > 1:
            sim.run_sources(runs, source=state["source"])
        else:
            r = runs[0]
            sim.run_source(energy=r["energy"], db_table=r["db_table"], source=state["source"], weight=r["weight"])
        return sim.detected_device() if case["dtype"] == "c16" else sim.final_field()
    plan = state["plan"]
    if case["kind"] == "fft":
        return (plan.ifft if case["inverse"] else plan.fft)(state["u"], state["out"])
    plan.propagate(state["u"], state["U"], **state["args"])
    return [state["u"]] if state["U"] is None else [state["u"], state["U"]]


def _split_steps(case):
    """Split steps of one source: gap, elements, gaps; the phase steps after
    the first start before the analyser."""
    first = (case["source"] == "point") + 2 * (case["steps"] + 1) + (case["rows"] + 1 if case["rows"] else 0)
    return first + case["phases"] * case["steps"]


def work(case):
    """Bytes: a propagation reads the field and writes it (and the spectrum);
    each split step of a simulation does, since a field of these lengths does
    not stay on the chip. Operations: 5 N log2 N per transform, and the
    transfer function's product."""
    n, size = case["n"], 16 if case["dtype"] == "c16" else 8
    fft = 5.0 * n * math.log2(n)
    if case["kind"] == "fft":
        return {"bytes": 2 * n * size, "flops": fft}
    if case["kind"] == "propagate":
        return {"bytes": (3 if case["spectrum"] else 2) * n * size, "flops": 2 * fft + 6.0 * n}
    k = _split_steps(case) * case["energies"]
    return {"bytes": k * 2 * n * size, "flops": k * (2 * fft + 12.0 * n)}


# ---------------------------------------------------------- 64-bit results
def _value(v):
    """A divisor as a tensor: by a Python number, torch multiplies with the rounded reciprocal."""
    return torch.tensor(v, device="cuda", dtype=torch.float64)


def _transfer(n, dx, wl, dz, cutoff_freq):
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    f = torch.where(k < (n - 1) // 2 + 1, k, k - n) * (1.0 / n) / _value(dx)
    phi = ((-2 * math.pi) / wl) * dz
    h = torch.polar(torch.ones_like(f), math.pi * wl * dz * (f * f)) * complex(math.cos(phi), math.sin(phi))
    start = math.ceil(n * (cutoff_freq * dx))
    if start <= n / 2:
        h[start:n - start + 1] = 0
    return h


def _sample_factor(el, row, db, case, dx, wl):
    """exp(2 pi i dz / wl * db(x)), db interpolated between the pixels of a row, 0 outside."""
    n, psx = case["n"], el["pixel_size_x"]
    x = (torch.arange(n, device="cuda", dtype=torch.float64) - n / 2) * dx
    rx = (torch.arange(len(row), device="cuda", dtype=torch.float64) * psx + el["x_positions"][0]) - len(row) * psx * 0.5
    v = torch.from_numpy(np.asarray(row)).cuda().to(torch.float64)
    j = (torch.searchsorted(rx, x, right=True) - 1).clamp(0, len(row) - 2)
    w = v[j] + (v[j + 1] - v[j]) / (rx[j + 1] - rx[j]) * (x - rx[j])
    w = torch.where((x < rx[0]) | (x > rx[-1]), torch.zeros_like(w), w)
    y = 2 * math.pi * el["pixel_size_z"] / wl
    return torch.polar(torch.exp(-y * db[1] * w), y * db[0] * w)


def _exact_sim(case, seed):
    """The field at the detector after the last phase step."""
    config, grids = _sim_config(case, seed)
    energy = _energies(case, seed)[0]
    n, dx, wl = case["n"], config["sim_params"]["dx"], wavelength(energy)
    table = {m[0]: v for m, v in _table(energy)}
    z_detector = config["sim_params"]["z_detector"]
    z = Z0
    if case["source"] == "point":
        x = (torch.arange(n, device="cuda", dtype=torch.float64) - n / 2) * dx - 1e-6
        r = torch.sqrt(x * x + z * z)
        u = torch.polar(1 / torch.sqrt(r), r * ((-2 * math.pi) / wl))
    else:
        u = torch.ones(n, device="cuda", dtype=torch.complex128)

    transfers = {}

    def step(u, dz):
        if dz not in transfers:
            transfers[dz] = _transfer(n, dx, wl, dz, 1.0 / wl)
        return torch.fft.ifft(torch.fft.fft(u) * transfers[dz])

    for i, el in enumerate(config["elements"]):
        if el["z_start"] > z:
            u = step(u, el["z_start"] - z)
        z = el["z_start"]
        if el["type"] == "sample":
            for row in grids[i]:
                u = step(u * _sample_factor(el, row, table["Al"], case, dx, wl), el["pixel_size_z"])
            z += el["pixel_size_z"] * len(grids[i])
            continue
        start = -(n // 2) * dx + el["x_positions"][-1]
        x = torch.arange(n, device="cuda", dtype=torch.float64) * (((start + n * dx) - start) / n) + start
        dz = el["thickness"] / el["nr_steps"]
        d, b = table[el["mat_a"][0]]
        y = 2 * math.pi * dz / wl
        factor = complex(math.exp(-y * b) * math.cos(y * d), math.exp(-y * b) * math.sin(y * d))
        for k in range(el["nr_steps"]):
            # the duty cycle of a sub-step, interpolated as the reference does
            dc = (1.0 - k / el["nr_steps"]) * el["dc"][0] + k / el["nr_steps"] * el["dc"][1]
            a = x / _value(el["pitch"]) + dc / 2
            mask = (a - torch.floor(a) < dc).to(torch.complex128)
            u = step(u * (1.0 + (factor - 1.0) * mask), dz)
        z += el["thickness"]
    return step(u, z_detector - z) if z < z_detector - 1e-8 else u


def exact(case, seed):
    if case["kind"] == "sim":
        # complex128 runs return detector sums: the field's own dtype bounds them closely already
        return _exact_sim(case, seed) if case["dtype"] == "c8" else None
    u = _field(case, seed).to(torch.complex128)
    if case["kind"] == "fft":
        return (torch.fft.ifft if case["inverse"] else torch.fft.fft)(u)
    p = _propagation(case, seed)
    U = torch.fft.fft(u) * _transfer(case["n"], p["dx"], p["wl"], p["dz"], p["cutoff_freq"])
    return [torch.fft.ifft(U), U] if case["spectrum"] else [torch.fft.ifft(U)]
