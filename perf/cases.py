"""The work that a user of this framework has it do, as cases that can be timed and checked.

A case is a dict of plain values. `listed()` gives the named ones, `draw(rng)` one more of the
same ranges, `prepare(case, seed)` what a program holds before the call (a simulation, a batch, a
design problem), `run(state)` one pass through the public entry points, `work(case)` the bytes and
operations that the pass cannot do without, and `exact(case, seed)` what the pass returns in 64
bits by plain torch, without this package's code.

A pass continues the state's run: its fields after the pass, as the engine holds them on the
device, and its transform sums so far. Sizes are those of the package's configurations
(photonoxide_b200/configs.py), of its serving stream and of its tests; grids are 20 nm cells of
silicon in silica unless a case says otherwise.
"""
import ctypes
import math

import numpy as np
import torch

from photonoxide_b200 import configs
from photonoxide_b200.adjoint import TeFlux
from photonoxide_b200.batch import Batch
from photonoxide_b200.fdtd import Simulation, library
from photonoxide_b200.serving import Server
from photonoxide_b200.types import (INF, Axis, Bloch, Boundaries, Boxes, Cpml, Current, Dispersive,
                                    Field, FluxPlane, Grid3d, Periodic, PlaneWave, Pml, Pole, Source,
                                    Waveform)

N_SI2, N_SIO2 = 3.48 ** 2, 1.444 ** 2
H = 0.02  # um, the cells of the silicon grids
TAU = 2.0 * math.pi
C_UM_PER_S = 299_792_458e6


def listed():
    return [
        # the smallest grid in the tests (odd sizes, CPMLs with kappa and alpha, a wall, a lossy
        # block, sources of every kind, a transform box and a flux box): latency
        {"name": "small-3d", "kind": "block", "nx": 37, "ny": 21, "nz": 19, "edges": "mixed",
         "lossy": True, "bits": 32, "steps": 128},
        # a straight 2D guide with a transform of the whole plane at 21 wavelengths
        {"name": "strip-2d", "kind": "strip", "nx": 400, "ny": 200, "freqs": 21, "bits": 32,
         "steps": 4000},
        # a 2D scattering run: an oblique plane wave's box around a block, a flux box around it
        {"name": "plane-wave-2d", "kind": "wave", "nx": 320, "ny": 260, "bits": 32, "steps": 256},
        # a periodic cell between Bloch sides (complex fields), transmission through its layers
        {"name": "bloch-3d", "kind": "bloch", "nx": 48, "ny": 48, "nz": 120, "bits": 32,
         "steps": 400},
        # a dielectric block in a box whose rows are not whole vectors
        {"name": "odd-3d", "kind": "block", "nx": 301, "ny": 157, "nz": 83, "edges": "cpml",
         "lossy": False, "bits": 32, "steps": 64},
        # the same stepping in double precision, periodic along x and y (a grating's cell)
        {"name": "double-3d", "kind": "block", "nx": 160, "ny": 120, "nz": 96, "edges": "xy",
         "lossy": False, "bits": 64, "steps": 64},
        # the 3D splitter, the framework's headline: flux through both arms at 51 wavelengths
        {"name": "mmi-3d", "kind": "mmi", "nx": 600, "ny": 200, "nz": 100, "freqs": 51, "bits": 32,
         "steps": 400},
        # metal and resonant dielectric boxes in vacuum
        {"name": "dispersive-3d", "kind": "dispersive", "nx": 256, "ny": 256, "nz": 128, "bits": 32,
         "steps": 64},
        # uneven 2D designs stepped together (an ensemble of 64, sides 256 to 1024)
        {"name": "batch-2d", "kind": "batch", "count": 64, "lo": 256, "hi": 1024, "quad": False,
         "freqs": 1, "bits": 32, "steps": 512},
        # a few served-size 2D grids, widths of whole vectors
        {"name": "batch-2d-few", "kind": "batch", "count": 6, "lo": 316, "hi": 640, "quad": True,
         "freqs": 21, "bits": 32, "steps": 512},
        # one step of a topology optimisation: the flux of a 40 x 40 design and its gradient
        {"name": "adjoint-2d", "kind": "adjoint", "nx": 240, "ny": 180, "design": 40,
         "segment": 500, "bits": 32, "steps": 2000},
        # a burst of served jobs, made, stepped together and read back
        {"name": "serving", "kind": "serving", "flat": 5, "solid": 2, "lo": 100_000, "hi": 400_000,
         "freqs": 21, "bits": 32, "steps": 2000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "strip", "wave", "bloch", "mmi", "dispersive", "batch", "batch",
                       "adjoint", "serving"])
    bits = 64 if rng.random() < 0.25 else 32
    if kind == "block":  # grids of 6e3 to 5e6 cells, any sizes
        cells = _log(rng, 6_000, 5_000_000)
        nz = max(12, int(round(cells ** (1 / 3) * rng.uniform(0.4, 1.0))))
        nx = max(20, int(round(math.sqrt(cells / nz) * rng.uniform(0.7, 1.6))))
        ny = max(16, int(round(cells / nz / nx)))
        if rng.random() < 0.4:
            nx = max(20, nx - nx % 4)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz,
                "edges": rng.choice(["mixed", "cpml", "xy", "walls"]),
                "lossy": rng.random() < 0.3, "bits": bits, "steps": rng.randint(40, 160)}
    if kind == "strip":
        return {"kind": kind, "nx": _log(rng, 150, 700), "ny": _log(rng, 100, 400),
                "freqs": rng.randint(1, 24), "bits": bits, "steps": rng.randint(500, 3000)}
    if kind == "wave":
        return {"kind": kind, "nx": _log(rng, 120, 700), "ny": _log(rng, 120, 500), "bits": bits,
                "steps": rng.randint(100, 400)}
    if kind == "bloch":
        return {"kind": kind, "nx": rng.randint(16, 80), "ny": rng.randint(16, 80),
                "nz": rng.randint(80, 200), "bits": bits, "steps": rng.randint(100, 300)}
    if kind == "mmi":  # splitters of 1 to 10 million cells
        s = math.exp(rng.uniform(math.log(0.45), math.log(0.92)))
        return {"kind": kind, "nx": int(600 * s), "ny": int(200 * s), "nz": int(100 * s),
                "freqs": rng.randint(5, 51), "bits": 32, "steps": rng.randint(100, 400)}
    if kind == "dispersive":
        s = math.exp(rng.uniform(math.log(0.3), math.log(0.9)))
        return {"kind": kind, "nx": int(256 * s), "ny": int(256 * s), "nz": int(128 * s), "bits": bits,
                "steps": rng.randint(30, 64)}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 1, 40), "lo": rng.randint(96, 256),
                "hi": rng.randint(300, 900), "quad": rng.random() < 0.5, "freqs": rng.randint(1, 30),
                "bits": bits, "steps": rng.randint(100, 512)}
    if kind == "adjoint":
        return {"kind": kind, "nx": rng.randint(140, 320), "ny": rng.randint(120, 240),
                "design": rng.randint(16, 44), "segment": rng.choice([200, 333, 500]), "bits": bits,
                "steps": rng.randint(1600, 2200)}
    return {"kind": kind, "flat": rng.randint(1, 5), "solid": rng.randint(0, 2), "lo": 60_000,
            "hi": _log(rng, 100_000, 400_000), "freqs": rng.randint(1, 30), "bits": 32,
            "steps": rng.randint(1000, 2000)}


# -- the problems, as plain data that both a simulation and the 64-bit check are made from --------

def _gauss(frequency, bandwidth):
    """The numbers of Waveform.pulse(frequency, bandwidth): frequency, width, delay."""
    width = math.sqrt(2.0 * math.log(2.0)) / (math.pi * bandwidth)
    return frequency, width, 6.0 * width


def _freqs(count, lo=1.5, hi=1.6):
    return [1.0 / w for w in np.linspace(lo, hi, count)] if count > 1 else [1.0 / 1.55]


def _centred(n, h):
    return (-n[0] * h / 2.0, -n[1] * h / 2.0, -n[2] * h / 2.0)


def _problem(n, h, edges, courant, origin=None, cpml=(1.0, 0.0)):
    """A problem with nothing in it: `edges` per axis ("pml", low, high), ("periodic",) or ("bloch",
    k); `cpml` its kappa and alpha."""
    return {"n": tuple(n), "h": h, "origin": origin or _centred(n, h), "edges": edges,
            "courant": courant, "cpml": cpml, "background": N_SIO2, "boxes": [], "sigma": [], "media": [],
            "points": [], "currents": [], "monitors": [], "noise": None, "probes": []}


def _block(case, seed):
    """A block and a slab, fields everywhere at the start, sources on E and H and a current."""
    rng = np.random.default_rng(seed)
    n, h = (case["nx"], case["ny"], case["nz"]), 0.05
    pml = max(3, min(10, min(n) // 6))
    edges = {"cpml": [("pml", pml, pml)] * 3,
             "mixed": [("pml", pml, pml + 1), ("pml", pml, 0), ("pml", pml, pml)],
             "xy": [("periodic",), ("periodic",), ("pml", pml, pml)],
             "walls": [("pml", 0, 0)] * 3}[case["edges"]]
    p = _problem(n, h, edges, 0.9, cpml=(3.0, 0.2) if case["edges"] == "mixed" else (1.0, 0.0))
    lx, ly, lz = (0.5 * m * h for m in n)
    a = rng.uniform(0.3, 0.6, 3)
    p["background"] = 1.0
    p["boxes"] = [((-a[0] * lx, -a[1] * ly, -INF), (a[0] * lx, a[1] * ly, INF), 12.0),
                  ((-INF, -INF, a[2] * lz), (INF, INF, INF), 2.25)]
    if case["lossy"]:
        p["sigma"] = [((0.4 * lx, 0.2 * ly, -INF), (INF, INF, INF), 2.0)]
    w = _gauss(1.0, 0.6)
    mid = tuple(m // 2 for m in n)
    p["points"] = [(0, 2, mid, w), (1, 0, (n[0] // 4, mid[1], mid[2]), w)]
    p["currents"] = [(0, [(2, mid, 0.5), (1, (mid[0] + 3, mid[1], mid[2]), -0.3),
                          (0, (mid[0] - 2, mid[1] + 1, mid[2]), float(rng.uniform(0.2, 0.8)))], w)]
    p["monitors"] = [("dft", tuple(max(0, m - 6) for m in mid[:2]) + (mid[2] - 2,),
                      tuple(min(n[q] - 1, mid[q] + 6) for q in range(2)) + (mid[2] + 2,),
                      [0.8, 1.0, 1.3]),
                     ("flux", 2, n[2] - pml - 2, None, [0.8, 1.0, 1.3])]
    p["noise"] = (seed, 0.01)
    return p


def _strip(case, seed):
    """A straight guide, its half width from the seed, a line source, the whole plane's transform."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], 1)
    p = _problem(n, H, [("pml", 12, 12), ("pml", 12, 12), ("periodic",)], 0.5)
    half = float(rng.uniform(0.2, 0.3))
    p["boxes"] = [((-INF, -half, -INF), (INF, half, INF), N_SI2)]
    p["points"] = [(1, 2, (62, n[1] // 2, 0), _gauss(1.0 / 1.55, 0.6))]
    p["monitors"] = [("dft", (0, 0, 0), (n[0] - 1, n[1] - 1, 0), _freqs(case["freqs"]))]
    p["probes"] = [(1, 2, (n[0] - 62, n[1] // 2, 0))]
    p["noise"] = (seed, 1e-3, (0, 1, 5))
    return p


def _wave(case, seed):
    """A block of silicon in a box of an oblique plane wave, E in the plane, a flux box about it."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], 1)
    p = _problem(n, H, [("pml", 12, 12), ("pml", 12, 12), ("periodic",)], 0.5)
    a = rng.uniform(0.15, 0.3, 2)
    p["background"] = 1.0
    p["boxes"] = [((-a[0] * n[0] * H, -a[1] * n[1] * H, -INF), (a[0] * n[0] * H, a[1] * n[1] * H, INF), N_SI2)]
    p["wave"] = ((24, 24, 0), (n[0] - 25, n[1] - 25, 1), (2, 1, 0), (-1.0, 2.0, 0.0), _gauss(1.0 / 1.55, 0.6))
    p["monitors"] = [("flux", 0, 18, ((18, n[1] - 19), None), _freqs(11)),
                     ("flux", 0, n[0] - 19, ((18, n[1] - 19), None), _freqs(11)),
                     ("dft", (24, n[1] // 2, 0), (n[0] - 25, n[1] // 2, 0), _freqs(11))]
    return p


def _bloch(case, seed):
    """Layers across z in a cell with a phase across x and y, a sheet of current above them."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    k = TAU * rng.uniform(0.1, 0.3, 2)
    p = _problem(n, H, [("bloch", float(k[0])), ("bloch", float(k[1])), ("pml", 10, 10)], 0.9)
    p["background"] = 1.0
    top = 0.5 * n[2] * H
    p["boxes"] = [((-INF, -INF, -0.4 * top), (INF, INF, -0.1 * top), 4.0),
                  ((-0.25 * n[0] * H, -0.25 * n[1] * H, -0.1 * top), (0.25 * n[0] * H, 0.25 * n[1] * H, 0.2 * top), N_SI2)]
    z = n[2] - 20
    values = [(0, (i, j, z), complex(np.exp(1j * (k[0] * (i + 0.5) + k[1] * j) * H)))
              for j in range(n[1]) for i in range(n[0])]
    p["currents"] = [(0, values, _gauss(1.0 / 1.55, 0.6))]
    p["monitors"] = [("dft", (0, 0, 14), (n[0] - 1, n[1] - 1, 14), _freqs(5)),
                     ("dft", (0, 0, z - 6), (n[0] - 1, n[1] - 1, z - 6), _freqs(5))]
    p["noise"] = (seed, 1e-2)
    return p


def _mmi(case, seed):
    """A 1 x 2 splitter scaled to the grid: a guide, a body, two arms; a mode-like current, flux
    planes across the arms."""
    rng = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    p = _problem(n, H, [("pml", 10, 10)] * 3, 0.9)
    sx, sy = n[0] / 600.0, n[1] / 200.0
    yc, half = 0.75 * sy, 0.25 * min(1.0, 2 * sy)
    body = float(rng.uniform(3.6, 4.2)) * sx
    core = 0.11
    p["boxes"] = [((-INF, -half, -core), (-body, half, core), N_SI2),
                  ((-body, -1.5 * sy, -core), (body, 1.5 * sy, core), N_SI2),
                  ((body, -yc - half, -core), (INF, -yc + half, core), N_SI2),
                  ((body, yc - half, -core), (INF, yc + half, core), N_SI2)]
    values = []
    for k in range(n[2]):
        for j in range(n[1]):
            y, z = p["origin"][1] + (j + 0.5) * H, p["origin"][2] + k * H
            a = math.exp(-(y / 0.25) ** 2 - (z / 0.15) ** 2)
            if a > 1e-3:
                values.append((1, (35, j, k), a))
    p["currents"] = [(0, values, _gauss(1.0 / 1.55, 0.5))]
    plane = n[0] - 40

    def cells(v, axis):
        return int(round((v - p["origin"][axis]) / H))
    for y in (-yc, yc):
        w = ((max(11, cells(y - 0.5, 1)), min(n[1] - 12, cells(y + 0.5, 1))),
             (max(11, cells(-0.4, 2)), min(n[2] - 12, cells(0.4, 2))))
        p["monitors"].append(("flux", 0, plane, w, _freqs(case["freqs"])))
    p["probes"] = [(0, 1, (plane, cells(yc, 1), n[2] // 2))]
    p["noise"] = (seed, 1e-3, (1, 5))
    return p


def _dispersive(case, seed):
    """Boxes of a Drude metal and of a two-pole Lorentz dielectric over about an eighth of a grid of
    10 nm cells, fields everywhere at the start."""
    rng = np.random.default_rng(seed)
    n, h = (case["nx"], case["ny"], case["nz"]), 0.01
    p = _problem(n, h, [("pml", 10, 10)] * 3, 0.5)
    p["background"] = 1.0
    lo = np.array(p["origin"]) + 12 * h
    size = np.array(n) * h - 24 * h
    groups, filled = ([], []), 0.0
    while filled < 0.12:
        s = rng.uniform(0.05, 0.3, 3)
        at = lo + rng.uniform(0, 1 - s) * size
        groups[int(rng.random() < 0.5)].append((tuple(at), tuple(at + s * size), 1.0))
        filled += float(np.prod(s))
    plasma, damping = 1.37e16 / TAU / C_UM_PER_S, 1e14 / TAU / C_UM_PER_S
    lorentz = [(float(rng.uniform(0.5, 2.0)), 1.0 / float(rng.uniform(1.0, 3.0)), 0.01) for _ in range(2)]
    p["media"] = [(1.0, [("drude", plasma, damping)], groups[0]),
                  (2.25, [("lorentz",) + q for q in lorentz], groups[1])]
    p["points"] = [(0, 2, tuple(m // 2 for m in n), _gauss(1.0 / 1.6, 1.0 / 1.2 - 1.0 / 2.0))]
    p["noise"] = (seed, 0.01)
    return p


def _flat(n, freqs, seed, pml=12, noise=0.0):
    """One 2D design: a guide through random patches, a line current, a flux plane a little after it
    (so that a pass of some hundred steps sees the pulse there)."""
    rng = np.random.default_rng(seed)
    p = _problem((n[0], n[1], 1), H, [("pml", pml, pml), ("pml", pml, pml), ("periodic",)], 0.5)
    a = rng.uniform(0.5, 0.95, 2)
    p["boxes"] = [((-INF, -0.25, -INF), (INF, 0.25, INF), N_SI2),
                  ((-0.6, -a[0], -INF), (-0.05, a[0], INF), N_SI2),
                  ((0.05, -a[1], -INF), (0.7, a[1], INF), float(rng.uniform(2.2, 12.0)))]
    jc = n[1] // 2
    values = [(1, (pml + 20, j, 0), math.exp(-((j + 0.5 - n[1] / 2) * H / 0.25) ** 2))
              for j in range(jc - 20, jc + 20)]
    p["currents"] = [(0, values, _gauss(1.0 / 1.55, 1.2))]
    p["monitors"] = [("flux", 0, min(n[0] - pml - 16, pml + 80), ((jc - 20, jc + 20), None), _freqs(freqs))]
    if noise:
        p["noise"] = (seed, noise, (0, 1, 5))
    return p


def _sides(case, seed):
    """The batch's grids: their sides log-uniform, the same for every seed (an ensemble's sizes are
    part of the case)."""
    rng = np.random.default_rng(7)
    sides = [tuple(int(v) for v in np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), 2)))
             for _ in range(case["count"])]
    return [(a - a % 4, b) if case["quad"] else (a, b) for a, b in sides]


def _jobs(case, seed):
    """The burst's problems: 2D and 3D, cells log-uniform, as the serving stream draws them."""
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(11)
    out = []
    for q in range(case["flat"] + case["solid"]):
        c = math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))
        aspect = sizes.uniform(0.5, 2.0)
        two_d = q < case["flat"]
        nz = 1 if two_d else max(24, int(round((c / 8.0) ** (1 / 3))))
        nx = max(80, int(round(math.sqrt(c / nz * aspect))))
        nx -= nx % 4
        ny = max(64, int(round(c / nz / nx)))
        if two_d:
            out.append(_flat((nx, ny), case["freqs"], int(rng.integers(1 << 30)), pml=10))
            continue
        p = _problem((nx, ny, nz), H, [("pml", 10, 10)] * 3, 0.5)
        x, y = rng.uniform(-0.5, 0.1, 2)
        p["boxes"] = [((float(x), float(y), -INF), (float(x + 0.4), float(y + 0.3), INF), N_SI2)]
        p["points"] = [(0, 1, (16, ny // 2, nz // 2), _gauss(1.0 / 1.55, 1.2))]
        p["monitors"] = [("flux", 0, min(nx - 16, 64), None, _freqs(case["freqs"]))]
        out.append(p)
    return out


_ONE = {"block": _block, "strip": _strip, "wave": _wave, "bloch": _bloch, "mmi": _mmi,
        "dispersive": _dispersive}


def _noise(p, field, c):
    """The initial values of one component (None: zero)."""
    if p["noise"] is None or (len(p["noise"]) > 2 and 3 * field + c not in p["noise"][2]):
        return None
    rng = np.random.default_rng([p["noise"][0], field, c])
    cells = p["n"][0] * p["n"][1] * p["n"][2]
    return p["noise"][1] * (2.0 * rng.random(cells) - 1.0)


def _simulation(p, bits):
    """The problem through the package's API."""
    g = Grid3d(*p["n"], p["h"], p["h"], p["h"], *p["origin"])
    sides = [Periodic() if e[0] == "periodic" else Bloch(e[1]) if e[0] == "bloch" else Pml(e[1], e[2])
             for e in p["edges"]]
    eps = Boxes(p["background"])
    for lo, hi, v in p["boxes"]:
        eps.add(lo, hi, v)
    s = Simulation(g, eps, Boundaries(*sides, Cpml(kappa=p["cpml"][0], alpha=p["cpml"][1])),
                   p["courant"], precision=bits)
    if p["sigma"]:
        s.with_conductivity(Boxes(0.0, list(p["sigma"])))
    for eps_inf, poles, boxes in p["media"]:
        s.with_medium(Dispersive(eps_inf, [Pole.drude(*q[1:]) if q[0] == "drude" else Pole.lorentz(*q[1:])
                                           for q in poles]), Boxes(0.0, list(boxes)))
    for field in range(2):
        for c in range(3):
            v = _noise(p, field, c)
            if v is not None:
                s.set_field(Field(field), Axis(c), v)
    for field, c, at, w in p["points"]:
        s.add_source(Source(Field(field), Axis(c), at, Waveform.gaussian(*w)))
    for field, values, w in p["currents"]:
        s.add_current(Current(Field(field), [(Axis(c), at, complex(a)) for c, at, a in values],
                              Waveform.gaussian(*w)))
    if "wave" in p:
        lo, hi, direction, polarization, w = p["wave"]
        s.add_plane_wave(PlaneWave(lo, hi, direction, polarization, p["background"], Waveform.gaussian(*w)))
    for field, c, at in p["probes"]:
        s.add_probe(Field(field), Axis(c), at)
    for m in p["monitors"]:
        if m[0] == "dft":
            s.add_dft(m[1], m[2], m[3])
        else:
            plane = FluxPlane(Axis(m[1]), m[2])
            s.add_flux(plane if m[3] is None else FluxPlane(Axis(m[1]), m[2], m[3]), m[4])
    return s


# -- the passes -------------------------------------------------------------------------------------

class _OnDevice:
    """A simulation's device array for torch.as_tensor, which takes it without a copy and holds on
    to this object, and so to the simulation that owns the memory."""

    def __init__(self, sim, address, shape, bits):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f%d" % (bits // 8),
                                         "data": (address, False), "version": 3, "strides": None}


def _fields(sim, bits):
    """E and H as the engine holds them, (3, cells) each, valid until the next run."""
    e, h = ctypes.c_void_p(), ctypes.c_void_p()
    sim._check(library().fdtd_device_fields(ctypes.c_void_p(sim.engine()), ctypes.byref(e), ctypes.byref(h)))
    shape = (3, sim.grid.cells())
    return [torch.as_tensor(_OnDevice(sim, q.value, shape, bits), device="cuda") for q in (e, h)]


def prepare(case, seed):
    kind, bits = case["kind"], case["bits"]
    state = {"case": case}
    if kind in _ONE:
        state["sim"] = _simulation(_ONE[kind](case, seed), bits)
    elif kind == "batch":
        state["sims"] = [_simulation(_flat(n, case["freqs"], 1000 * seed + q, noise=0.01), bits)
                         for q, n in enumerate(_sides(case, seed))]
        state["batch"] = Batch(state["sims"])
    elif kind == "adjoint":
        state["problem"] = configs.te_design(case["nx"], case["ny"], precision=bits, steps=case["steps"],
                                             segment=case["segment"], design_cells=case["design"])
        state["eps"] = torch.tensor(_design(case, seed), requires_grad=True)
    else:
        state["jobs"] = _jobs(case, seed)
    return state


def _design(case, seed):
    d = case["design"]
    return N_SIO2 + np.random.default_rng(seed).uniform(0, 1, (d, d)) * (N_SI2 - N_SIO2)


def run(state):
    case = state["case"]
    steps, bits = case["steps"], case["bits"]
    if "sim" in state:
        sim = state["sim"]
        sim.run(steps)
        out = {"fields": _fields(sim, bits)}
        if case["kind"] != "dispersive":
            out["sums"] = sim.transforms()
        return out
    if "batch" in state:
        state["batch"].run(steps)
        sums = np.concatenate([s.transforms() for s in state["sims"]])
        fields = [_fields(s, bits) for s in state["sims"]]
        return {"sums": sums, "e": torch.cat([f[0].reshape(-1) for f in fields]),
                "h": torch.cat([f[1].reshape(-1) for f in fields])}
    if "problem" in state:
        eps = state["eps"]
        eps.grad = None
        flux = TeFlux.apply(eps, state["problem"])
        flux.sum().backward()
        return {"flux": flux.detach(), "gradient": eps.grad}
    # a served program makes its simulations as jobs arrive, hands them over and reads the results
    with Server() as server:
        jobs = [server.submit(_simulation(p, bits), steps, keep_fields=False) for p in state["jobs"]]
        for j in jobs:
            j.wait()
        return {"sums": [j.sim.transforms() for j in jobs]}


# -- what a pass cannot do without --------------------------------------------------------------------

def _count(p, bits):
    """(bytes and operations of one step, resident bytes) of a problem: E and H read and written and
    cb read (TE grids: three components and two), CPML psi, media's state read and written, the
    monitored values read; 51 operations a cell (17 in TE), 8 a psi, 4 a monitored value and
    frequency, 12 a media value and pole."""
    n, r = p["n"], bits // 8
    cells = n[0] * n[1] * n[2]
    te = n[2] == 1
    psi = sum((4 if not te else 2) * (e[1] + e[2]) * (cells // n[a])
              for a, e in enumerate(p["edges"]) if e[0] == "pml")
    comps = 3 if te else 6
    per_step = (2 * comps + (2 if te else 3)) * r * cells + 2 * r * psi
    flops = (17 if te else 51) * cells + 8 * psi
    if p["sigma"] or p["media"]:
        per_step += 3 * r * cells
    for _, poles, boxes in p["media"]:
        inside = sum(float(np.prod(np.subtract(b[1], b[0]))) for b in boxes) / p["h"] ** 3
        inside = 3 * min(inside, 0.2 * cells)
        per_step += inside * r * (2 + 4 * len(poles))
        flops += 12 * inside * len(poles)
    for m in p["monitors"]:
        if m[0] == "dft":
            values = 6 * int(np.prod([m[2][a] - m[1][a] + 1 for a in range(3)])) * (0.5 if te else 1)
            nf = len(m[3])
        else:
            b, c = (m[1] + 1) % 3, (m[1] + 2) % 3
            spans = [n[a] if not m[3] or m[3][q] is None else m[3][q][1] - m[3][q][0] + 1
                     for q, a in enumerate((b, c))]
            values, nf = (3 if te else 6) * spans[0] * spans[1], len(m[4])
        flops += 4 * values * nf
    if any(e[0] == "bloch" for e in p["edges"]):
        per_step, flops = 2 * per_step, 2 * flops
    return per_step, flops, per_step


ON_CHIP = 126e6  # bytes that stay on the chip between steps (its last-level cache)


def _work(problems, bits, steps):
    """Grids that stay on the chip between steps have to be read and written once a pass, larger ones
    once a step."""
    parts = [_count(p, bits) for p in problems]
    step, flops = sum(q[0] for q in parts), sum(q[1] for q in parts)
    return {"bytes": float(step * (1 if step <= ON_CHIP else steps)), "flops": float(flops * steps)}


def work(case):
    kind, bits, steps = case["kind"], case["bits"], case["steps"]
    if kind in _ONE:
        return _work([_ONE[kind](case, 0)], bits, steps)
    if kind == "batch":
        return _work([_flat(n, case["freqs"], 0) for n in _sides(case, 0)], bits, steps)
    if kind == "serving":
        return _work(_jobs(case, 0), bits, steps)
    p = _flat((case["nx"], case["ny"]), 1, 0)
    # the forward steps, and back through them their transpose (the fields' history kept or remade)
    w = _work([p], bits, steps)
    return {"bytes": 3 * w["bytes"], "flops": 3 * w["flops"]}


# -- the same in 64 bits, in plain torch ----------------------------------------------------------------

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _inside(axis_positions, boxes):
    """Per box, which of each axis' positions it holds (open intervals)."""
    return [[(pos > lo[a]) & (pos < hi[a]) for a, pos in enumerate(axis_positions)] for lo, hi, _ in boxes]


def _value(axis_positions, background, boxes):
    """The boxes' value at every point of a grid of positions, (z, y, x); later boxes on top."""
    x, y, z = axis_positions
    v = torch.full((z.numel(), y.numel(), x.numel()), float(background), dtype=torch.float64, device=DEVICE)
    for (ix, iy, iz), (_, _, val) in zip(_inside(axis_positions, boxes), boxes):
        v = torch.where(iz[:, None, None] & iy[None, :, None] & ix[None, None, :], float(val), v)
    return v


def _positions(p, c):
    """Component c of E's positions along each axis."""
    out = []
    for a in range(3):
        i = torch.arange(p["n"][a], dtype=torch.float64, device=DEVICE)
        out.append(p["origin"][a] + i * p["h"] + (0.5 * p["h"] if a == c else 0.0))
    return out


def _average(p, c):
    """The cell average at component c of E: over 8 x 8 x 8 points of the cell about the value, the
    harmonic mean along c, its arithmetic mean across."""
    pos = _positions(p, c)
    off = [((s + 0.5) / 8.0 - 0.5) * p["h"] for s in range(8)]
    b, d = (c + 1) % 3, (c + 2) % 3
    total = None
    for sb in off:
        for sd in off:
            inverse = 0.0
            for sa in off:
                at = list(pos)
                at[c], at[b], at[d] = pos[c] + sa, pos[b] + sb, pos[d] + sd
                inverse = inverse + 1.0 / _value(at, p["background"], p["boxes"])
            v = 8.0 / inverse
            total = v if total is None else total + v
    return total / 64.0


def _shift(f, a, forward, edge):
    """The neighbour along axis a of every value: zero beyond a wall, across a periodic side the other
    end's, across a Bloch side that times the phase."""
    dim = 2 - a
    out = torch.roll(f, -1 if forward else 1, dim)
    last = out.narrow(dim, f.shape[dim] - 1 if forward else 0, 1)
    if edge[0] == "pml":
        last.zero_()
    elif edge[0] == "bloch":
        last.mul_(complex(math.cos(edge[2]), math.sin(edge[2])) if forward
                  else complex(math.cos(edge[2]), -math.sin(edge[2])))
    return out


def _pulse(w, t):
    """A current's complex waveform; its real part is the point source's."""
    u = (t - w[2]) / w[1]
    g = math.exp(-u * u)
    a = TAU * w[0] * (t - w[2])
    return complex(g * math.sin(a), g * math.cos(a))


class _Plain:
    """Yee's scheme with CPMLs, Drude and Lorentz media and running transforms, in 64 bits."""

    def __init__(self, p):
        self.p, n, h = p, p["n"], p["h"]
        self.bloch = any(e[0] == "bloch" for e in p["edges"])
        self.kind = torch.complex128 if self.bloch else torch.float64
        self.edges = [e if e[0] != "bloch" else (e[0], e[1], e[1] * n[a] * h) for a, e in enumerate(p["edges"])]
        self.shape = (n[2], n[1], n[0])
        self.te = n[2] == 1 and not any(3 * q[0] + q[1] in (2, 3, 4) for q in p["points"])
        self.on = [0, 1, 5] if self.te else list(range(6))  # the components that move
        # an axis a cell long between periodic sides has no differences (a phase would give some)
        self.flat = [n[a] == 1 and p["edges"][a][0] == "periodic" for a in range(3)]
        self.dt = p["courant"] / math.sqrt(sum(1.0 / h ** 2 for a in range(3) if not self.flat[a]))
        self._medium()
        self._cpml()
        self.f = []
        for q in range(6):
            v = _noise(p, q // 3, q % 3)
            z = torch.zeros(self.shape, dtype=self.kind, device=DEVICE)
            self.f.append(z if v is None else z + torch.tensor(v, device=DEVICE).reshape(self.shape))
        self._monitors()
        self.step = 0

    def _medium(self):
        p, dt = self.p, self.dt
        self.ca, self.cb, self.media = [], [], []
        for c in range(3):
            if c not in self.on:
                self.ca.append(None), self.cb.append(None)
                continue
            cb = dt / _average(p, c)
            ca = torch.ones_like(cb)
            held = torch.zeros(self.shape, dtype=torch.bool, device=DEVICE)
            for a in range(3):
                if a != c and p["edges"][a][0] == "pml":
                    held.narrow(2 - a, 0, 1).fill_(True)
            if p["sigma"]:
                half = _value(_positions(p, c), 0.0, p["sigma"]) * cb / 2.0
                ca, cb = (1.0 - half) / (1.0 + half), cb / (1.0 + half)
            self.ca.append(torch.where(held, 0.0, ca))
            self.cb.append(torch.where(held, 0.0, cb))
        groups = []
        for eps_inf, poles, boxes in p["media"]:
            co = []
            for q in poles:
                if q[0] == "drude":
                    a, w0sq, gamma = (TAU * q[1]) ** 2, 0.0, TAU * q[2]
                else:
                    w0 = TAU * q[2]
                    a, w0sq, gamma = q[1] * w0 * w0, w0 * w0, TAU * q[3]
                d = 1.0 + gamma * dt / 2.0
                co.append(((2.0 - w0sq * dt * dt) / d, (gamma * dt / 2.0 - 1.0) / d, a * dt * dt / d))
            groups.append((eps_inf, co, sum(q[2] for q in co) / (4.0 * dt), boxes))
        for c in range(3 if groups else 0):
            which = torch.full(self.shape, -1, device=DEVICE)
            for g, (_, _, _, boxes) in enumerate(groups):
                which = torch.where((_value(_positions(p, c), 0.0, boxes) != 0.0) & (self.cb[c] != 0.0), g, which)
            for g, (eps_inf, co, chi, _) in enumerate(groups):
                at = (which == g).reshape(-1).nonzero()[:, 0]
                nu = 1.0 + dt / eps_inf * chi
                self.ca[c].view(-1)[at] = 1.0 / nu
                self.cb[c].view(-1)[at] = dt / eps_inf / nu
                zeros = torch.zeros((len(co), at.numel()), dtype=self.kind, device=DEVICE)
                self.media.append({"c": c, "at": at, "co": co, "chi": chi, "scale": dt / eps_inf / nu,
                                   "before": torch.zeros(at.numel(), dtype=self.kind, device=DEVICE),
                                   "now": zeros, "last": zeros.clone()})

    def _cpml(self):
        p, h = self.p, self.p["h"]
        kappa_max, alpha = p["cpml"]
        self.factor = [[None] * 3, [None] * 3]  # per field, axis: kappa/h along it
        self.slabs = [[], []]  # per field: component, axis, side and the recursion there
        for a, e in enumerate(p["edges"]):
            n = p["n"][a]
            lo, hi = (e[1], e[2]) if e[0] == "pml" else (0, 0)
            for field in range(2):
                m = np.arange(n) + (0.5 if field else 0.0)
                x, thick = np.zeros(n), np.ones(n)
                if lo:
                    x[m < lo], thick[m < lo] = ((lo - m) / lo)[m < lo], lo * h
                if hi:
                    x[m > n - hi], thick[m > n - hi] = ((m - (n - hi)) / hi)[m > n - hi], hi * h
                x = np.clip(x, 0, 1) ** 3
                sigma = 4.0 * -math.log(1e-8) / (2.0 * thick) * x
                kappa = 1.0 + (kappa_max - 1.0) * x
                b = np.exp(-(sigma / kappa + alpha) * self.dt)
                den = sigma * kappa + kappa * kappa * alpha
                aa = np.where((sigma > 0) & (den > 0), sigma * (b - 1.0) / np.where(den > 0, den, 1.0), 0.0)
                view = [1, 1, 1]
                view[2 - a] = -1
                self.factor[field][a] = torch.tensor(1.0 / kappa / h, device=DEVICE).view(view)
                for start, count in ((0, lo), (n - hi, hi)):
                    for c in range(3):
                        if count == 0 or c == a or 3 * field + c not in self.on:
                            continue
                        shape = list(self.shape)
                        shape[2 - a] = count
                        s = slice(start, start + count)
                        self.slabs[field].append({"c": c, "a": a, "start": start, "count": count,
                                                  "b": torch.tensor(b[s], device=DEVICE).view(view),
                                                  "k": torch.tensor(aa[s], device=DEVICE).view(view),
                                                  "psi": torch.zeros(shape, dtype=self.kind, device=DEVICE)})

    def _monitors(self):
        self.series = []  # field, component, slices, frequencies, sums
        for m in self.p["monitors"]:
            if m[0] == "dft":
                parts = [(f, c, m[1], [m[2][a] - m[1][a] + 1 for a in range(3)], m[3])
                         for f in range(2) for c in range(3)]
            else:
                axis, plane, window, freqs = m[1:]
                bc = ((axis + 1) % 3, (axis + 2) % 3)
                lo, length = [0, 0, 0], [0, 0, 0]
                lo[axis] = plane
                for q, a in enumerate(bc):
                    w = None if window is None else window[q]
                    lo[a], length[a] = (0, self.p["n"][a]) if w is None else (w[0], w[1] + 1 - w[0])
                parts = []
                for f in range(2):
                    length[axis] = 2 if f == 0 else 1
                    parts += [(f, c, tuple(lo), list(length), freqs) for c in bc]
            for f, c, lo, length, freqs in parts:
                cut = tuple(slice(lo[a], lo[a] + length[a]) for a in (2, 1, 0))
                om = torch.tensor([TAU * q for q in freqs], dtype=torch.float64, device=DEVICE)
                sums = torch.zeros([len(freqs)] + [length[a] for a in (2, 1, 0)], dtype=torch.complex128, device=DEVICE)
                self.series.append((f, c, cut, om, sums))
        self.values = []
        for field, values, w in self.p["currents"]:
            n = self.p["n"]
            for c in sorted({q[0] for q in values}):
                mine = [q for q in values if q[0] == c]
                at = torch.tensor([(q[1][2] * n[1] + q[1][1]) * n[0] + q[1][0] for q in mine], device=DEVICE)
                self.values.append((field, c, at, torch.tensor([complex(q[2]) for q in mine], dtype=torch.complex128, device=DEVICE), w))

    def _half(self, field):
        """One field's update: H from E's forward differences, E from H's back ones."""
        other, p = (0, 3) if field else (3, 0), self.p
        src = 0 if field else 3
        t = self.step * self.dt + (0.0 if field else 0.5 * self.dt)
        diff = {}
        for c in range(3):
            if 3 * field + c not in self.on:
                continue
            for a in range(3):
                d = 3 - c - a
                if a == c or src + d not in self.on or self.flat[a]:
                    continue
                f = self.f[src + d]
                g = _shift(f, a, bool(field), self.edges[a])
                diff[c, a] = g - f if field else f - g
        for c in range(3):
            if 3 * field + c not in self.on:
                continue
            curl = 0.0
            for a in range(3):
                if (c, a) in diff:
                    sign = 1.0 if a == (c + 1) % 3 else -1.0
                    curl = curl + sign * diff[c, a] * self.factor[field][a]
            k = 3 * field + c
            self.f[k] = self.f[k] - self.dt * curl if field else self.ca[c] * self.f[k] + self.cb[c] * curl
        for s in self.slabs[field]:
            c, a = s["c"], s["a"]
            if (c, a) not in diff:
                continue
            sign = 1.0 if a == (c + 1) % 3 else -1.0
            s["psi"] = s["b"] * s["psi"] + s["k"] * diff[c, a].narrow(2 - a, s["start"], s["count"]) / p["h"]
            v = self.f[3 * field + c].narrow(2 - a, s["start"], s["count"])
            if field:
                v -= self.dt * sign * s["psi"]
            else:
                v += self.cb[c].narrow(2 - a, s["start"], s["count"]) * sign * s["psi"]
        for f, c, at, w in p["points"]:
            if f == field:
                i = (at[2], at[1], at[0])
                amount = _pulse(w, t).real
                self.f[3 * f + c][i] -= (self.dt if f else self.cb[c][i]) * amount
        for f, c, at, amp, w in self.values:
            if f == field:
                v = amp * _pulse(w, t)
                v = v if self.bloch else v.real
                self.f[3 * f + c].view(-1)[at] -= (self.dt if f else self.cb[c].reshape(-1)[at]) * v

    def run(self, steps):
        for _ in range(steps):
            self._half(1)
            old = [self.f[m["c"]].reshape(-1)[m["at"]] for m in self.media]
            self._half(0)
            for m, e_old in zip(self.media, old):
                v = self.f[m["c"]].view(-1)
                rest = m["chi"] * m["before"]
                for q, (al, xi, _) in enumerate(m["co"]):
                    rest = rest - 0.5 * ((al + 1.0) * m["now"][q] + xi * m["last"][q])
                new = v[m["at"]] + m["scale"] * rest
                slope = (new - m["before"]) / (2.0 * self.dt)
                j = torch.stack([al * m["now"][q] + xi * m["last"][q] + ga * slope
                                 for q, (al, xi, ga) in enumerate(m["co"])])
                m["last"], m["now"], m["before"] = m["now"], j, e_old
                v[m["at"]] = new
            self.step += 1
            for f, c, cut, om, sums in self.series:
                if 3 * f + c not in self.on:
                    continue
                t = self.step * self.dt - (0.5 * self.dt if f else 0.0)
                ph = torch.polar(torch.full_like(om, self.dt), om * t)
                sums += ph.view(-1, 1, 1, 1) * self.f[3 * f + c][cut]
        return self

    def fields(self):
        return [torch.stack([q.real.reshape(-1) for q in self.f[k:k + 3]]) for k in (0, 3)]

    def sums(self):
        return torch.cat([s[4].reshape(-1) for s in self.series]).cpu().numpy()


def _plain_adjoint(case, seed):
    """The design's flux and its gradient by autograd through every step of the 2D TE run."""
    nx, ny, d = case["nx"], case["ny"], case["design"]
    n = (nx, ny, 1)
    half = 0.5 * d * H
    p = _problem(n, H, [("pml", 12, 12), ("pml", 12, 12), ("periodic",)], 0.5, origin=(-0.5 * nx * H, -0.5 * ny * H, -H / 2))
    p["boxes"] = [((-INF, -0.25, -INF), (-half, 0.25, INF), N_SI2), ((half, -0.25, -INF), (INF, 0.25, INF), N_SI2)]
    g = _Plain(p)
    dt = g.dt
    cells = torch.tensor(_design(case, seed), device=DEVICE, requires_grad=True)
    x0, y0 = nx // 2 - d // 2, ny // 2 - d // 2
    full = torch.nn.functional.pad(cells, (x0, nx - x0 - d, y0, ny - y0 - d))
    share = torch.nn.functional.pad(torch.ones_like(cells), (x0, nx - x0 - d, y0, ny - y0 - d))

    def over(v, dim):  # half of the cell before and half of the cell, across the component
        return 0.5 * (v + torch.roll(v, 1, dim))
    cb = []
    for c, dim in ((0, 0), (1, 1)):
        base = dt / g.cb[c][0]
        eps = torch.where(g.cb[c][0] == 0, base, torch.where(torch.isfinite(base), base, 1.0) * (1.0 - over(share, dim)) + over(full, dim))
        cb.append(torch.where(g.cb[c][0] == 0, 0.0, dt / eps))
    ca = [g.ca[0][0], g.ca[1][0]]
    fh = [g.factor[1][0].reshape(1, -1), g.factor[1][1].reshape(-1, 1)]
    fe = [g.factor[0][0].reshape(1, -1), g.factor[0][1].reshape(-1, 1)]
    slab = {}
    for field in range(2):
        for s in g.slabs[field]:
            key = (field, s["a"])
            b, k = slab.setdefault(key, [torch.zeros(nx if s["a"] == 0 else ny, dtype=torch.float64, device=DEVICE) for _ in range(2)])
            b[s["start"]:s["start"] + s["count"]] = s["b"].reshape(-1)
            k[s["start"]:s["start"] + s["count"]] = s["k"].reshape(-1)
    view = {0: (1, -1), 1: (-1, 1)}
    psi = {q: torch.zeros((ny, nx), dtype=torch.float64, device=DEVICE) for q in slab}
    co = {q: [v.view(view[q[1]]) for v in vv] for q, vv in slab.items()}
    ex, ey, hz = (torch.zeros((ny, nx), dtype=torch.float64, device=DEVICE) for _ in range(3))
    jc = ny // 2
    rows = torch.arange(jc - 25, jc + 26, device=DEVICE)
    profile = torch.zeros((ny, nx), dtype=torch.float64, device=DEVICE)
    profile[rows, 37] = torch.exp(-(((rows.double() + 0.5 - ny / 2) * H) / 0.25) ** 2)
    wave = _gauss(1.0 / 1.55, 0.3)
    plane = nx - 37
    lo, hi = max(jc - 50, 13), min(jc + 50, ny - 14)
    weight = torch.ones(hi + 1 - lo, dtype=torch.float64, device=DEVICE)
    weight[0] = weight[-1] = 0.5
    om = TAU / 1.55
    ef = torch.zeros((hi + 1 - lo, 2), dtype=torch.complex128, device=DEVICE)
    hf = torch.zeros(hi + 1 - lo, dtype=torch.complex128, device=DEVICE)
    pad = torch.nn.functional.pad
    for m in range(case["steps"]):
        t = m * dt
        dx = pad(ey, (0, 1))[:, 1:] - ey
        dy = pad(ex, (0, 0, 0, 1))[1:] - ex
        psi[1, 0] = co[1, 0][0] * psi[1, 0] + co[1, 0][1] * dx / H
        psi[1, 1] = co[1, 1][0] * psi[1, 1] + co[1, 1][1] * dy / H
        hz = hz - dt * (dx * fh[0] - dy * fh[1] + psi[1, 0] - psi[1, 1])
        dx = hz - pad(hz, (1, 0))[:, :-1]
        dy = hz - pad(hz, (0, 0, 1, 0))[:-1]
        psi[0, 0] = co[0, 0][0] * psi[0, 0] + co[0, 0][1] * dx / H
        psi[0, 1] = co[0, 1][0] * psi[0, 1] + co[0, 1][1] * dy / H
        ex = ca[0] * ex + cb[0] * (dy * fe[1] + psi[0, 1])
        ey = ca[1] * ey - cb[1] * (dx * fe[0] + psi[0, 0]) - cb[1] * profile * _pulse(wave, t + 0.5 * dt).real
        te = (m + 1) * dt
        ef = ef + ey[lo:hi + 1, plane:plane + 2] * (dt * complex(math.cos(om * te), math.sin(om * te)))
        th = te - 0.5 * dt
        hf = hf + hz[lo:hi + 1, plane] * (dt * complex(math.cos(om * th), math.sin(om * th)))
    mean = 0.5 * (ef[:, 0] + ef[:, 1])
    flux = (0.5 * weight * (mean * hf.conj()).real).sum() * H * H
    flux.backward()
    return {"flux": flux.detach().reshape(1), "gradient": cells.grad}


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "adjoint":
        return _plain_adjoint(case, seed)
    if kind == "wave":
        # the incident wave on the grid is a 1D run of the library's own making: nothing plain gives it
        return None
    with torch.no_grad():
        if kind in _ONE:
            s = _Plain(_ONE[kind](case, seed)).run(steps)
            out = {"fields": s.fields()}
            if kind != "dispersive":
                out["sums"] = s.sums()
            return out
        if kind == "batch":
            every = [_Plain(_flat(n, case["freqs"], 1000 * seed + q, noise=0.01)).run(steps) for q, n in enumerate(_sides(case, seed))]
            fields = [s.fields() for s in every]
            return {"sums": np.concatenate([s.sums() for s in every]),
                    "e": torch.cat([f[0].reshape(-1) for f in fields]), "h": torch.cat([f[1].reshape(-1) for f in fields])}
        return {"sums": [_Plain(p).run(steps).sums() for p in _jobs(case, seed)]}
