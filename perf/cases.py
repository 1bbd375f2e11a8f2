"""The work that a program has this library do, as cases that can be timed and compared.

A program builds a case from a deck, keeps its handle and calls `Case.step(n)` for as long as the discharge
runs; it does so for one case, for a batch of cases, or hands decks to a server and takes the results.  The
cases below are those three forms and the stand-alone deposit, over the range of the decks in
hpic/workloads.py, bench.py and the tests: 33x17 to 513x257 nodes (cells of 312.5 um), 10 to 200 macro-particles
per cell and species, the three gases, the three field solves, and the options a run is made with (energy
distribution, smoothing, circuit, dielectric electrode).  Every case is a running one: it has passed its first
averaging window, so that the continuity solve of the fluid species is part of its steps.

The state of a case stays on the device between calls, as in a program; what `run` returns are views of that
state (`OnDevice`), which copy a field to the host when it is looked up.
"""
import ctypes
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hybrid-final_b200"))

import hpic  # noqa: E402
from hpic.decks import ccp_deck  # noqa: E402
from hpic.workloads import batched_cases, served_stream  # noqa: E402

CELL = 3.125e-4  # m, the cell of every benchmark deck

SPECIES = {"Ar": 2, "O2": 4, "ArO2": 5}
# particles of all species per unit of `ppc` (the decks load the ions at these fractions of the electrons)
LOAD = {"Ar": 2.0, "O2": 2.2, "ArO2": 2.4}
ION_DENSITY = {
    "O2": {"O2+": 1e15, "O+": 1e14, "O-": 1e14},
    "ArO2": {"Ar+": 1e15, "O2+": 2e14, "O+": 0.0, "O-": 2e14},
}


def step_case(name, nx, ny, ppc, steps, gas="Ar", field_mode=2, volts=100.0, mtorr=50.0, eedf=0, smooth=0,
              circuit=False, dielectric=False, all_species=0, room=8):
    c = dict(kind="step", nx=nx, ny=ny, ppc=ppc, steps=steps, gas=gas, field_mode=field_mode, volts=volts, mtorr=mtorr,
             eedf=eedf, smooth=smooth, circuit=circuit, dielectric=dielectric, all_species=all_species, room=room)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest grid of the batched workload at its smallest load: a step is launches and latency
        step_case("step_ar_65x33_20ppc", 65, 33, 20, 100),
        # the CPU-sized benchmark case (bench.py ar_129x65_50ppc)
        step_case("step_ar_129x65_50ppc", 129, 65, 50, 50),
        # odd sizes, with the options of a diagnosed run: energy distribution, one smoothing pass, R-L-C circuit
        step_case("step_ar_191x94_85ppc_diag", 191, 94, 85, 20, volts=160.0, mtorr=80.0, eedf=4, smooth=1,
                  circuit=True),
        # the large precision-form case (bench.py's default workload): the particle kernels' bandwidth and rates
        step_case("step_ar_513x257_200ppc", 513, 257, 200, 10, room=4),
        # the Ar/O2 mixture (bench.py aro2_257x129_100ppc): five species, 68 collision channels
        step_case("step_aro2_257x129_100ppc", 257, 129, 100, 20, gas="ArO2", volts=200.0, mtorr=100.0, room=4),
        # an oxygen discharge in which every species collides
        step_case("step_o2_129x65_60ppc", 129, 65, 60, 30, gas="O2", volts=200.0, mtorr=100.0, all_species=1),
        # the reference's own solver rule, the library's default: FP32 Jacobi-PCG to its absolute tolerance
        step_case("step_ar_129x65_50ppc_pcg", 129, 65, 50, 4, field_mode=0),
        # a dielectric-covered electrode: the operator is not separable, so FP64 refinement around PCG
        step_case("step_ar_129x65_30ppc_diel", 129, 65, 30, 2, field_mode=1, volts=200.0, dielectric=True, room=16),
        # the reference's rule on the largest grid, where the solve takes the whole GPU
        step_case("step_ar_513x257_20ppc_pcg", 513, 257, 20, 2, field_mode=0),
        # the batched form: mixed grids, pressures, voltages and loads in one batch
        dict(name="batch_ar_24_mixed", kind="batch", n=24, mix=2024, steps=10),
        # the served form, from the decks' text to the averaged results on the host: set-up, admission, steps
        dict(name="serve_6_mixed", kind="serve", n=6, mix=7, scale=0.2, slots=4, largest=129),
        # the densities into a caller's buffer, for a program that owns the device memory
        dict(name="deposit_ar_201x99_150ppc", kind="deposit", nx=201, ny=99, ppc=150),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["batch", "serve", "deposit"])
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(2, 24), mix=rng.randrange(1, 10 ** 6), steps=rng.randint(4, 10))
    if kind == "serve":
        return dict(kind="serve", n=rng.randint(1, 6), mix=rng.randrange(1, 10 ** 6), scale=0.2,
                    slots=rng.randint(1, 6), largest=rng.choice([65, 129]))
    nx = int(round(33 * (513 / 33) ** rng.random()))
    ny = max(17, min(257, int(round(nx * rng.uniform(0.4, 0.6)))))
    ppc = int(round(10 * 20 ** rng.random()))
    if kind == "deposit":
        while nx * ny > 201 * 99:
            nx, ny = nx * 3 // 4, ny * 3 // 4
        return dict(kind="deposit", nx=nx, ny=ny, ppc=ppc)
    gas = rng.choice(["Ar", "Ar", "Ar", "ArO2", "O2"])
    mode = rng.choice([2, 2, 2, 2, 0, 1])
    diel = mode == 1 and rng.random() < 0.6
    if mode == 1:
        nx, ny = min(nx, 141), min(ny, 71)
    if gas != "Ar":
        while nx * ny * ppc > 257 * 129 * 100:
            ppc = max(10, ppc * 3 // 4)
            nx, ny = max(33, nx * 9 // 10), max(17, ny * 9 // 10)
    # passes of a few milliseconds: many steps of a small case, few of a large one or of an iterative solve
    cost = 80.0 + nx * ny * ppc * LOAD[gas] * (3e-5 if gas == "Ar" else 9e-5) + (0.0, 10.0, 20.0)[(2 - mode) % 3] * nx
    steps = max(2, min(100, int(7000.0 / cost)))
    return step_case(None, nx, ny, ppc, steps, gas=gas, field_mode=mode, volts=round(rng.uniform(50.0, 300.0), 1),
                     mtorr=round(10.0 * 20.0 ** rng.random(), 1), eedf=rng.choice([0, 0, 4]),
                     smooth=rng.choice([0, 0, 0, 1, 2]), circuit=mode != 1 and rng.random() < 0.15, dielectric=diel,
                     all_species=int(gas == "O2" and rng.random() < 0.5), room=16 if nx * ny < 40000 else 8)


class OnDevice(dict):
    """Fields of running cases, copied from the device when they are looked up; a field of several cases is
    their concatenation.  The particles of a species, in cell order, are followed by zeros up to `room` (their
    number depends on the draws)."""

    def __init__(self, cases, grids, room):
        nsp = max(c.info.nsp for c in cases)
        names = list(grids) + ["%d.%s" % (s, a) for s in range(nsp) for a in ("count", "x", "y", "vx", "vy", "vz")]
        super().__init__(dict.fromkeys(names))
        self.cases, self.room, self.kept = cases, room, (None, None)

    def __getitem__(self, name):
        if "." not in name:
            return np.concatenate([c.grid(name) for c in self.cases])
        s, a = int(name.split(".")[0]), name.split(".")[1]
        if self.kept[0] != s:
            self.kept = (s, [c.particles(s) for c in self.cases])
        if a == "count":
            return np.concatenate([n for n, _ in self.kept[1]])
        k = ("x", "y", "vx", "vy", "vz").index(a)
        out, at = np.zeros(self.room, np.float32), 0
        for _, v in self.kept[1]:
            out[at:at + v[k].size] = v[k]
            at += v[k].size
        return out

    def items(self):
        return [(k, self[k]) for k in self]

    def values(self):
        return [self[k] for k in self]


GRIDS = ("EX", "EY", "PHI", "DEN", "AVE_DEN", "AVE_PHI", "COND_CHARGE", "MCC_COUNT", "EEDF", "FLUID_DEN",
         "SURFACE_CHARGE")


def deck_of(case):
    nx, ny, gas = case["nx"], case["ny"], case["gas"]
    extra = {}
    if gas != "Ar":
        extra = dict(te_ev=3.0, ion_density=ION_DENSITY[gas])
    window = 400 if case["field_mode"] == 2 else 40
    deck = ccp_deck(nx, ny, (nx - 1) * CELL, (ny - 1) * CELL, gas=gas, ppc=case["ppc"], voltage=case["volts"],
                    pressure_torr=case["mtorr"] * 1e-3, max_np_factor=case["room"], smoothing=case["smooth"],
                    average_iter=window, circuit=(50.0, 1e-7, 1e-9) if case["circuit"] else None, **extra)
    if case["dielectric"]:  # a slab over the driven electrode and a block inside, as hpic.decks.dielectric_deck
        deck["Geometry"]["DielectricSpec"] = [
            {"M_ID": 3, "X0": 0, "X1": nx - 1, "Y0": 0, "Y1": 3, "Epsilon": 4.0},
            {"M_ID": 4, "X0": nx // 3, "X1": nx // 2, "Y0": ny // 2, "Y1": ny // 2 + 3, "Epsilon": 3.9},
        ]
    return deck, window


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    seed = 1 + seed % (2 ** 31 - 3)  # the loader's Park-Miller seeds
    kind = case["kind"]
    run_as = dict(move_mode=1, gas_temp_mode=1, gpu_load=1)
    if kind == "step":
        deck, window = deck_of(case)
        c = hpic.Case(deck, seed=seed, field_mode=case["field_mode"], eedf_every=case["eedf"],
                      o2_all_species=case["all_species"], **run_as)
        c.step(window + 2, stream())
        return case, c
    if kind == "batch":
        cases = [hpic.Case(deck, seed=1 + (s + seed) % (2 ** 31 - 3), field_mode=2, **run_as)
                 for deck, s, _ in batched_cases(case["n"], case["mix"])]
        b = hpic.Batch(cases)
        b.step(20, stream())
        room = 2 * sum(c.info.Csize * d["ppc"] for c, (_, _, d) in zip(cases, batched_cases(case["n"], case["mix"])))
        return case, b, room
    if kind == "serve":
        return case, requests_of(case, seed)
    # deposit: a case of this size whose particles the program sets, a sheath-bounded cosine profile
    nx, ny = case["nx"], case["ny"]
    c = hpic.Case(ccp_deck(nx, ny, (nx - 1) * CELL, (ny - 1) * CELL, ppc=case["ppc"]), seed=seed, **run_as)
    for s, (counts, arrays) in enumerate(particles_of(case, seed)):
        c.set_particles(s, counts, *arrays)
    return case, c, torch.empty(c.info.nsp * c.info.Gsize, dtype=torch.float64, device="cuda")


def requests_of(case, seed):
    """The first n small requests of the served workload's stream, (deck, steps, seed) each."""
    got = []
    for _, deck, steps, s, _ in served_stream(20 * case["n"] + 40, seed=case["mix"], cycles=(1, 4)):
        if deck["Geometry"]["SystemSpec"]["NumGridx"] <= case["largest"] and len(got) < case["n"]:
            got.append((deck, max(10, int(steps * case["scale"])), 1 + (s + seed) % (2 ** 31 - 3)))
    return got


def particles_of(case, seed):
    """Per species: counts per cell and (x, y, vx, vy, vz), denser in the middle of the gap."""
    rng = np.random.default_rng(seed)
    ncx, ncy = case["nx"] - 1, case["ny"] - 1
    profile = 0.25 + np.sin(np.pi * (np.arange(ncy) + 0.5) / ncy)
    for s in range(2):
        counts = rng.poisson(case["ppc"] * np.broadcast_to(profile, (ncx, ncy))).astype(np.int32).ravel()
        n = int(counts.sum())
        xy = [rng.random(n, dtype=np.float32) for _ in range(2)]
        v = [rng.standard_normal(n, dtype=np.float32) * np.float32(6e5 if s == 0 else 250.0) for _ in range(3)]
        yield counts, xy + v


def run(state):
    case = state[0]
    kind = case["kind"]
    if kind == "step":
        state[1].step(case["steps"], stream())
        return OnDevice([state[1]], GRIDS, 3 * (case["nx"] - 1) * (case["ny"] - 1) * case["ppc"] // 2)
    if kind == "batch":
        state[1].step(case["steps"], stream())
        return OnDevice(state[1].cases, ("EX", "EY", "PHI", "DEN", "AVE_DEN", "AVE_PHI", "MCC_COUNT"), state[2])
    if kind == "serve":
        server = hpic.Server(max_slots=case["slots"], steps_per_launch=20, field_mode=2, move_mode=1, gas_temp_mode=1,
                             gpu_load=1)
        for deck, steps, seed in state[1]:
            server.submit(deck, steps, seed)
        results = sorted(server.run(stream()), key=lambda r: r[0].request_id)
        server.close()
        return dict(density=np.concatenate([d.ravel() for _, d, _ in results]),
                    potential=np.concatenate([p for _, _, p in results]),
                    pushes=[r.particle_pushes for r, _, _ in results], status=[r.status for r, _, _ in results])
    c, out = state[1], state[2]
    hpic._check(hpic.lib().hp_Deposit_noalloc(c.h, ctypes.c_void_p(out.data_ptr()), stream()))
    return out


def step_bytes(nx, ny, particles, species, channels):
    """A step reads and writes every particle's position and in-plane velocity (32 bytes) and, per node, the
    charge densities, the potential, the field and their running sums."""
    return 32.0 * particles + (nx * ny) * (24.0 * species + 64.0)


def work(case):
    kind = case["kind"]
    if kind == "step":
        nx, ny, gas = case["nx"], case["ny"], case["gas"]
        n = (nx - 1) * (ny - 1) * case["ppc"] * LOAD[gas]
        one, flops = step_bytes(nx, ny, n, SPECIES[gas], 0), 60.0 * n
        return {"bytes": case["steps"] * one, "flops": case["steps"] * flops}
    if kind in ("batch", "serve"):
        total, flops = 0.0, 0.0
        if kind == "batch":
            todo = [(deck, case["steps"]) for deck, _, _ in batched_cases(case["n"], case["mix"])]
        else:
            todo = [(deck, steps) for deck, steps, _ in requests_of(case, 0)]
        for deck, steps in todo:
            g, gas = deck["Geometry"]["SystemSpec"], deck["GasSpecies"]
            name = ("Ar", "O2", "ArO2")[gas["Type(0:Ar,1:O2,2:Ar/O2)"]]
            nx, ny, e = g["NumGridx"], g["NumGridy"], gas["ChargeSpecies"]["Electron"]
            n = e["Density"] * g["X_length(m)"] * g["Y_length(m)"] / e["np2c"] * LOAD[name]
            total += steps * step_bytes(nx, ny, n, SPECIES[name], 0)
            flops += steps * 60.0 * n
        return {"bytes": total, "flops": flops}
    n = (case["nx"] - 1) * (case["ny"] - 1) * case["ppc"] * 2 * (0.25 + 2 / np.pi)
    return {"bytes": 8.0 * n + 16.0 * case["nx"] * case["ny"], "flops": 10.0 * n}


def tolerance(case):
    # The steps, batches and served results are defined bit for bit: the order of every sum, the draws of every
    # particle and its place in its cell are part of the entry points, and a case's results are the same alone, in
    # a batch and through the server.  The densities of the deposit are sums of 32-bit weights of some 100
    # particles: 4.1e-9 from the 64-bit sums as measured (2-norm), four times that.
    return {"rel": 1.6e-8} if case["kind"] == "deposit" else "exact"


def exact(case, seed):
    if case["kind"] != "deposit":
        return None  # hundreds of Monte Carlo steps of up to 50 million particles
    ncx, ncy = case["nx"] - 1, case["ny"] - 1
    out = []
    for counts, (x, y, _, _, _) in particles_of(case, 1 + seed % (2 ** 31 - 3)):
        x, y = x.astype(np.float64), y.astype(np.float64)
        cell = np.repeat(np.arange(ncx * ncy), counts)
        den = np.zeros((ncx + 1, ncy + 1))
        for di, wx in ((0, 1 - x), (1, x)):
            for dj, wy in ((0, 1 - y), (1, y)):
                den[di:di + ncx, dj:dj + ncy] += np.bincount(cell, wx * wy, ncx * ncy).reshape(ncx, ncy)
        den[0, 1:-1] *= 2.0  # a node on a Neumann side wall stands for half a cell
        den[-1, 1:-1] *= 2.0
        out.append(den.ravel())
    return torch.from_numpy(np.concatenate(out))
