"""The framework's work as its users call it: cases for measuring speed and accuracy.

Every case is one pass of a disorder scan, the way the framework is used in earnest: a program builds
a device and its leads once (geometry, elimination plan, lead self-energies), and each pass brings the
Hamiltonian values of new disorder configurations from host memory and solves them through the public
entry points. The kinds:

``t``         transmissions of one two-terminal device at some energies x configurations
              (``NestedTwoTerminal.transmissions_with``), in FP64 (the entry points' default) or mixed
              precision; ``leads="device"`` forms the lead self-energies on the GPU in each pass
              (``self_energies_on_device``: an energy scan that never holds them on the host)
``systems``   several devices of uneven sizes in one batch (``solve_systems``)
``grad``      transmissions with dT/dV of every orbital and dT/dJ (``transmissions_with_grad``)
``states``    scattering states of both leads on every orbital (``scattering_states_batch``)
``cross``     every T_pq of a four-terminal cross (``NestedMultiTerminal.solve_batch``)

``CAROLI_SINGLE`` has no case: its unrefined transmissions carry errors of 1e-3 to 1, whatever the code.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from caroli_gb300 import Interface, NestedMultiTerminal, NestedTwoTerminal, Precision, Region, bhz, cubic, graphene, square
from caroli_gb300.disorder import Moments, disordered
from caroli_gb300.lattice import Site
from caroli_gb300.model import bhz_spin
from caroli_gb300.nested import solve_systems

MODELS = {"square": square, "bhz": bhz, "graphene": graphene, "cubic": cubic}
# The energies a model is scanned over: the square and cubic bands, graphene's first subbands and the
# BHZ gap with the band edges around it (the reference's benchmark and the headline workload).
BAND = {"square": (-1.9, 1.7), "cubic": (-1.3, 1.1), "graphene": (-0.5, 0.5), "bhz": (-0.16, 0.16)}


def _case(name, kind, model, shape, energies, **more):
    length, width, depth = shape
    case = {"kind": kind, "model": model, "length": length, "width": width, "depth": depth, "energies": energies,
            "configs": 1, "precision": "double", "disorder": "anderson", "strength": 1.0, "leads": "host"}
    case.update(more)
    return dict(case, name=name) if name else case


def listed():
    magnetic = {"disorder": "magnetic", "strength": 0.4}
    return [
        # The smallest call: one energy of the benchmark's smallest square problem.
        _case("square32_one", "t", "square", (32, 32, 1), 1, strength=2.0),
        # A small mixed-precision call, where its fixed costs show.
        _case("bhz40x16_mixed_one", "t", "bhz", (40, 16, 1), 1, precision="mixed", **magnetic),
        # The benchmark's graphene problem: an energy scan of one sample in FP64.
        _case("graphene64_scan", "t", "graphene", (64, 64, 1), 8),
        # The headline device in FP64: what a user gets without asking for a precision.
        _case("bhz200x64_double", "t", "bhz", (200, 64, 1), 4, configs=4, **magnetic),
        # The headline workload: a conductance map, energies x configurations, refined.
        _case("bhz200x64_mixed", "t", "bhz", (200, 64, 1), 16, configs=8, precision="mixed", **magnetic),
        # Zigzag ribbons of uneven (also odd) widths and lengths in one refined batch.
        _case("ribbons_mixed", "systems", "graphene", (150, 75, 1), 6, precision="mixed", configs=5),
        # Sensitivities: every site's potential and the exchange coupling (spin blocks coupled).
        _case("bhz100x40_grad", "grad", "bhz", (100, 40, 1), 16, disorder="isotropic", strength=0.3, precision="mixed"),
        # Wave functions for local currents and densities.
        _case("bhz120x32_states", "states", "bhz", (120, 32, 1), 4, precision="mixed", **magnetic),
        # The benchmark's four-terminal cross in FP64.
        _case("square_cross128", "cross", "square", (1, 128, 1), 8),
        # A four-terminal topological device: few channels, refined.
        _case("bhz_cross64_mixed", "cross", "bhz", (1, 64, 1), 8, precision="mixed", strength=0.5),
        # Three-dimensional wires near the Anderson transition; lead self-energies formed on the GPU.
        _case("cubic32x16x16", "t", "cubic", (32, 16, 16), 4, strength=16.5, leads="device"),
        _case("cubic48x24x24", "t", "cubic", (48, 24, 24), 2, strength=16.5, leads="device"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    which = rng.choice(["double", "double", "mixed", "mixed", "cubic", "cross", "cross_mixed", "grad", "states",
                        "systems"])
    if which == "double":
        model = rng.choice(["square", "graphene", "bhz"])
        more = {"disorder": "magnetic", "strength": 0.4} if model == "bhz" else {"strength": rng.choice([1.0, 2.0])}
        return _case(None, "t", model, (size(24, 200), size(16, 64), 1), size(1, 8), configs=rng.choice([1, 2]), **more)
    if which == "mixed":
        model = rng.choice(["square", "graphene", "bhz"])
        more = {"disorder": "magnetic", "strength": 0.4} if model == "bhz" else {}
        width = size(16, 64) if model != "square" else size(16, 40)
        return _case(None, "t", model, (size(24, 200), width, 1), size(1, 16), configs=size(1, 8), precision="mixed",
                     **more)
    if which == "cubic":
        return _case(None, "t", "cubic", (size(8, 32), size(8, 20), size(8, 20)), size(1, 4), strength=16.5,
                     leads=rng.choice(["host", "device"]))
    if which == "cross":
        return _case(None, "cross", rng.choice(["square", "graphene"]), (1, 4 * size(5, 24), 1), size(1, 8))
    if which == "cross_mixed":
        return _case(None, "cross", "bhz", (1, 4 * size(4, 14), 1), size(1, 8), precision="mixed", strength=0.5)
    if which == "grad":
        return _case(None, "grad", "bhz", (size(16, 100), size(8, 40), 1), size(1, 12), disorder="isotropic",
                     strength=0.3, precision="mixed")
    if which == "states":
        return _case(None, "states", "bhz", (size(20, 140), size(8, 40), 1), size(1, 4), precision="mixed",
                     disorder="magnetic", strength=0.4)
    return _case(None, "systems", "graphene", (size(40, 160), size(24, 72), 1), size(2, 6), precision="mixed",
                 configs=rng.choice([2, 3, 4, 5]))


# ---- devices: built once per program, shared by its passes ---------------------------------------------

def _energies(case):
    lo, hi = BAND[case["model"]]
    n = case["energies"]
    return [float(e) for e in (np.linspace(lo, hi, n) if n > 1 else [lo + 0.31 * (hi - lo)])]


def _shapes(case):
    """(length, width, depth) of every device: one, or uneven ones around the case's for ``systems``."""
    shape = (case["length"], case["width"], case["depth"])
    if case["kind"] != "systems":
        return [shape]
    return [(max(6, shape[0] - 17 * ((3 * k) % 5) + 40), max(6, shape[1] + 7 * ((2 * k) % 5) - 16), 1)
            for k in range(case["configs"])]


class _Device:
    """One device as a program keeps it, with what is needed to write the Hamiltonian values of a new
    disorder configuration on its pattern."""

    def __init__(self, case, shape):
        clean = MODELS[case["model"]]()
        if case["kind"] == "cross":
            region, interfaces = _cross(clean.lattice, shape[1])
        else:
            region = Region.cuboid(clean.lattice, list(shape))
        entries = [{"kind": "anderson", "strength": 1.0}]
        self.spin = None
        if case["disorder"] in ("magnetic", "isotropic"):
            moments = Moments.polarized(1.0) if case["disorder"] == "magnetic" else Moments.isotropic()
            self.spin = bhz_spin("opposite-g")
            entries.append({"kind": "magnetic", "concentration": 1.0, "exchange": 1.0, "moments": moments,
                            "spin": self.spin})
        full = disordered(clean, region, entries, 0)  # every on-site entry the disorder can fill
        if case["kind"] == "cross":
            self.solver = NestedMultiTerminal.from_models([clean, full], clean, region, interfaces)
        else:
            self.solver = NestedTwoTerminal.from_models([clean, full], clean, region, 0)
        s = self.system = self.solver.system
        self.clean = s.values[0]
        rows = np.repeat(np.arange(s.n), np.diff(s.row_ptr))
        site = np.repeat(np.arange(len(s.site_offsets)), s.site_orbitals)
        cols = s.cols.astype(np.int64)
        self.on = np.nonzero(site[rows] == site[cols])[0]  # stored entries inside an on-site block
        self.site = site[rows[self.on]]
        self.a = rows[self.on] - s.site_offsets[self.site]
        self.b = cols[self.on] - s.site_offsets[self.site]
        self.sites = len(s.site_offsets)
        self.sigmas = None
        if case["leads"] == "host":
            self.sigmas = [self.solver.self_energies(e) for e in _energies(case)]

    def values(self, case, rng):
        """H values of one configuration, and dH/dJ of the exchange term."""
        out = self.clean.copy()
        n, derivative = self.sites, np.zeros(len(self.clean), np.complex128)
        if case["disorder"] == "anderson" or case["disorder"] == "isotropic":
            w = case["strength"] if case["disorder"] == "anderson" else 0.02
            out[self.on] += np.where(self.a == self.b, (w * (rng.uniform(size=n) - 0.5))[self.site], 0.0)
        if self.spin is not None:
            concentration = 0.2 if case["disorder"] == "magnetic" else 0.1
            z = np.ones(n) if case["disorder"] == "magnetic" else rng.uniform(-1.0, 1.0, n)
            phi = rng.uniform(0.0, 2.0 * np.pi, n)
            occupied = np.zeros(n)
            occupied[rng.permutation(n)[:int(concentration * n)]] = 1.0
            perp = np.sqrt(1.0 - z * z)
            for m, s in zip((perp * np.cos(phi), perp * np.sin(phi), z), self.spin):
                derivative[self.on] += (occupied * m)[self.site] * s[self.a, self.b]
            out += case["strength"] * derivative
        return out, derivative


def _cross(lattice, w):
    """A w x w square with arms of length w / 4 and a lead on each (left, right, bottom, top): the
    benchmark's cross."""
    arm, subs = w // 4, range(len(lattice.sublattices))
    sites = lambda cells: [Site((x, y, 0), s) for x, y in cells for s in subs]  # noqa: E731
    span = range(-arm, w + arm)
    region = Region.from_sites(lattice, sites((x, y) for x in span for y in span if 0 <= x < w or 0 <= y < w))
    column = lambda x: Region.from_sites(lattice, sites((x, y) for y in range(w)))  # noqa: E731
    row = lambda y: Region.from_sites(lattice, sites((x, y) for x in range(w)))  # noqa: E731
    return region, [Interface(column(-arm), (-1, 0, 0)), Interface(column(w + arm - 1), (1, 0, 0)),
                    Interface(row(-arm), (0, -1, 0)), Interface(row(w + arm - 1), (0, 1, 0))]


@functools.lru_cache(maxsize=32)
def _devices(key):
    case = dict(key)
    return [_Device(case, shape) for shape in _shapes(case)]


def _of(case):
    return _devices(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


def _inputs(case, seed):
    """Per device: the values (configurations x entries) and dH/dJ of every configuration."""
    rng = np.random.RandomState(seed % (1 << 32))
    configs = 1 if case["kind"] == "systems" else case["configs"]
    out = []
    for d in _of(case):
        pairs = [d.values(case, rng) for _ in range(configs)]
        out.append((np.stack([p[0] for p in pairs]), np.stack([p[1][None] for p in pairs])))
    return out


def prepare(case, seed):
    devices = _of(case)
    for d in devices:
        d.solver.plan()
    inputs = []
    for values, derivs in _inputs(case, seed):
        pinned = torch.empty(values.shape, dtype=torch.complex128, pin_memory=torch.cuda.is_available())
        pinned.copy_(torch.from_numpy(values))
        inputs.append((pinned.numpy(), derivs, pinned))  # the tensor owns the pinned memory
    return {"case": case, "devices": devices, "inputs": inputs}


def run(state):
    case, devices = state["case"], state["devices"]
    precision = Precision.MIXED if case["precision"] == "mixed" else Precision.DOUBLE
    for d, (values, _, _) in zip(devices, state["inputs"]):
        d.solver.plan().upload_values(values)
    solver, sigmas = devices[0].solver, devices[0].sigmas
    configs = range(case["configs"])
    if case["kind"] == "systems":
        t, _, _ = solve_systems([(d.solver, s, 0) for d in devices for s in d.sigmas], precision)
        return t
    if case["leads"] == "device":
        sigmas = [solver.self_energies_on_device(e) for e in _energies(case)]
    if case["kind"] == "cross":
        return solver.solve_batch(sigmas, [0] * len(sigmas), precision)[0]
    pairs = [(s, c) for s in sigmas for c in configs]
    if case["kind"] == "grad":
        solver.set_parameter_derivatives(state["inputs"][0][1])
        t, _, dv, dp = solver.transmissions_with_grad([s for s, _ in pairs], [c for _, c in pairs])
        return {"t": t, "dv": dv, "dp": dp}
    if case["kind"] == "states":
        return [list(s.leads) for s in solver.scattering_states_batch([s for s, _ in pairs], [c for _, c in pairs])]
    return np.array(solver.transmissions_with([s for s, _ in pairs], [c for _, c in pairs], precision))


# ---- what a pass cannot do without ---------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _elimination(dims, faces, orbitals):
    """Complex LU flops of the nested dissection of a box of ``dims`` sites: the separator's variables
    eliminated against the box's boundary, ``faces[a]`` of whose two sides along axis a are open."""
    boundary = orbitals * sum(f * math.prod(dims) // dims[a] for a, f in enumerate(faces))
    if math.prod(dims) * orbitals <= 16:
        ne, below = math.prod(dims) * orbitals, 0.0
    else:
        a = max(range(3), key=lambda k: dims[k])
        half = (dims[a] // 2, dims[a] - 1 - dims[a] // 2)
        ne = orbitals * math.prod(dims) // dims[a]
        # The separator opens one side of each half; the box's own open sides go to the halves in turn.
        sides = ((faces[a] + 1) // 2 + 1, faces[a] // 2 + 1)
        below = sum(_elimination(dims[:a] + (h,) + dims[a + 1:], faces[:a] + (min(2, s),) + faces[a + 1:], orbitals)
                    for h, s in zip(half, sides) if h > 0)
    return below + 8.0 / 3.0 * ((ne + boundary) ** 3 - boundary ** 3)


def work(case):
    blocks = 2 if case["model"] == "bhz" and case["disorder"] != "isotropic" else 1
    per_cell = {"square": 1, "cubic": 1, "graphene": 2, "bhz": 4}[case["model"]]
    k = per_cell // blocks
    flops = moved = 0.0
    solves = case["energies"] * (1 if case["kind"] == "systems" else case["configs"])
    for length, width, depth in _shapes(case):
        slice_ = k * width * depth  # orbitals of a lead slice, per block
        if case["kind"] == "cross":
            arm, cells = width // 4, width * width + 4 * width * (width // 4)
            one = _elimination((width, width, 1), (2, 2, 0), k) + 4.0 * _elimination((arm, width, 1), (2, 0, 0), k)
            root, leads = 4 * slice_, 4
            one += 8.0 * root ** 3  # every pair of leads wants the whole inverse
        else:
            cells = length * width * depth
            one = _elimination((length - 2, width, depth), (2, 0, 0), k)
            root, leads = 2 * slice_, 2
            one += 8.0 / 3.0 * root ** 3 + 8.0 * slice_ ** 3
        one += 16.0 * slice_ ** 3 if case["precision"] == "double" else 0.0  # the trace with both broadenings
        flops += blocks * one * solves
        n = cells * per_cell
        nnz = n * (1 + 2 * {"square": 2, "cubic": 3, "graphene": 1.5, "bhz": 4}[case["model"]])
        moved += 16.0 * nnz * (1 if case["kind"] == "systems" else case["configs"])
        moved += 16.0 * blocks * leads * slice_ ** 2 * case["energies"]
        if case["kind"] == "grad":
            moved += 16.0 * nnz * case["configs"] + 8.0 * n * solves
        if case["kind"] == "states":
            moved += 16.0 * n * 2 * 2 * solves
        moved += 8.0 * solves * (16 if case["kind"] == "cross" else 1)
    return {"bytes": moved, "flops": flops}


# ---- the same in 64 bits, by elimination slice after slice ----------------------------------------------

class _Slices:
    """A = z - H - Σ of one block over a batch of (z, values), as dense slices along the first axis
    (the Hamiltonians couple neighbouring slices only)."""

    def __init__(self, system, block, device):
        s = self.system = system
        self.device = device
        site = np.repeat(np.arange(len(s.site_offsets)), s.site_orbitals)
        x = np.asarray(s.cells)[site, 0]
        self.rows = np.nonzero(np.asarray(s.labels) == block)[0]
        order = np.argsort(x[self.rows], kind="stable")
        self.rows = self.rows[order]
        xs = x[self.rows]
        self.starts = np.concatenate([np.nonzero(np.diff(xs, prepend=xs[0] - 1))[0], [len(xs)]])
        self.at = np.full(s.n, -1)
        self.at[self.rows] = np.arange(len(self.rows))
        slice_of = np.searchsorted(self.starts, np.arange(len(self.rows)), side="right") - 1
        r = np.repeat(np.arange(s.n), np.diff(s.row_ptr))
        c = s.cols.astype(np.int64)
        q = np.nonzero((self.at[r] >= 0) & (self.at[c] >= 0))[0]
        i, j = self.at[r[q]], self.at[c[q]]
        si, sj = slice_of[i], slice_of[j]
        assert np.all(np.abs(si - sj) <= 1)
        self.parts = {}
        for step in (-1, 0, 1):
            for k in range(len(self.starts) - 1):
                self.parts[k, step] = []
            sel = np.nonzero(sj - si == step)[0]
            by = sel[np.argsort(si[sel], kind="stable")]
            cuts = np.searchsorted(si[by], np.arange(len(self.starts)))
            for k in range(len(self.starts) - 1):
                e = by[cuts[k]:cuts[k + 1]]
                self.parts[k, step] = (q[e], i[e] - self.starts[k], j[e] - self.starts[k + step] if len(e) else j[e])

    def size(self, k):
        return int(self.starts[k + 1] - self.starts[k])

    def dense(self, values, k, step):
        """-H between slices k and k + step for every configuration (values: configurations x entries)."""
        q, i, j = (torch.as_tensor(p, device=self.device, dtype=torch.long) for p in self.parts[k, step])
        out = torch.zeros(values.shape[0], self.size(k), self.size(k + step), dtype=torch.complex128, device=self.device)
        out[:, i, j] = -values[:, q]
        return out

    def solve(self, z, values, sigma, rhs):
        """X = A^-1 B for a batch: z[i], values[i]; ``sigma``: [(orbitals, [matrix per i])], ``rhs``: batch x
        rows x columns in this block's row order. Orbitals of one slice or of neighbouring ones."""
        n = len(self.starts) - 1
        eye = lambda m: torch.eye(m, dtype=torch.complex128, device=self.device)  # noqa: E731
        zt = torch.as_tensor(z, dtype=torch.complex128, device=self.device).reshape(-1, 1, 1)
        diag = [self.dense(values, k, 0) + zt * eye(self.size(k)) for k in range(n)]
        upper = [self.dense(values, k, 1) for k in range(n - 1)]
        lower = [self.dense(values, k, -1) for k in range(1, n)]
        for orbitals, mats in sigma:
            rows = self.at[np.asarray(orbitals)]
            si = np.searchsorted(self.starts, rows, side="right") - 1
            m = torch.stack([torch.as_tensor(np.ascontiguousarray(x), device=self.device) for x in mats])
            for k in np.unique(si):
                for l in np.unique(si):
                    a, b = np.nonzero(si == k)[0], np.nonzero(si == l)[0]
                    ia = torch.as_tensor(rows[a] - self.starts[k], device=self.device).reshape(-1, 1)
                    ib = torch.as_tensor(rows[b] - self.starts[l], device=self.device).reshape(1, -1)
                    part = m[:, torch.as_tensor(a, device=self.device)][:, :, torch.as_tensor(b, device=self.device)]
                    if abs(k - l) > 1:
                        assert not part.abs().max() > 0
                        continue
                    (diag[k] if k == l else upper[k] if l > k else lower[l])[:, ia, ib] -= part
        gain, y = [], []
        for k in range(n):
            b = rhs[:, self.starts[k]:self.starts[k + 1]]
            d = diag[k]
            if k:
                d = d - lower[k - 1] @ gain[-1]
                b = b - lower[k - 1] @ y[-1]
            both = torch.linalg.solve(d, torch.cat([upper[k], b], dim=2) if k + 1 < n else b)
            width = self.size(k + 1) if k + 1 < n else 0
            gain.append(both[:, :, :width])
            y.append(both[:, :, width:])
            diag[k] = None
        for k in range(n - 2, -1, -1):
            y[k] = y[k] - gain[k] @ y[k + 1]
        return torch.cat(y, dim=1)


def _adjoint(m):
    return m.conj().transpose(-1, -2)


def _broadening(m):
    return 1j * (m - _adjoint(m))


def _definite_sigmas(h00, h01, energy):
    """(Σ_L, Σ_R) of a lead whose coupling is a multiple c of the identity, from the cell's modes."""
    c = h01[0, 0].real
    theta, y = np.linalg.eigh(h00)
    mu = (energy - theta) / c
    inner = np.abs(mu) < 2.0
    root = np.where(inner, mu / 2 - 1j * np.sign(c) * np.sqrt(np.maximum(4 - mu * mu, 0.0)) / 2, 0.0)
    outer = np.where(inner, 1.0, (mu + np.sign(mu) * np.sqrt(np.maximum(mu * mu - 4, 0.0))) / 2)
    lam = np.where(inner, root, 1.0 / outer)
    sigma = c * (y * lam) @ y.conj().T
    return sigma, sigma


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    energies, devices, inputs = _energies(case), _of(case), _inputs(case, seed)
    put = lambda v: torch.as_tensor(v, dtype=torch.complex128, device=device)  # noqa: E731
    outs = []
    for d, (values, derivs) in zip(devices, inputs):
        s = d.system
        configs = 1 if case["kind"] == "systems" else case["configs"]
        pairs = [(e, c) for e in range(len(energies)) for c in range(configs)]
        total, psi = 0.0, None
        dv, dp = torch.zeros(len(pairs), s.n, dtype=torch.float64, device=device), 0.0
        for b, block in enumerate(s.blocks):
            sl = _Slices(s, b, device)
            z = [energies[e] for e, _ in pairs]
            vals = put(values)[[c for _, c in pairs]]
            if case["kind"] == "cross":
                leads = [(l.orbitals, [d.sigmas[e].blocks[b][p] for e, _ in pairs])
                         for p, l in enumerate(d.solver.block_leads[b]) if l is not None]
                kept = np.unique(np.concatenate([o for o, _ in leads]))
                rhs = torch.zeros(len(sl.rows), len(kept), dtype=torch.complex128, device=device)
                rhs[sl.at[kept], np.arange(len(kept))] = 1.0
                # The leads of the vertical arms couple every slice, so the sweep runs with -i on the kept
                # orbitals instead of Σ, and G = (1 - G' (Σ + i))^-1 G' on them follows.
                local = [(kept[k:k + 1], [np.full((1, 1), -1j)] * len(pairs)) for k in range(len(kept))]
                g = sl.solve(z, vals, local, rhs.expand(len(pairs), -1, -1))[:, sl.at[kept]]
                change = torch.diag(torch.full((len(kept),), 1j, dtype=torch.complex128, device=device)).repeat(len(pairs), 1, 1)
                for o, ms in leads:
                    at = np.searchsorted(kept, o)
                    change[:, at[:, None], at[None, :]] += torch.stack([put(m) for m in ms])
                g = torch.linalg.solve(torch.eye(len(kept), dtype=torch.complex128, device=device) - g @ change, g)
                at = [torch.as_tensor(np.searchsorted(kept, o), device=device) for o, _ in leads]
                gamma = [_broadening(torch.stack([put(m) for m in ms])) for _, ms in leads]
                t = torch.zeros(len(pairs), len(leads), len(leads), dtype=torch.float64, device=device)
                for p in range(len(leads)):
                    for q in range(len(leads)):
                        gpq = g[:, at[p]][:, :, at[q]]
                        t[:, p, q] = torch.einsum("bij,bij->b", gamma[p] @ gpq @ gamma[q], gpq.conj()).real
                total = total + t
                continue
            if case["leads"] == "device":
                pairs_sigma = [_definite_sigmas(block.left_h00, block.left_h01, e) for e in energies]
            else:
                pairs_sigma = [d.sigmas[e].blocks[b] for e in range(len(energies))]
            sig = [(block.left, [pairs_sigma[e][0] for e, _ in pairs]), (block.right, [pairs_sigma[e][1] for e, _ in pairs])]
            left, right = sl.at[np.asarray(block.left)], sl.at[np.asarray(block.right)]
            if case["kind"] == "states":
                psi = psi or [[np.zeros((s.n, 0), complex)] * 2 for _ in pairs]
                for i, (e, c) in enumerate(pairs):
                    w = d.sigmas[e].w_left()[b], d.sigmas[e].w_right()[b]
                    rhs = torch.zeros(1, len(sl.rows), w[0].shape[1] + w[1].shape[1], dtype=torch.complex128, device=device)
                    rhs[0, left, :w[0].shape[1]] = put(w[0])
                    rhs[0, right, w[0].shape[1]:] += put(w[1])
                    x = sl.solve(z[i:i + 1], vals[i:i + 1], [(o, m[i:i + 1]) for o, m in sig], rhs)[0].cpu().numpy()
                    full = np.zeros((s.n, x.shape[1]), complex)
                    full[sl.rows] = x
                    cut = w[0].shape[1]
                    psi[i] = [np.concatenate([psi[i][0], full[:, :cut]], 1), np.concatenate([psi[i][1], full[:, cut:]], 1)]
                continue
            gl, gr = (_broadening(torch.stack([put(m) for m in ms])) for _, ms in sig)
            if case["kind"] == "grad":
                rhs = torch.zeros(len(pairs), len(sl.rows), len(right), dtype=torch.complex128, device=device)
                rhs[:, right] = gr  # G Γ_R
                ggr = sl.solve(z, vals, sig, rhs)
                rhs.zero_()
                rhs[:, right, torch.arange(len(right), device=device)] = 1.0
                gg = sl.solve(z, vals, sig, rhs)  # G's right-slice columns
                back = torch.zeros(len(pairs), len(sl.rows), len(right), dtype=torch.complex128, device=device)
                back[:, left] = gl @ gg[:, left]
                # A^† y = Γ_L G: the same elimination with Σ^† (H is Hermitian, the energy real).
                y = sl.solve(z, vals, [(o, [m.conj().T for m in ms]) for o, ms in sig], back)
                total = total + torch.einsum("bij,bij->b", gl @ ggr[:, left], gg[:, left].conj()).real
                rows = torch.as_tensor(sl.rows, device=device)
                dv[:, rows] += 2.0 * (ggr * y.conj()).sum(2).real
                r = torch.as_tensor(np.repeat(np.arange(s.n), np.diff(s.row_ptr)), device=device)
                c = torch.as_tensor(s.cols.astype(np.int64), device=device)
                at = torch.as_tensor(sl.at, device=device)
                dh = put(derivs)[:, 0]
                q = torch.nonzero((dh != 0).any(0) & (at[r] >= 0))[:, 0]
                prod = torch.stack([(y[i][at[r[q]]].conj() * ggr[i][at[c[q]]]).sum(1) for i in range(len(pairs))])
                dp = dp + 2.0 * (dh[[c_ for _, c_ in pairs]][:, q] * prod).sum(1).real[:, None]
                continue
            rhs = torch.zeros(len(sl.rows), len(right), dtype=torch.complex128, device=device)
            rhs[right, np.arange(len(right))] = 1.0
            step = max(1, int(4e9 / (16.0 * len(sl.rows) * (2 * len(right) + sl.size(0)))))
            got = []
            for i in range(0, len(pairs), step):
                part = slice(i, i + step)
                g = sl.solve(z[part], vals[part], [(o, m[part]) for o, m in sig],
                             rhs.expand(len(pairs[part]), -1, -1))[:, left]
                got.append(torch.einsum("bij,bij->b", gl[part] @ g @ gr[part], g.conj()).real)
            total = total + torch.cat(got)
        if case["kind"] == "states":
            return psi
        if case["kind"] == "grad":
            return {"t": total.cpu().numpy(), "dv": dv.cpu().numpy(), "dp": dp.cpu().numpy()}
        outs.append(total)
    return torch.cat(outs).cpu().numpy()
