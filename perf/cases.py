"""The work a user of fdtd3d_b200 has it do, as cases that can be timed and compared.

A case is one pass of a running simulation: a block of time steps and the
read-out that ends it (all field components, a DFT plane, an energy, a
gradient).  ``prepare`` makes what the program holds before the call: the
simulation with its materials, started from noise fields (a resumed run) or
advanced until the wave has entered the grid, and the buffers the fields are
read into.  ``exact`` is the same run restated in FP64 torch, from the update
equations alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fdtd3d_b200 as fd

PRECISION = {"fp64": fd.PREC_FP64_PLAIN, "fp32": fd.PREC_FP32, "fp16": fd.PREC_FP16S}
WORD = {"fp64": 8, "fp32": 4, "fp16": 2}
DX, WAVELENGTH, COURANT = 0.0005, 0.02, 0.5
C0 = 299792458.0
MU0 = 4 * math.pi * 1e-7
EPS0 = 1 / (MU0 * C0 * C0)
DEVICE = "cuda:0"
RESUMED = 500   # the time step a resumed run goes on from (time step 0 only starts a run: it updates no field)


def listed():
    return [
        # the reference's smallest runs: a 2-D TMz plane wave in FP64 (the bit-faithful form), dumped to the host
        {"name": "tmz_fp64_small", "kind": "tmz", "precision": "fp64", "nx": 120, "ny": 100, "pml": 10, "source": "tfsf",
         "tfsf": 16, "warm": 20, "steps": 100},
        # a 2-D photonics design run: dielectric blocks, a pulsed point source
        {"name": "tmz_fp32_512", "kind": "tmz", "precision": "fp32", "nx": 512, "ny": 512, "pml": 16, "source": "point",
         "warm": 60, "steps": 200},
        # the reference's 80^3 plane-wave run, FP64: a dielectric body, 40 cells per wavelength
        {"name": "grid_fp64_80", "kind": "grid", "precision": "fp64", "nx": 80, "ny": 80, "nz": 80, "pml": 10,
         "source": "tfsf", "tfsf": 15, "resume": False, "warm": 40, "steps": 50},
        # a mid-size FP64 run on sides that fit no tile, resumed from a saved state
        {"name": "grid_fp64_odd", "kind": "grid", "precision": "fp64", "nx": 203, "ny": 181, "nz": 165, "pml": 12,
         "source": "tfsf", "tfsf": 20, "resume": True, "warm": 0, "steps": 20},
        # the 80^3 plane wave in FP32: small enough that launches count
        {"name": "grid_fp32_80", "kind": "grid", "precision": "fp32", "nx": 80, "ny": 80, "nz": 80, "pml": 10,
         "source": "tfsf", "tfsf": 15, "resume": False, "warm": 40, "steps": 100},
        # sides that fit no tile and no 16-byte row, FP32, resumed
        {"name": "grid_fp32_odd", "kind": "grid", "precision": "fp32", "nx": 203, "ny": 181, "nz": 165, "pml": 12,
         "source": "tfsf", "tfsf": 20, "resume": True, "warm": 0, "steps": 40},
        # an antenna in a box: point source, no TF/SF, the field energy watched for the stop criterion
        {"name": "grid_fp32_point", "kind": "grid", "precision": "fp32", "nx": 256, "ny": 224, "nz": 240, "pml": 16,
         "source": "point", "resume": True, "warm": 0, "steps": 40},
        # the benchmark: 512^3 scattering of an oblique plane wave, FP32
        {"name": "grid_fp32_512", "kind": "grid", "precision": "fp32", "nx": 512, "ny": 512, "nz": 512, "pml": 16,
         "source": "tfsf", "tfsf": 32, "resume": False, "warm": 120, "steps": 40},
        # FP16 storage, taken for its memory: the same physics
        {"name": "grid_fp16_320", "kind": "grid", "precision": "fp16", "nx": 320, "ny": 320, "nz": 320, "pml": 16,
         "source": "tfsf", "tfsf": 32, "resume": True, "warm": 0, "steps": 20},
        # a Drude slab at normal incidence with a running DFT behind it
        {"name": "drude_fp32_384", "kind": "drude", "precision": "fp32", "nx": 384, "ny": 384, "nz": 384, "pml": 16,
         "source": "tfsf", "tfsf": 24, "resume": True, "warm": 0, "steps": 20},
        # a parameter sweep: 2-D grids of uneven sizes advanced together
        {"name": "batch_20", "kind": "batch", "count": 20, "low": 64, "high": 1024, "pml": 10, "steps": 1000},
        # inverse design: objective and its gradient with respect to every cell's eps
        {"name": "adjoint_512", "kind": "adjoint", "nx": 512, "ny": 512, "pml": 16, "steps": 800, "every": 100},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tmz", "grid", "grid", "grid", "grid", "drude", "batch", "adjoint"])
    pml = rng.randint(6, 16)
    box = pml + rng.randint(5, 16)
    if kind == "tmz":
        return {"kind": kind, "precision": rng.choice(["fp64", "fp32"]), "nx": spread(96, 1024), "ny": spread(96, 1024),
                "pml": pml, "source": rng.choice(["tfsf", "point"]), "tfsf": box, "warm": 20, "steps": spread(50, 300)}
    if kind == "grid":
        source = rng.choice(["tfsf", "tfsf", "point"])
        resume = source == "point" or rng.random() < 0.6   # (a pulse is still near zero after a few steps)
        return {"kind": kind, "precision": rng.choice(["fp64", "fp32", "fp32", "fp16"]), "nx": spread(72, 400),
                "ny": spread(72, 400), "nz": spread(72, 400), "pml": pml,
                "source": source, "tfsf": box, "resume": resume,
                "warm": 0 if resume else 60, "steps": rng.randint(11, 60)}
    if kind == "drude":
        return {"kind": kind, "precision": "fp32", "nx": spread(96, 320), "ny": spread(96, 320), "nz": spread(128, 320),
                "pml": pml, "source": "tfsf", "tfsf": box, "resume": True, "warm": 0, "steps": rng.randint(8, 40)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 20), "low": 64, "high": spread(128, 1024), "pml": 10,
                "steps": spread(200, 1000)}
    # (long enough for the pulse to reach the probe)
    return {"kind": kind, "nx": spread(160, 400), "ny": spread(160, 512), "pml": pml,
            "steps": rng.randint(700, 1000), "every": rng.randint(40, 150)}


# ------------------------------------------------------------------ inputs


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _blocks(shape, edge, top, gen):
    """FP64 map of 8-cell blocks, uniform in [1, top] (values FP32 holds exactly), 1 within `edge` cells of a face."""
    v = torch.rand([-(-n // 8) for n in shape], generator=gen, device=DEVICE, dtype=torch.float32) * (top - 1) + 1
    for a in range(len(shape)):
        v = v.repeat_interleave(8, dim=a)
    v = v[tuple(slice(0, n) for n in shape)].double()
    out = torch.ones(shape, dtype=torch.float64, device=DEVICE)
    inner = tuple(slice(edge, n - edge) for n in shape)
    out[inner] = v[inner]
    return out.contiguous()


def _sides(case):
    return (case["nx"], case["ny"], case["nz"]) if "nz" in case else (case["nx"], case["ny"])


def _physics(case):
    """Keyword arguments of fd.Simulation (and of the restatement below)."""
    n = _sides(case)
    kw = dict(size=n, use_pml=True, pml=case["pml"], dx=DX, wavelength=WAVELENGTH, courant=COURANT)
    if len(n) == 2:
        kw.update(mode=fd.MODE_TMZ, teta=90.0, phi=30.0, psi=90.0)
    elif case["kind"] == "drude":
        kw.update(mode=fd.MODE_DIM3, teta=0.0, phi=0.0, psi=25.0, use_metamaterials=True)
    else:
        kw.update(mode=fd.MODE_DIM3, teta=30.0, phi=45.0, psi=25.0)
    if case["kind"] == "adjoint":
        kw.update(point_source=_adjoint_places(n)[2])
    if case.get("source") == "tfsf":
        kw.update(use_tfsf=True, tfsf_left=case["tfsf"], tfsf_right=case["tfsf"])
    else:
        kw.setdefault("point_source", tuple(v // 2 for v in n))
        kw.update(point_source_mask=1 << 2, point_source_kind=1, point_source_bandwidth=0.5)
    return kw


def _noise(case, seed):
    """The fields a resumed run starts from: noise, 0 on the grid's faces (H in the units of E / eta0)."""
    gen = _generator(seed + 7919)
    eta0 = math.sqrt(MU0 / EPS0)
    for name in fd.COMPONENTS:
        v = torch.zeros(_sides(case), dtype=torch.float32, device=DEVICE)
        v[1:-1, 1:-1, 1:-1] = torch.randn([n - 2 for n in v.shape], generator=gen, device=DEVICE, dtype=torch.float32)
        yield name, (v if name[0] == "E" else v / eta0).double()


def _materials(case, seed):
    n = _sides(case)
    gen = _generator(seed)
    if case["kind"] == "drude":
        # a slab 1/6 of the grid thick normal to z, two cells inside the TF/SF box at its sides; the plasma frequency
        # varies from run to run
        om = torch.zeros(n, dtype=torch.float64, device=DEVICE)
        ga = torch.zeros(n, dtype=torch.float64, device=DEVICE)
        m = case["tfsf"] + 2
        z0 = n[2] // 2 - n[2] // 12
        box = (slice(m, n[0] - m), slice(m, n[1] - m), slice(z0, z0 + n[2] // 6))
        f = 25 + 10 * float(torch.rand(1, generator=gen, device=DEVICE))
        om[box] = float(np.float32(2 * np.pi * f * 1e9))
        ga[box] = float(np.float32(2 * np.pi * 1e9))
        eps = _blocks(n, m, 2.0, gen)
        eps[box] = 1.0
        return {"eps": eps, "omegape": om, "omegapm": om, "gammae": ga, "gammam": ga}
    if case["kind"] == "adjoint":
        lo, hi, _, _, _ = _adjoint_places(n)
        eps = torch.ones(n, dtype=torch.float64, device=DEVICE)
        shape = (hi[0] - lo[0], hi[1] - lo[1])
        eps[lo[0]:hi[0], lo[1]:hi[1]] = (torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float32) * 11 + 1).double()
        return {"eps": eps}
    return {"eps": _blocks(n, case["tfsf"] + 2 if case["source"] == "tfsf" else case["pml"] + 2, 4.0 if len(n) == 3 else 12.0, gen)}


def _adjoint_places(n):
    """Design box, source, probe box of the inverse-design case: a quarter of the sides, the probe right of it."""
    c = (n[0] // 2, n[1] // 2)
    h = (n[0] // 8, n[1] // 8)
    lo, hi = (c[0] - h[0], c[1] - h[1]), (c[0] + h[0], c[1] + h[1])
    probe = (hi[0] + h[0], c[1] - 8)
    return lo, hi, (lo[0] - h[0], c[1]), probe, (probe[0] + 16, probe[1] + 16)


def _batch_sizes(case):
    # the sizes belong to the case (its work does not change from seed to seed), the maps to the seed
    rng = np.random.default_rng([case["count"], case["high"], case["steps"]])
    return [(int(a), int(b)) for a, b in rng.integers(case["low"], case["high"] + 1, (case["count"], 2))]


def _batch_inputs(case, seed):
    sizes = _batch_sizes(case)
    gen = _generator(seed)
    return sizes, [_blocks(s, 0, 12.0, gen) for s in sizes]


BATCH_PHYSICS = dict(dx=DX, wavelength=WAVELENGTH, courant=COURANT, use_pml=True, point_source_mask=1 << 2,
                     point_source_kind=1, point_source_bandwidth=0.5, teta=90.0, phi=0.0, psi=90.0)


# -------------------------------------------------------------------- runs


def prepare(case, seed):
    if case["kind"] == "batch":
        sizes, maps = _batch_inputs(case, seed)
        batch = fd.Batch(sizes, pml=case["pml"], **BATCH_PHYSICS)
        for i, m in enumerate(maps):
            batch.set_eps(i, m.cpu().numpy())
        batch.tune(8)
        return {"case": case, "batch": batch}
    precision = PRECISION[case.get("precision", "fp32")]
    sim = fd.Simulation(device=0, precision=precision, **_physics(case))
    for name, values in _materials(case, seed).items():
        torch.cuda.synchronize()
        sim.set_material_device(name, values.data_ptr())
        sim.sync()
    state = {"case": case, "sim": sim}
    if case["kind"] == "adjoint":
        state["places"] = _adjoint_places(_sides(case))
        return state
    if case.get("resume"):
        for name, values in _noise(case, seed):
            sim.set_field(name, values.cpu().numpy())
        sim.t = RESUMED
    if case["warm"]:
        sim.step(case["warm"])
    if case["kind"] == "drude":
        sim.dft_setup("Ex", 2, _dft_plane(case), [15e9])
    names = fd.MODE_COMPONENTS[sim.mode]
    if case["kind"] == "tmz":
        state["out"] = {c: np.empty(sim.cells) for c in names}
    else:
        state["out"] = {c: torch.empty(sim.shape, dtype=torch.float64, device=DEVICE) for c in names}
    sim.sync()
    return state


def _dft_plane(case):
    n = case["nz"]
    return n // 2 - n // 12 + n // 6


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        batch = state["batch"]
        batch.step(case["steps"])
        fields = [[batch.field(i, c).reshape(-1) for c in ("Ez", "Hx", "Hy")] for i in range(case["count"])]
        return {c: np.concatenate([f[j] for f in fields]) for j, c in enumerate(("Ez", "Hx", "Hy"))}
    sim = state["sim"]
    if case["kind"] == "adjoint":
        _, _, _, lo, hi = state["places"]
        value, gradient = sim.backward(case["steps"], case["every"], lo, hi, fd.PREC_FP32)
        return {"objective": value, "gradient": gradient}
    sim.step(case["steps"])
    if case["kind"] == "tmz":
        return {c: sim.field(c, out=v) for c, v in state["out"].items()}
    for c, v in state["out"].items():
        sim.field_device(c, v.data_ptr())
    out = dict(state["out"])
    if case["kind"] == "drude":
        spectrum = sim.dft()
        out["dft_re"], out["dft_im"] = spectrum.real, spectrum.imag
    elif case["source"] == "point":
        out["energy"] = float(sim.reduce(fd.REDUCE_ENERGY)[0])
    return out


def work(case):
    """One pass with the state in memory: fields, PML auxiliaries and materials read once and written once, the outputs
    written once; the floating-point operations of every cell and step (the least of the update: six components of
    three differences, a product and a sum; the PML's second update; the Drude recurrence)."""
    if case["kind"] == "batch":
        sizes = _batch_sizes(case)
        cells = sum(a * b for a, b in sizes)
        inner = sum(max(0, a - 2 * case["pml"]) * max(0, b - 2 * case["pml"]) for a, b in sizes)
        return {"bytes": cells * (4 * (2 * 3 + 1) + 3 * 8) + 4 * 6 * (cells - inner),
                "flops": case["steps"] * (16.0 * cells + 21.0 * (cells - inner))}
    n = _sides(case)
    cells = math.prod(n)
    outer = cells - math.prod(v - 2 * case["pml"] for v in n)
    if case["kind"] == "adjoint":
        # forward, recomputed forward and reverse sweep; eps read, the gradient written
        return {"bytes": cells * (4 + 8) + 16 * 16 * 4, "flops": case["steps"] * 3 * (16.0 * cells + 21.0 * outer)}
    word = WORD[case["precision"]]
    comps = 6 if len(n) == 3 else 3
    aux = 8 if word == 8 else 4
    data = cells * (2 * comps * word + aux) + outer * 2 * comps * aux + cells * comps * 8
    ops = case["steps"] * ((5.0 * comps if len(n) == 3 else 12.0) * cells + 7.0 * comps * outer)
    if case["kind"] == "drude":
        m = case["tfsf"] + 2
        slab = (n[0] - 2 * m) * (n[1] - 2 * m) * (n[2] // 6)
        data += slab * comps * 4 * (2 * 4) + 4 * 4 * slab
        ops += case["steps"] * slab * comps * 12.0
    return {"bytes": float(data), "flops": float(ops)}


def tolerance(case):
    # the FP64 form keeps the reference's order of operations: its fields are the same bit for bit
    if case.get("precision") == "fp64":
        return "exact"
    # FP16 storage rounds every field to 11 bits each step: two correct forms differ by that rounding's walk (8e-4 to
    # 2e-3 off the restatement)
    if case.get("precision") == "fp16":
        return {"rel": 1e-2}
    # FP32 forms are 1e-7 to 4e-6 off the FP64 restatement, the weakest components most
    return {"rel": 1e-5}


# ------------------------------------------------------- FP64 restatement


def _sigma(n, pml, first):
    """The PML conductivity along one axis (sixth-order profile; the first axis keeps the fractional distance, the
    others truncate it and end half a cell later)."""
    out = np.zeros(n)
    bound = pml * DX32
    peak = -math.log(1e-16) * 7.0 / (2.0 * math.sqrt(MU0 / EPS0) * bound)
    scale = peak / (DX32 * bound ** 6 * 7)
    for i in range(n):
        size = n if first else n + 0.5
        d = pml - (i + 0.5) if i + 0.5 < pml else ((i + 0.5) - (size - pml) if i + 0.5 >= size - pml else None)
        if d is not None:
            d = d if first else int(d)
            out[i] = scale * (((d + 1) * DX32) ** 7 - (d * DX32) ** 7)
    return out


# the run's scalars are single-precision numbers, as the command line parses them
DX32, WAVELENGTH32 = float(np.float32(DX)), float(np.float32(WAVELENGTH))
DT = DX32 * COURANT / C0
FREQUENCY = C0 / WAVELENGTH32


def _phase_velocity(a1, a2):
    """Numerical phase velocity along the direction (a1, a2)."""
    s = math.sin(math.pi * COURANT / (WAVELENGTH32 / DX32))
    flat = [any(abs(a - q * math.pi / 2) < 1e-12 for q in range(4)) for a in (a1, a2)]
    if all(flat):
        k = 2.0 / DX32 * math.asin(s / COURANT)
    else:
        # the plane wave's numerical dispersion relation, by Newton's method to the accuracy the step uses
        nd = DX32 / WAVELENGTH32
        a = (nd * math.sin(a1) * math.cos(a2) / 2, nd * math.sin(a1) * math.sin(a2) / 2, nd * math.cos(a1) / 2)
        k, last = 2 * math.pi, 2 * math.pi + 1
        while (last - k) ** 2 >= 1e-7:
            last = k
            f = sum(math.sin(v * k) ** 2 for v in a) - (s / COURANT) ** 2
            k -= f / sum(v * math.sin(2 * v * k) for v in a)
        k /= WAVELENGTH32
    return C0 * 2 * math.pi / WAVELENGTH32 / k


class _Exact:
    """The leapfrog step in FP64 torch: curl, PML (D and B), Drude, TF/SF with its 1-D grid, a hard point source.
    Components E_a sit at 1.0 on their own axis and 0.5 on the others, H_a the other way round."""

    def __init__(self, kw, materials):
        n = tuple(kw["size"])
        self.flat = len(n) == 2
        self.n = n + (1,) if self.flat else n
        self.kw = kw
        self.comps = (2, 3, 4) if self.flat else tuple(range(6))
        self.F = {k: self._zeros() for k in self.comps}
        self.D = {k: [self._zeros()] for k in self.comps}
        self.drude = bool(kw.get("use_metamaterials"))
        if self.drude:
            self.D = {k: [self._zeros() for _ in range(2)] for k in self.comps}
            self.Z = {k: [self._zeros() for _ in range(2)] for k in self.comps}
        self.inner = tuple(slice(1, v - 1) if v > 1 else slice(0, 1) for v in self.n)
        self.sigma = [_sigma(self.n[a], kw["pml"], a == 0) if self.n[a] > 1 else np.zeros(1) for a in range(3)]
        self.eps = materials["eps"].reshape(self.n)
        self.t = 0
        self._coefficients()
        self.mean = {k: self._mean(self.eps, k) for k in self.comps if k < 3}
        if self.drude:
            self.medium = {k: [self._mean(materials[q], k) for q in names] for k in self.comps
                           for names in [("omegape", "gammae") if k < 3 else ("omegapm", "gammam")]}
        if kw.get("use_tfsf"):
            self._incident()

    def _zeros(self):
        return torch.zeros(self.n, dtype=torch.float64, device=DEVICE)

    def _at(self, v, shift=(0, 0, 0)):
        """The inner cells of v, moved by `shift` (nothing moves along a dropped axis)."""
        return v[tuple(slice(s.start + d, s.stop + d) if m > 1 else s for s, d, m in zip(self.inner, shift, self.n))]

    @staticmethod
    def _unit(axis, step):
        return tuple(step if a == axis else 0 for a in range(3))

    def _mean(self, v, k):
        a = k % 3
        if k < 3:
            return (self._at(v) + self._at(v, self._unit(a, 1))) / 2
        b, c = self._unit((a + 1) % 3, 1), self._unit((a + 2) % 3, 1)
        return (self._at(v) + self._at(v, b) + self._at(v, c) + self._at(v, tuple(p + q for p, q in zip(b, c)))) / 4

    def _profile(self, k, axis):
        s = self.sigma[axis]
        if self.n[axis] > 1 and (axis == k % 3) == (k < 3):
            s = np.concatenate([(s[:-1] + s[1:]) / 2, s[-1:]])
        shape = [1, 1, 1]
        shape[axis] = -1
        return torch.from_numpy(s[self.inner[axis]]).to(DEVICE).reshape(shape)

    def _coefficients(self):
        self.coef = {}
        for k in self.comps:
            a = k % 3
            s1, s4, s5 = (self._profile(k, x) for x in ((a + 1) % 3, a, (a + 2) % 3))
            ca, cb = (2 * EPS0 - s1 * DT) / (2 * EPS0 + s1 * DT), (2 * EPS0 * DT / DX32) / (2 * EPS0 + s1 * DT)
            ca2 = (2 * EPS0 - s5 * DT) / (2 * EPS0 + s5 * DT)
            p4, m4 = (2 * EPS0 + s4 * DT) / (2 * EPS0 + s5 * DT), (2 * EPS0 - s4 * DT) / (2 * EPS0 + s5 * DT)
            self.coef[k] = (ca, cb, ca2, p4, m4)

    # the incident wave

    def _incident(self):
        kw = self.kw
        a1, a2, a3 = (float(kw[v]) * math.pi / 180 for v in ("teta", "phi", "psi"))
        ratio = _phase_velocity(math.pi / 2, 0.0) / _phase_velocity(a1, a2)
        self.mod = (DT / (ratio * EPS0 * DX32), DT / (ratio * MU0 * DX32))
        s1, c1, s2, c2, s3, c3 = (f(v) for v in (a1, a2, a3) for f in (math.sin, math.cos))
        if self.flat:
            self.k = (c2, s2, 0.0)
            self.proj = {2: 1.0, 3: s2, 4: -c2}
        else:
            self.k = (s1 * c2, s1 * s2, c1)
            self.proj = dict(enumerate((c3 * s2 - s3 * c1 * c2, -c3 * c2 - s3 * c1 * s2, s3 * s1,
                                        s3 * s2 + c3 * c1 * c2, -s3 * c2 + c3 * c1 * s2, -c3 * s1)))
        left = kw["tfsf_left"]
        self.origin = [left - 2.5 * v if m > 1 else 0.0 for v, m in zip(self.k, self.n)]
        self.inc = torch.zeros(2, 500 * self.n[0], dtype=torch.float64, device=DEVICE)
        self.boxes = {k: list(self._borders(k)) for k in self.comps}

    def _positions(self, k, axis):
        edge = (axis == k % 3) == (k < 3)
        return np.arange(self.n[axis]) + (0.0 if self.n[axis] == 1 else (1.0 if edge else 0.5))

    def _borders(self, k):
        """(cells, sign, axis, offset, component) of every border term: on `cells`, the neighbour at `offset` along
        `axis` is on the other side of the box, and the incident value of `component` there makes up for it."""
        a, is_h = k % 3, k >= 3
        for number, (other, axis) in enumerate(self._circuit(k)):
            if other not in self.comps or self.n[axis] == 1:
                continue
            for upper in (False, True):
                lo, hi = self.kw["tfsf_left"], self.n[axis] - self.kw["tfsf_right"]
                place = (hi if upper else lo) + (0.0 if is_h else (0.5 if upper else -0.5))
                cells = []
                for b in range(3):
                    x = self._positions(k, b)
                    if self.n[b] == 1:
                        ok = np.ones(1, bool)
                    else:
                        l, r = self.kw["tfsf_left"], self.n[b] - self.kw["tfsf_right"]
                        if b == axis:
                            ok = np.abs(x - place) < 1e-6
                        elif (b == a) == is_h:
                            ok = (x > l + 0.4) & (x < r - 0.4)
                        else:
                            ok = (x > l - 0.1) & (x < r + 0.1)
                        ok[[0, -1]] = False
                    at = np.nonzero(ok)[0]
                    if not len(at):
                        break
                    cells.append(slice(int(at[0]), int(at[-1]) + 1))
                else:
                    # E takes it from the neighbour inside the box, H from the one outside
                    offset = (0 if not upper else -1) if not is_h else (0 if not upper else 1)
                    far = (offset == 0) if not is_h else (offset == 1)
                    sign = (-1.0 if far else 1.0) * (1.0 if number == 0 else -1.0) * (-1.0 if is_h else 1.0)
                    yield tuple(cells), sign, self._unit(axis, offset), other

    def _circuit(self, k):
        """The two (component, axis) whose differences make the curl of component k: first minus second."""
        a = k % 3
        if k < 3:
            return ((a + 2) % 3 + 3, (a + 1) % 3), ((a + 1) % 3 + 3, (a + 2) % 3)
        return ((a + 1) % 3, (a + 2) % 3), ((a + 2) % 3, (a + 1) % 3)

    def _incident_at(self, k, cells, shift):
        d = torch.zeros(1, 1, 1, dtype=torch.float64, device=DEVICE)
        for b in range(3):
            if self.n[b] > 1:
                x = self._positions(k, b)[cells[b]] + shift[b] - self.origin[b]
                shape = [1, 1, 1]
                shape[b] = -1
                d = d + torch.from_numpy(x * self.k[b]).to(DEVICE).reshape(shape)
        d = d - (0.5 if k >= 3 else 0.0)
        i = d.to(torch.int64)
        w = d - i
        line = self.inc[1 if k >= 3 else 0]
        return (line[i] * (1 - w) + line[i + 1] * w) * self.proj[k]

    # one half step

    def _half(self, family):
        update = self.t > 0
        for k in self.comps:
            if not update or (k >= 3) != (family == 1):
                continue
            low, high = (-1, 0) if family == 0 else (0, 1)
            curl = None
            for sign, (other, axis) in zip((1, -1), self._circuit(k)):
                if other in self.F:
                    v = self._at(self.F[other], self._unit(axis, high)) - self._at(self.F[other], self._unit(axis, low))
                    curl = sign * v if curl is None else (curl.add_(v, alpha=sign) if not v.requires_grad else curl + sign * v)
            if self.kw.get("use_tfsf"):
                for cells, sign, shift, other in self.boxes[k]:
                    at = tuple(slice(c.start - s.start, c.stop - s.start) for c, s in zip(cells, self.inner))
                    curl[at] += sign * self._incident_at(other, cells, shift)
            ca, cb, ca2, p4, m4 = self.coef[k]
            old = self.D[k][0]
            new = self._at(old) * ca + curl * cb
            unit = EPS0 if k < 3 else MU0
            m = self.mean.get(k)
            if self.drude:
                w, g = self.medium[k]
                m = 1.0 if m is None else m
                sq = unit * (DT * w) ** 2
                A = 4 * unit * m + 2 * DT * unit * m * g + sq
                z0, z1 = (self._at(v) for v in self.Z[k])
                z = ((4 + 2 * DT * g) * new - 8 * self._at(old) + (4 - 2 * DT * g) * self._at(self.D[k][1])
                     - (2 * sq - 8 * unit * m) * z0 - (4 * unit * m - 2 * DT * unit * m * g + sq) * z1) / A
                field = self._at(self.F[k]) * ca2 + z * p4 - z0 * m4
                self.Z[k] = [self._put(self.Z[k][1], z), self.Z[k][0]]
                self.D[k] = [self._put(self.D[k][1], new), self.D[k][0]]
            else:
                step = (new * p4 - self._at(old) * m4) / unit
                field = self._at(self.F[k]) * ca2 + (step if m is None else step / m)
                self.D[k] = [self._put(old, new)]
            self.F[k] = self._put(self.F[k], field)
        if self.kw.get("point_source_mask") and family == 0:
            at = tuple(self.kw["point_source"]) + ((0,) if self.flat else ())
            self.F[2] = self._set(self.F[2], at, self._pulse())

    def _put(self, v, inner):
        v[self.inner] = inner
        return v

    def _set(self, v, at, value):
        v[at] = value
        return v

    def _pulse(self):
        w = 4 * math.sqrt(math.log(2)) / (math.pi * FREQUENCY * self.kw["point_source_bandwidth"])
        tau = DT * (self.t + 0.5) - 3 * w
        return math.exp(-(tau / w) ** 2) * math.sin(2 * math.pi * FREQUENCY * tau)

    def step(self):
        for family in (0, 1):
            if self.kw.get("use_tfsf"):
                e, h = self.inc
                if family == 0:
                    e[1:] += (h[:-1] - h[1:]) * self.mod[0]
                    e[0] = math.sin(DT * self.t * 2 * math.pi * FREQUENCY)
                else:
                    h[:-1] += (e[:-1] - e[1:]) * self.mod[1]
            self._half(family)
        self.t += 1

    def fields(self):
        return {fd.COMPONENTS[k]: (v[..., 0] if self.flat else v) for k, v in self.F.items()}

    def energy(self):
        total = sum(float(((self.eps if k < 3 else MU0 / EPS0) * v * v).sum()) for k, v in self.F.items())
        return total


class _Differentiable(_Exact):
    """The same step with nothing written in place, so that torch differentiates it."""

    def _put(self, v, inner):
        return torch.nn.functional.pad(inner, [0, 0, 1, 1, 1, 1])

    def _set(self, v, at, value):
        return v.index_put([torch.tensor([q], device=DEVICE) for q in at],
                           torch.tensor([value], dtype=v.dtype, device=DEVICE))


def exact(case, seed):
    if case["kind"] == "batch":
        sizes, maps = _batch_inputs(case, seed)
        got = {c: [] for c in ("Ez", "Hx", "Hy")}
        for size, eps in zip(sizes, maps):
            ref = _Exact(dict(BATCH_PHYSICS, size=size, pml=case["pml"], point_source=(size[0] // 2, size[1] // 2)),
                         {"eps": eps})
            for _ in range(case["steps"]):
                ref.step()
            for c, v in ref.fields().items():
                got[c].append(v.cpu().numpy().reshape(-1))
        return {c: np.concatenate(v) for c, v in got.items()}
    kw, materials = _physics(case), _materials(case, seed)
    if case["kind"] == "adjoint":
        _, _, _, lo, hi = _adjoint_places(_sides(case))
        eps = materials["eps"].requires_grad_(True)
        ref = _Differentiable(kw, {"eps": eps})
        value = torch.zeros((), dtype=torch.float64, device=DEVICE)
        for _ in range(case["steps"]):
            # the objective takes Ez after the E half step and the source: H does not touch it
            ref.step()
            value = value + ref.F[2][lo[0]:hi[0], lo[1]:hi[1], 0].square().sum()
        (gradient,) = torch.autograd.grad(value, eps)
        return {"objective": float(value.detach()), "gradient": gradient.cpu().numpy()}
    ref = _Exact(kw, materials)
    if case.get("resume"):
        for name, values in _noise(case, seed):
            ref.F[fd.COMPONENTS.index(name)] = values
        ref.t = RESUMED
    for _ in range(case["warm"]):
        ref.step()
    spectrum = None
    if case["kind"] == "drude":
        spectrum = torch.zeros(case["nx"], case["ny"], dtype=torch.complex128, device=DEVICE)
    for _ in range(case["steps"]):
        ref.step()
        if spectrum is not None:
            phase = 2 * math.pi * 15e9 * (ref.t - 0.5) * DT
            spectrum += ref.F[0][:, :, _dft_plane(case)] * complex(math.cos(phase), -math.sin(phase))
    out = ref.fields()
    if spectrum is not None:
        out["dft_re"], out["dft_im"] = spectrum.real[None].contiguous(), spectrum.imag[None].contiguous()
    elif case["kind"] == "grid" and case["source"] == "point":
        out["energy"] = ref.energy()
    elif case["kind"] == "tmz":
        out = {c: v.cpu().numpy() for c, v in out.items()}
    return out
