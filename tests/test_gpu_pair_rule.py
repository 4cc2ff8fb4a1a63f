"""Which 3-D FP32 / FP16-storage runs advance in pairs of steps by default.

FP16 storage rounds once per pass over the fields: pairs are its more exact
form, so grids whose rows are whole 16-byte units take them at every size.
Other runs take them where they measured faster; on either side of each line
the fields are the same to the accuracy of the form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
TFSF = dict(use_tfsf=True, tfsf_left=14, tfsf_right=14, teta=30, phi=45, psi=25)


def _error(got, want):
    return max(np.linalg.norm(np.concatenate([(got[c] - want[c]).ravel() for c in COMPS if c[0] == f])) /
               np.linalg.norm(np.concatenate([want[c].ravel() for c in COMPS if c[0] == f])) for f in "EH")


@pytest.mark.parametrize("tfsf", [False, True])
def test_fp16_default_is_as_exact_as_pairs(fdtd, monkeypatch, tfsf):
    n = (64, 60, 72)
    rng = np.random.default_rng(3)
    fields = {}
    for c in COMPS:
        fields[c] = np.zeros(n)
        fields[c][1:-1, 1:-1, 1:-1] = rng.standard_normal([v - 2 for v in n]) / (1 if c[0] == "E" else 376.73)
    kw = dict(mode=3, size=n, use_pml=True, pml=6, **(TFSF if tfsf else {}))
    out = {}
    for name, prec, tb2 in (("fp64", 0, None), ("default", 2, None), ("pairs", 2, "1"), ("single", 2, "0")):
        monkeypatch.delenv("FDTDB_TB2", raising=False)
        if tb2:
            monkeypatch.setenv("FDTDB_TB2", tb2)
        with fdtd.Simulation(precision=prec, **kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.step(40, t_start=500)
            out[name] = {c: sim.field(c) for c in COMPS}
            if name == "default":
                assert sim.step_kernel == "sweep2_tma", sim.step_kernel
    err = {k: _error(v, out["fp64"]) for k, v in out.items() if k != "fp64"}
    assert err["default"] == err["pairs"] < err["single"], err


PS = dict(point_source_mask=1 << 2)
PML = dict(use_pml=True, pml=6)


# (cells, what is on, precision, pairs)
@pytest.mark.parametrize("n,kw,prec,pairs", [
    ((64, 64, 64), {}, 1, False),                  # no PML: from 3 M cells
    ((128, 128, 128), PS, 1, False),
    ((128, 128, 128), PS, 2, False),
    ((145, 144, 144), PS, 1, True),
    ((145, 144, 144), PS, 2, True),
    ((64, 64, 64), {}, 2, True),                   # FP16, whole rows
    ((60, 60, 61), {}, 2, False),                  # FP16, padded rows
    ((64, 64, 64), PML, 2, True),
    ((248, 246, 245), PML, 1, False),              # PML: from 15 M cells
    ((248, 248, 248), {**PML, **PS}, 1, True),
    ((260, 230, 33), {**PML, **PS}, 1, False),     # short rows: from 2 M cells
    ((260, 240, 33), {**PML, **PS}, 1, True),
    ((260, 240, 33), PS, 2, True),
    ((128, 128, 128), {**PML, **TFSF, "tfsf_left": 22, "tfsf_right": 22, "pml": 12}, 1, True),   # PML and TF/SF: 2 M
    ((120, 128, 128), {**PML, **TFSF, "tfsf_left": 22, "tfsf_right": 22, "pml": 12}, 1, False),
])
def test_runs_in_pairs(fdtd, monkeypatch, n, kw, prec, pairs):
    kw = dict(kw, mode=3, size=n)
    if kw.get("point_source_mask"):
        kw["point_source"] = tuple(v // 2 for v in n)
    out = []
    for tb2 in (None, "0" if pairs else "1"):
        monkeypatch.delenv("FDTDB_TB2", raising=False)
        if tb2:
            monkeypatch.setenv("FDTDB_TB2", tb2)
        with fdtd.Simulation(precision=prec, **kw) as sim:
            rng = np.random.default_rng(1)
            for c in ("Ex", "Hz"):
                v = np.zeros(n)
                v[1:-1, 1:-1, 1:-1] = rng.standard_normal([k - 2 for k in n]) / (1 if c[0] == "E" else 376.73)
                sim.set_field(c, v)
            sim.step(4, t_start=100)
            if tb2 is None:
                assert sim.step_kernel == ("sweep2_tma" if pairs else "sweep3d_tma"), sim.step_kernel
            out.append({c: sim.field(c) for c in COMPS})
    # 4 steps of the two forms: their roundings
    assert _error(out[0], out[1]) <= (2e-6 if prec == 1 else 5e-3)
