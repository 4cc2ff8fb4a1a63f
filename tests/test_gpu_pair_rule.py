"""Which 3-D FP32 / FP16-storage runs advance in pairs of steps by default.

FP16 storage rounds once per pass over the fields: pairs are its more exact
form, so grids whose rows are whole 16-byte units take them at every size."""
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
