"""The Drude fix-up of the sweep (four cells per thread, levels two steps back
kept in the alternating sets): boxes at every remainder of the vector, FP32
and FP16, against the FP64 plain form; and a run that moves between the sweep
and the register-blocked kernel keeps its Drude state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
OM, GA = np.float32(2 * np.pi * 30e9), np.float32(2 * np.pi * 1e9)


def _case(shape, box):
    om, ga = np.zeros(shape), np.zeros(shape)
    om[box], ga[box] = OM, GA
    rng = np.random.default_rng(4)
    fields = {c: np.zeros(shape) for c in COMPS}
    for c in COMPS:
        fields[c][1:-1, 1:-1, 1:-1] = rng.standard_normal(tuple(n - 2 for n in shape)) / (1 if c[0] == "E" else 376.73)
    eps = 1 + np.kron(rng.uniform(0, 2, tuple(n // 5 + 1 for n in shape)), np.ones((5, 5, 5)))
    eps = eps[: shape[0], : shape[1], : shape[2]].astype(np.float32).astype(np.float64)
    return {"eps": eps, "omegape": om, "omegapm": om, "gammae": ga, "gammam": ga}, fields


def _family(got, want, fam):
    g = np.concatenate([got[c].ravel() for c in COMPS if c[0] == fam])
    w = np.concatenate([want[c].ravel() for c in COMPS if c[0] == fam])
    return np.linalg.norm(g - w) / np.linalg.norm(w)


@pytest.mark.parametrize("z0", [8, 9, 10, 11])
@pytest.mark.parametrize("dz", [1, 2, 5, 16])
@pytest.mark.parametrize("nz", [40, 43])
@pytest.mark.parametrize("prec,tol", [(1, 1e-5), (2, 2e-2)])
def test_fix_up_matches_fp64(fdtd, z0, dz, nz, prec, tol):
    shape = (20, 18, nz)
    mats, fields = _case(shape, (slice(7, 13), slice(6, 11), slice(z0, z0 + dz)))
    kw = dict(mode=3, size=shape, use_pml=True, pml=3, use_metamaterials=True)
    out = {}
    for p in (0, prec):
        with fdtd.Simulation(materials=mats, precision=p, **kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.step(21, t_start=9)
            out[p] = {c: sim.field(c) for c in COMPS}
            assert not p or sim.step_kernel == "sweep3d_tma", sim.step_kernel
    for fam in "EH":
        assert _family(out[prec], out[0], fam) <= tol, (fam, _family(out[prec], out[0], fam))


def test_drude_state_moves_between_the_kernels(fdtd, monkeypatch):
    shape = (20, 18, 40)
    mats, fields = _case(shape, (slice(7, 13), slice(6, 11), slice(10, 21)))
    kw = dict(mode=3, size=shape, use_pml=True, pml=3, use_metamaterials=True)
    out = {}
    for p in (0, 1):
        with fdtd.Simulation(materials=mats, precision=p, **kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.t = 9
            kernels = []
            for sweep in "1010":
                monkeypatch.setenv("FDTDB_SWEEP", sweep)
                sim.set_material("omegape", mats["omegape"])   # (an upload has the steps planned again)
                sim.step(7)
                kernels.append(sim.step_kernel)
            out[p] = {c: sim.field(c) for c in COMPS}
            if p:
                assert kernels == ["sweep3d_tma", "fused3d_regblock"] * 2, kernels
    for fam in "EH":
        assert _family(out[1], out[0], fam) <= 1e-5, (fam, _family(out[1], out[0], fam))
