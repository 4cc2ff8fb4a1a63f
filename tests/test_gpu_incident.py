"""The 1-D incident grid as a job of other launches (one combined launch, the
sweep's own launch, the FP64 half-steps'): the same bits in every form, and the
sweep's corrections from it as right as the pairs'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(40, 44, 48), (40, 30, 27)])
@pytest.mark.parametrize("steps", [1, 2, 3, 64])
def test_incident_levels_agree_between_forms(fdtd, monkeypatch, size, steps):
    kw = dict(mode=3, size=size, use_pml=True, pml=4, use_tfsf=True, tfsf_left=8, tfsf_right=8, teta=30, phi=45,
              psi=20)
    got = {}
    for name, prec, tb2 in (("plain", 0, "0"), ("single", 1, "0"), ("pairs", 1, "1"), ("half", 2, "0")):
        monkeypatch.setenv("FDTDB_TB2", tb2)
        with fdtd.Simulation(precision=prec, **kw) as sim:
            sim.step(steps)
            sim.step(steps + 1)
            got[name] = {"E": sim.incident("E"), "H": sim.incident("H"),
                         "f": np.concatenate([sim.field(c).ravel() for c in ("Ex", "Ey", "Ez")])}
    ref = got["plain"]
    assert np.any(ref["E"] != 0)
    for name, g in got.items():
        for f in ("E", "H"):
            assert np.array_equal(g[f], ref[f]), (name, f)
        # (a wave of a few steps is below what FP16 storage holds)
        tol = 2e-2 if name == "half" else 1e-5
        if steps == 64:
            assert np.linalg.norm(g["f"] - ref["f"]) <= tol * np.linalg.norm(ref["f"]), name
