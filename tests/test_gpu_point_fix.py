"""Point sources of the FP32 / FP16 3-D runs as the step's (or the pair's)
linear response, against the FP64 plain form: places from next to the PML to
the middle of a tile, every component, runs that end on pairs and on single
steps, with and without TF/SF."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _run(fdtd, kw, prec, mats, calls):
    with fdtd.Simulation(precision=prec, materials=mats, **kw) as sim:
        for n in calls:
            sim.step(n)
        return sim.step_kernel, {c: sim.field(c) for c in COMPS}


# PML 4: cells 4 .. n - 5 are free of it.  4: the cell below is PML (inside
# the sweep); 5, 6: single steps only; 7: the first with pairs; (17, 15, 63)
# and 64: a z tile's seam of the two-step sweep; 20: middle; n - 6, n - 8: the
# high side
@pytest.mark.parametrize("pos", [(4, 9, 20), (5, 9, 20), (9, 6, 20), (9, 7, 20), (17, 15, 63), (17, 15, 64),
                                 (16, 14, 20), (27, 9, 20), (30, 24, 66)])
@pytest.mark.parametrize("mask", [1 << 2, 1 << 4, (1 << 0) | (1 << 1) | (1 << 5), 0x3f])
@pytest.mark.parametrize("tfsf", [False, True])
def test_point_source_response_matches_fp64(fdtd, monkeypatch, pos, mask, tfsf):
    monkeypatch.setenv("FDTDB_TB2", "1")   # (pairs on a grid too small for them by default)
    shape = (36, 30, 72)
    rng = np.random.default_rng(1)
    eps = 1 + np.kron(rng.uniform(0, 3, (6, 5, 12)), np.ones((6, 6, 6))).astype(np.float32).astype(np.float64)
    kw = dict(mode=3, size=shape, use_pml=True, pml=4, point_source=pos, point_source_mask=mask)
    if tfsf:
        kw.update(use_tfsf=True, tfsf_left=8, tfsf_right=8, teta=30, phi=40, psi=20)
    for calls in ([30], [1, 22, 8]):
        _, want = _run(fdtd, kw, 0, {"eps": eps}, calls)
        for prec, tol in ((1, 1e-5), (2, 2e-2)):
            kernel, got = _run(fdtd, kw, prec, {"eps": eps}, calls)
            assert kernel in ("sweep3d_tma", "sweep2_tma"), kernel
            if not tfsf and calls == [1, 22, 8] and all(7 <= c <= n - 8 for c, n in zip(pos, shape)):
                assert kernel == "sweep2_tma", kernel
            for fam in "EH":
                g = np.concatenate([got[c].ravel() for c in COMPS if c[0] == fam])
                w = np.concatenate([want[c].ravel() for c in COMPS if c[0] == fam])
                err = np.linalg.norm(g - w) / np.linalg.norm(w)
                # a point source concentrates the field on a few cells (1e-5 for plane waves, 2e-5 here)
                assert err <= 2 * tol, (prec, calls, fam, err)
