"""Point sources of the FP32 / FP16 3-D runs outside the sweep (the cells the
source's value reaches worked out again after the step or the pair), against
the FP64 plain form: places from next to the PML to the middle of a tile, every
component, runs that end on pairs and on single steps, with and without TF/SF;
and against the same source inside the sweep, bit for bit."""
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


def _noise_run(fdtd, monkeypatch, prec, pos, mask, steps, tb2, fix, **kw):
    monkeypatch.setenv("FDTDB_TB2", tb2)
    monkeypatch.setenv("FDTDB_POINT_FIX", fix)
    shape = (36, 30, 72)
    rng = np.random.default_rng(2)
    eps = 1 + np.kron(rng.uniform(0, 3, (6, 5, 12)), np.ones((6, 6, 6))).astype(np.float32).astype(np.float64)
    with fdtd.Simulation(precision=prec, materials={"eps": eps}, mode=3, size=shape, use_pml=True, pml=4,
                         point_source=pos, point_source_mask=mask, **kw) as sim:
        for c in COMPS:
            v = np.zeros(shape)
            v[1:-1, 1:-1, 1:-1] = rng.standard_normal([n - 2 for n in shape]) / (1 if c[0] == "E" else 376.73)
            sim.set_field(c, v)
        sim.step(steps, t_start=100)
        return {c: sim.field(c) for c in COMPS}, sim.step_kernel


@pytest.mark.parametrize("pos", [(5, 9, 20), (9, 6, 20), (17, 15, 63), (17, 15, 64), (16, 14, 20), (30, 24, 66)])
@pytest.mark.parametrize("mask", [1 << 2, 1 << 4, 0x3f])
@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("tfsf", [False, True])
def test_single_steps_keep_the_bits_of_the_source_inside_the_sweep(fdtd, monkeypatch, pos, mask, prec, tfsf):
    kw = dict(use_tfsf=True, tfsf_left=8, tfsf_right=8, teta=30, phi=40, psi=20) if tfsf else {}
    got = [_noise_run(fdtd, monkeypatch, prec, pos, mask, 9, "0", fix, **kw)[0] for fix in "10"]
    for c in COMPS:
        assert np.array_equal(got[0][c], got[1][c]), (c, np.max(np.abs(got[0][c] - got[1][c])))


@pytest.mark.parametrize("pos", [(9, 7, 20), (17, 15, 63), (16, 14, 20)])
def test_pairs_lose_nothing_around_the_source(fdtd, monkeypatch, pos):
    box = tuple(slice(p - 5, p + 6) for p in pos)
    want, _ = _noise_run(fdtd, monkeypatch, 0, pos, 0x3f, 30, "0", "1")
    for prec in (1, 2):
        err = []
        for tb2, fix in (("1", "1"), ("0", "0")):
            got, kernel = _noise_run(fdtd, monkeypatch, prec, pos, 0x3f, 30, tb2, fix)
            assert kernel == ("sweep2_tma" if tb2 == "1" else "sweep3d_tma"), kernel
            err.append([np.linalg.norm(np.concatenate([(got[c] - want[c])[box].ravel() for c in COMPS if c[0] == f])) /
                        np.linalg.norm(np.concatenate([want[c][box].ravel() for c in COMPS if c[0] == f])) for f in "EH"])
        for pairs, single in zip(*err):
            # FP32: both forms round every operation the same number of times; FP16 pairs round the fields half as often
            assert pairs <= (1.2 if prec == 1 else 1.0) * single, (prec, err)


@pytest.mark.parametrize("nz", [28, 26])   # the TMA sweep, the register-blocked one
@pytest.mark.parametrize("off", [(0, 0, 0), (0, 0, 1), (0, 1, 0), (1, 0, 0)])
def test_current_on_and_beside_a_point_source(fdtd, nz, off):
    pos = (11, 10, 13)
    kw = dict(mode=3, size=(24, 22, nz), use_pml=True, pml=4, point_source=pos, point_source_mask=(1 << 2) | (1 << 4),
              current_source=tuple(p + o for p, o in zip(pos, off)), current_source_mask=(1 << 2) | (1 << 4) | (1 << 0))
    out = {}
    for prec in (0, 1):
        with fdtd.Simulation(precision=prec, **kw) as sim:
            sim.step(40)
            out[prec] = {c: sim.field(c) for c in COMPS}
            assert not prec or sim.step_kernel == ("sweep3d_tma" if nz == 28 else "fused3d_regblock"), sim.step_kernel
    for fam in "EH":
        g, w = (np.concatenate([out[p][c].ravel() for c in COMPS if c[0] == fam]) for p in (1, 0))
        # (the bound of the current sources' own FP32 test)
        assert np.linalg.norm(g - w) <= 2e-5 * np.linalg.norm(w), (fam, np.linalg.norm(g - w) / np.linalg.norm(w))
