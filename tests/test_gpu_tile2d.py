"""2-D modes: several steps per launch (tile2d) against one step per call.
A call of one step from t > 0 is a launch of one step; calls of n steps take
launches of up to seven.  FP64: bit for bit, and against the oracle in TMz;
FP32: to rounding."""
import numpy as np
import pytest

from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

MODES = {"tmz": 2, "tex": 4, "tey": 5, "tez": 6, "tmx": 7, "tmy": 8}
# 3 x 3: one updated cell; 18 x 18: exactly one small tile; 19 x 51 and 51 x
# 19: one cell past a tile of either kind; 420 x 380 and 330 x 700: large tiles
SIZES = [(3, 3), (18, 18), (19, 51), (51, 19), (97, 133), (420, 380)]


def _setup(fdtd, mode, size, source, seed, mu=False):
    rng = np.random.default_rng(seed)
    kw = dict(mode=mode, size=size, teta=40, phi=25, psi=20)
    if min(size) > 16:
        kw.update(use_pml=True, pml=4)
    if source == "tfsf" and min(size) > 16:
        kw.update(use_tfsf=True, tfsf_left=6, tfsf_right=6)
    else:
        kw.update(point_source=tuple(n // 2 for n in size), point_source_mask=0x3f)
    blocks = rng.uniform(1, 4, tuple(n // 5 + 1 for n in size)).astype(np.float32).astype(np.float64)
    mats = {"eps": np.kron(blocks, np.ones((5, 5)))[: size[0], : size[1]]}
    if mu:
        mats["mu"] = mats["eps"][::-1, ::-1] / 2 + 0.5
    # noise with nonzero faces: FP64 alternates two levels of the faces
    fields = {c: rng.standard_normal(size) / (1 if c[0] == "E" else 376.73) for c in fdtd.MODE_COMPONENTS[mode]}
    return kw, mats, fields


def _run(fdtd, kw, mats, fields, prec, calls):
    with fdtd.Simulation(materials=mats, precision=prec, **kw) as sim:
        sim.step(3)
        for c, v in fields.items():
            sim.set_field(c, v)
        for n in calls:
            sim.step(n)
        return {c: sim.field(c) for c in fields}


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("source", ["tfsf", "point"])
def test_fp64_launches_of_any_length_agree(fdtd, mode, size, source):
    for layout in (0, 1):
        kw, mats, fields = _setup(fdtd, MODES[mode], size, source, 7, mu=layout == 1)
        kw["layout"] = layout
        want = _run(fdtd, kw, mats, fields, 0, [1] * 24)
        for calls in ([24], [7, 2, 15], [4, 6, 14]):
            got = _run(fdtd, kw, mats, fields, 0, calls)
            for c in want:
                assert np.array_equal(got[c].view(np.int64), want[c].view(np.int64)), (layout, calls, c)


@pytest.mark.parametrize("size", SIZES[1:])
def test_fp64_tmz_matches_oracle(fdtd, size):
    kw, mats, _ = _setup(fdtd, 2, size, "tfsf", 9)
    o = Oracle(materials=mats, **kw)
    o.step(40)
    with fdtd.Simulation(materials=mats, **kw) as sim:
        sim.step(40)
        for c in ("Ez", "Hx", "Hy"):
            got, want = sim.field(c), np.asarray(o.field(c)).reshape(size)
            assert np.array_equal(got.view(np.int64), want.view(np.int64)), c
        inc = sim.incident("E")
        assert np.all(inc[41:] == 0) and np.any(inc[:41] != 0)
    o.close()


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("size", SIZES[1:])
@pytest.mark.parametrize("source", ["tfsf", "point"])
@pytest.mark.parametrize("prec,tol", [(1, 1e-5), (2, 2e-2)])
def test_fast_forms_match_fp64(fdtd, mode, size, source, prec, tol):
    for layout in (0, 1):
        kw, mats, fields = _setup(fdtd, MODES[mode], size, source, 3, mu=layout == 1)
        kw["layout"] = layout
        for v in fields.values():   # (FP64 alternates the faces' two levels, the fast forms keep one)
            v[[0, -1], :] = 0
            v[:, [0, -1]] = 0
        want = _run(fdtd, kw, mats, fields, 0, [25])
        got = _run(fdtd, kw, mats, fields, prec, [4, 21])
        for fam in "EH":
            g = np.concatenate([got[c].ravel() for c in got if c[0] == fam])
            w = np.concatenate([want[c].ravel() for c in want if c[0] == fam])
            assert np.linalg.norm(g - w) <= tol * np.linalg.norm(w), (layout, fam)


# one step of a call by the per-cell kernels (two launches or more) or by tiles
# (one), on either side of the lines; 8 steps of FP64 are 7 and 1
@pytest.mark.parametrize("prec,size,kw,cells", [
    (0, (316, 316), dict(use_pml=True, pml=8), False),
    (0, (320, 316), dict(use_pml=True, pml=8), True),
    (0, (320, 316), dict(), False),
    (1, (216, 216), "tfsf", False),
    (1, (217, 216), "tfsf", True),
    (2, (217, 216), "tfsf", True),
    (1, (420, 380), dict(use_pml=True, pml=8), False),
    (2, (420, 380), dict(use_pml=True, pml=8), False),
])
def test_single_steps_by_cells_or_by_tiles(fdtd, prec, size, kw, cells):
    if kw == "tfsf":
        kw = dict(use_pml=True, pml=8, use_tfsf=True, tfsf_left=14, tfsf_right=14, teta=90, phi=25, psi=90)
    rng = np.random.default_rng(8)
    fields = {c: np.zeros(size) for c in ("Ez", "Hx", "Hy")}
    for c, v in fields.items():
        v[1:-1, 1:-1] = rng.standard_normal([n - 2 for n in size]) / (1 if c[0] == "E" else 376.73)
    eps = {"eps": 1 + np.kron(rng.integers(0, 4, [n // 8 + 1 for n in size]), np.ones((8, 8)))[: size[0], : size[1]]}
    got = []
    for calls in ([1] * 9, [8, 1], [9]):
        with fdtd.Simulation(mode=2, size=size, precision=prec, materials=eps, **kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.t = 50
            sim.step(3)
            for n in calls:
                before = sim.launch_count()
                sim.step(n)
                if n == 1:
                    assert (sim.launch_count() - before > 1) == cells, sim.launch_count() - before
            got.append({c: sim.field(c) for c in fields})
    for g in got[1:]:
        for c in fields:
            if prec == 0:
                assert np.array_equal(g[c].view(np.int64), got[0][c].view(np.int64)), c
            else:   # (12 steps of FP32; FP16 storage rounds once per launch of tiles)
                assert np.linalg.norm(g[c] - got[0][c]) <= (1e-6 if prec == 1 else 5e-3) * np.linalg.norm(got[0][c]), c


# a step at t = 0 updates nothing but moves on a level: in FP64 the fields are
# then those of the step before the call's last, whatever its launches were
@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 9, 14, 15, 22])
@pytest.mark.parametrize("size", [(60, 45), (330, 340)])
@pytest.mark.parametrize("source", ["tfsf", "point"])
def test_fp64_step_at_zero_after_a_call(fdtd, n, size, source):
    kw, mats, fields = _setup(fdtd, 2, size, source, 11)
    out = []
    for calls in ([n], [1] * n):
        with fdtd.Simulation(materials=mats, precision=0, **kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.t = 20
            for k in calls:
                sim.step(k)
            sim.step(1, t_start=0)
            got = {c: sim.field(c) for c in fields}
            sim.step(5, t_start=40)
            got.update({c + "5": sim.field(c) for c in fields})
            out.append(got)
    for c in out[0]:
        assert np.array_equal(out[0][c].view(np.int64), out[1][c].view(np.int64)), c


@pytest.mark.parametrize("calls", [[1] * 30, [30], [8, 22]])
@pytest.mark.parametrize("mode", [2, 5])
def test_incident_grid_has_the_same_bits_in_every_form(fdtd, calls, mode):
    kw = dict(mode=mode, size=(64, 59), use_pml=True, pml=5, use_tfsf=True, tfsf_left=9, tfsf_right=9, teta=40, phi=25,
              psi=20)
    got = []
    for prec in (0, 1, 2):
        with fdtd.Simulation(precision=prec, **kw) as sim:
            for n in calls:
                sim.step(n)
            got.append((sim.incident("E"), sim.incident("H")))
    assert np.any(got[0][0] != 0)
    for g in got[1:]:
        assert np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1])
