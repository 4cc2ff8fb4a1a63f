"""FP16 storage: the TF/SF corrections after a single sweep step give the fields
of the same corrections inside the sweep, bit for bit (nothing is rounded twice),
on whole and on padded rows, with and without an eps map and a point source on
or beside the faces, and with a Drude medium in the box."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _run(fdtd, monkeypatch, post, n, prec=2, noise=True, mats=None, calls=(1, 9), **kw):
    monkeypatch.setenv("FDTDB_TB2", "0")
    monkeypatch.setenv("FDTDB_TFSF_POST", post)
    rng = np.random.default_rng(5)
    with fdtd.Simulation(mode=3, size=n, precision=prec, use_pml=True, pml=4, use_tfsf=True, teta=30, phi=40, psi=20,
                         materials=mats, **kw) as sim:
        if noise:
            for c in COMPS:
                v = np.zeros(n)
                v[1:-1, 1:-1, 1:-1] = rng.standard_normal([k - 2 for k in n]) / (1 if c[0] == "E" else 376.73)
                sim.set_field(c, v)
        sim.t = 100 if noise else 0
        for k in calls:
            sim.step(k)
        assert not prec or sim.step_kernel == "sweep3d_tma", sim.step_kernel
        return {c: sim.field(c) for c in COMPS}


# 7: the band is next to the PML of 4 cells; 1 cell between the faces
@pytest.mark.parametrize("n,left,right", [((36, 30, 40), 9, 9), ((33, 31, 37), 7, 8), ((40, 36, 150), (8, 9, 10), (9, 8, 7))])
@pytest.mark.parametrize("eps", [False, True])
@pytest.mark.parametrize("source", [None, (20, 15, 18), (9, 12, 20), (8, 9, 9)])
def test_corrections_after_the_step_keep_the_bits(fdtd, monkeypatch, n, left, right, eps, source):
    kw = dict(tfsf_left=left, tfsf_right=right)
    if source:
        kw.update(point_source=source, point_source_mask=0x3f)
    mats = None
    if eps:
        blocks = np.random.default_rng(3).integers(0, 12, [v // 5 + 1 for v in n]) / 4.0 + 1
        mats = {"eps": np.kron(blocks, np.ones((5, 5, 5)))[: n[0], : n[1], : n[2]]}
    got = [_run(fdtd, monkeypatch, post, n, mats=mats, **kw) for post in "10"]
    for c in COMPS:
        if n[2] <= 128:
            assert np.array_equal(got[0][c], got[1][c]), (c, np.max(np.abs(got[0][c] - got[1][c])))
        else:   # (two z tiles: PML cells of the z-edge class round in another order than those of the full class)
            assert np.linalg.norm(got[0][c] - got[1][c]) <= 3e-4 * np.linalg.norm(got[1][c]), c


@pytest.mark.parametrize("nz", [48, 45])
def test_wave_is_as_exact_as_with_corrections_inside(fdtd, monkeypatch, nz):
    n = (44, 40, nz)
    kw = dict(tfsf_left=10, tfsf_right=10, noise=False, calls=(25,))
    want = _run(fdtd, monkeypatch, "1", n, prec=0, **kw)
    got = [_run(fdtd, monkeypatch, post, n, **kw) for post in "10"]
    for c in COMPS:
        assert np.array_equal(got[0][c], got[1][c]), c
    for fam in "EH":
        g, w = (np.concatenate([f[c].ravel() for c in COMPS if c[0] == fam]) for f in (got[0], want))
        assert np.linalg.norm(g - w) <= 2e-2 * np.linalg.norm(w), fam


def test_drude_medium_in_the_box(fdtd, monkeypatch):
    n = (44, 40, 48)
    om = np.zeros(n)
    om[14:30, 13:28, 15:33] = np.float32(2 * np.pi * 30e9)
    mats = {"omegape": om, "gammae": om / 30}
    kw = dict(tfsf_left=9, tfsf_right=9, use_metamaterials=True, mats=mats, calls=(12,))
    got = _run(fdtd, monkeypatch, "1", n, **kw)
    want = _run(fdtd, monkeypatch, "1", n, prec=0, **kw)
    for fam in "EH":
        g, w = (np.concatenate([f[c].ravel() for c in COMPS if c[0] == fam]) for f in (got, want))
        assert np.linalg.norm(g - w) <= 2e-2 * np.linalg.norm(w), fam
