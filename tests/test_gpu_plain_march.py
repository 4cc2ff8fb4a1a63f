"""The FP64 plain form's 3-D half-steps by columns against the oracle, bit for
bit: sides around the column blocks and x chunks, both layouts, every material
form, with and without PML and TF/SF."""
import numpy as np
import pytest

from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


@pytest.fixture(autouse=True)
def _columns_at_every_size(monkeypatch):
    """The columns' edges are at small sizes, which take the per-cell kernel by default."""
    monkeypatch.setenv("FDTDB_MARCH", "1")


def _maps(shape, seed):
    rng = np.random.default_rng(seed)
    blocks = rng.uniform(1.0, 4.0, tuple(n // 4 + 1 for n in shape))
    return np.kron(blocks, np.ones((4, 4, 4)))[: shape[0], : shape[1], : shape[2]]


# 3 x 3 x 3: one updated cell; 10 x 18 x 10: exactly one block of 128 columns;
# 11 x 18 x 11: just over one; 70 x 9 x 13: several x chunks of few columns
@pytest.mark.parametrize("shape", [(3, 3, 3), (10, 18, 10), (11, 18, 11), (70, 9, 13)])
@pytest.mark.parametrize("form", ["vacuum", "eps", "mu", "eps_mu"])
@pytest.mark.parametrize("pml", [0, 2])
def test_columns_match_oracle_bit_for_bit(fdtd, shape, form, pml):
    tfsf = min(shape) >= 9
    kw = dict(mode=3, size=shape, point_source=tuple(n // 2 for n in shape), point_source_mask=1 << 2)
    if pml and min(shape) > 4:
        kw.update(use_pml=True, pml=pml)
    if tfsf:
        kw.update(use_tfsf=True, tfsf_left=3, tfsf_right=3, teta=35, phi=50, psi=20)
    mats = {}
    if "eps" in form:
        mats["eps"] = _maps(shape, 1)
    if "mu" in form:
        mats["mu"] = _maps(shape, 2)
    o = Oracle(materials=mats or None, **kw)
    o.step(23)
    with fdtd.Simulation(materials=mats or None, **kw) as sim:
        sim.step(9)
        sim.step(14)
        for c in COMPS:
            got, want = sim.field(c), o.field(c)
            assert np.array_equal(got.view(np.int64), want.view(np.int64)), (c, np.max(np.abs(got - want)))
    o.close()


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("mu", [False, True])
def test_columns_match_cells_in_h_centered_grids(fdtd, mu, double):
    """H_CENTERED and double material precision have no oracle: a current
    source of zero amplitude (t = 0) takes the per-cell kernel for E and H of
    the same run, so two runs of one step from the same noise differ only in
    the kernel."""
    shape = (14, 13, 37)
    fine = tuple(2 * n for n in shape) if double else shape
    rng = np.random.default_rng(5)
    fields = {c: rng.standard_normal(shape) for c in COMPS}
    mats = {"eps": _maps(fine, 3)}
    if mu:
        mats["mu"] = _maps(fine, 4)
    for layout in (0, 1):
        out = []
        for mask in (0, 0x3f):
            kw = dict(mode=3, size=shape, use_pml=True, pml=3, use_tfsf=True, tfsf_left=4, tfsf_right=4, teta=35,
                      phi=50, psi=20, layout=layout, double_material_precision=double, current_source=(7, 6, 5),
                      current_source_mask=mask)
            with fdtd.Simulation(materials=mats, **kw) as sim:
                for c, v in fields.items():
                    sim.set_field(c, v)
                sim.step(1, t_start=1)
                out.append({c: sim.field(c) for c in COMPS})
        far = np.ones(shape, bool)
        far[5:9, 4:8, 3:7] = False   # (the current acts on its cell and the H cells around it)
        for c in COMPS:
            assert np.array_equal(out[0][c][far].view(np.int64), out[1][c][far].view(np.int64)), (layout, c)


# a material of -1 on a column's first plane: the coefficients must be formed
# from it (with PML every component but the last is formed anew by the x
# coefficients all the same)
@pytest.mark.parametrize("where", ["everywhere", "first planes", "a block"])
@pytest.mark.parametrize("pml", [0, 3])
@pytest.mark.parametrize("which", [("eps",), ("mu",), ("eps", "mu")])
def test_material_of_minus_one(fdtd, where, pml, which):
    shape = (20, 13, 14)
    mats = {}
    for name in which:
        m = np.full(shape, -1.0)
        if where == "first planes":
            m[6:] = 2.5
        elif where == "a block":
            m[:] = 1.5
            m[1:5, 4:9, 3:8] = -1.0
        mats[name] = m
    kw = dict(mode=3, size=shape, point_source=(10, 6, 7), point_source_mask=1 << 2)
    if pml:
        kw.update(use_pml=True, pml=pml)
    o = Oracle(materials=mats, **kw)
    o.step(12)
    with fdtd.Simulation(materials=mats, **kw) as sim:
        sim.step(12)
        for c in COMPS:
            got, want = sim.field(c), o.field(c)
            assert np.array_equal(got.view(np.int64), want.view(np.int64)), (c, np.max(np.abs(got - want)))
    o.close()


# 40000 cells: the default route on either side of the line, with its incident
# grid, against the other one
@pytest.mark.parametrize("shape", [(33, 34, 35), (33, 34, 36), (40, 40, 25)])
def test_columns_or_cells_by_size(fdtd, monkeypatch, shape):
    kw = dict(mode=3, size=shape, use_pml=True, pml=4, use_tfsf=True, tfsf_left=7, tfsf_right=7, teta=35, phi=50, psi=20)
    out, launches = [], []
    for march in (None, "0", "1"):
        monkeypatch.delenv("FDTDB_MARCH", raising=False)
        if march:
            monkeypatch.setenv("FDTDB_MARCH", march)
        with fdtd.Simulation(materials={"eps": _maps(shape, 1)}, **kw) as sim:
            sim.step(20)
            before = sim.launch_count()
            sim.step(5)
            launches.append(sim.launch_count() - before)
            out.append({c: sim.field(c) for c in COMPS})
    # (by cells the incident grid's two updates are launches of their own)
    assert launches[1] == 2 * launches[2] and launches[0] == launches[2 if np.prod(shape) >= 40000 else 1], launches
    for got in out[1:]:
        for c in COMPS:
            assert np.array_equal(got[c].view(np.int64), out[0][c].view(np.int64)), c
