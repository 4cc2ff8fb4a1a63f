"""Drude media that end at the PML in z, on both sides, for every remainder of
the PML width and of nz by the sweep's four-cell vectors: some of those vectors
hold Drude cells and PML cells together, and the sweep stores the PML's
auxiliaries where the Drude fix-up keeps X two steps back.  FP32 and FP16,
against the FP64 plain form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
OM, GA = np.float32(2 * np.pi * 30e9), np.float32(2 * np.pi * 1e9)


def _first_last(nz, pml):
    """First and last z the medium may take in the sweep: the cell below is flagged too (it averages the first), and
    the H cells under that one must be clear of the PML, which ends at cell pml - 1 and begins at nz - pml - 1."""
    return pml + 2, nz - pml - 2


def _errors(fdtd, shape, pml, prec, z_range, switch=None):
    om, ga = np.zeros(shape), np.zeros(shape)
    box = (slice(9, 13), slice(8, shape[1] - 9), slice(z_range[0], z_range[1] + 1))
    om[box], ga[box] = OM, GA
    mats = {"omegape": om, "omegapm": om, "gammae": ga, "gammam": ga}
    rng = np.random.default_rng(4)
    fields = {}
    for c in COMPS:
        fields[c] = np.zeros(shape)
        fields[c][1:-1, 1:-1, 1:-1] = rng.standard_normal(tuple(n - 2 for n in shape)) / (1 if c[0] == "E" else 376.73)
    out, kernel = {}, None
    for p in (0, prec):
        with fdtd.Simulation(materials=mats, precision=p, mode=3, size=shape, use_pml=True, pml=pml,
                             use_metamaterials=True) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            if switch:
                sim.t = 9
                for sweep in "1010":
                    switch(sweep)
                    sim.set_material("omegape", om)   # (an upload has the steps planned again)
                    sim.step(7)
            else:
                sim.step(21, t_start=9)
            out[p] = {c: sim.field(c)[box] for c in COMPS}   # (the medium itself, where the error is)
            kernel = sim.step_kernel
    assert kernel == ("fused3d_regblock" if switch else "sweep3d_tma"), kernel
    return [np.linalg.norm(np.concatenate([(out[prec][c] - out[0][c]).ravel() for c in COMPS if c[0] == fam])) /
            np.linalg.norm(np.concatenate([out[0][c].ravel() for c in COMPS if c[0] == fam])) for fam in "EH"]


# 1e-5: 21 FP32 steps; 2e-2: 21 steps rounded to 11 bits (the bounds of the
# media away from the PML).  A wrong X is off by the whole recurrence term.
@pytest.mark.parametrize("pml", [3, 4, 5, 6])
@pytest.mark.parametrize("nz", [40, 41, 42, 43])
@pytest.mark.parametrize("prec,tol", [(1, 1e-5), (2, 2e-2)])
def test_medium_that_ends_at_the_pml(fdtd, pml, nz, prec, tol):
    # (rows of one z tile with PML at both ends: the sweep's PML class)
    err = _errors(fdtd, (24, 30, nz), pml, prec, _first_last(nz, pml))
    assert max(err) <= tol, err


@pytest.mark.parametrize("pml", [3, 4, 5, 6])
@pytest.mark.parametrize("nz", [152, 153, 154, 155])
@pytest.mark.parametrize("prec,tol", [(1, 1e-5), (2, 2e-2)])
def test_medium_that_ends_at_the_pml_of_a_z_edge_tile(fdtd, monkeypatch, capfd, pml, nz, prec, tol):
    # two z tiles and short x chunks: items without x and y PML take the z-edge class
    monkeypatch.setenv("FDTDB_SWEEP_CHUNK", "4")
    monkeypatch.setenv("FDTDB_SWEEP_VERBOSE", "1")
    err = _errors(fdtd, (24, 30, nz), pml, prec, _first_last(nz, pml))
    classes = capfd.readouterr().err.split("items lean/z-edge/full/PML=")[1].split()[0].split("/")
    assert int(classes[1]) > 0, classes
    assert max(err) <= tol, err


@pytest.mark.parametrize("pml,nz", [(5, 40), (6, 43)])
def test_the_state_moves_between_the_kernels(fdtd, monkeypatch, pml, nz):
    err = _errors(fdtd, (24, 30, nz), pml, 1, _first_last(nz, pml), lambda v: monkeypatch.setenv("FDTDB_SWEEP", v))
    assert max(err) <= 1e-5, err
