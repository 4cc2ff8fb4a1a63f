"""FP32 / FP16-storage 3-D grids whose rows are no whole number of 16-byte
units: they store padded rows, so that the TMA kernels serve them.  Fields,
uploads, the energy and the DFT are checked against the FP64 plain form (its
rows are never padded)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMPS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
ETA0 = 376.730313461770655


def _family(got, ref, fam):
    g = np.concatenate([got[c].ravel() for c in COMPS if c[0] == fam])
    r = np.concatenate([ref[c].ravel() for c in COMPS if c[0] == fam])
    return np.linalg.norm(g - r) / np.linalg.norm(r)


# nz = 31: the last length that keeps its rows; 32, 56: whole units of both
# types; 127 .. 133: around one 128-cell tile; 33 .. 36, 63: every remainder
@pytest.mark.parametrize("nz", [31, 32, 33, 34, 35, 36, 56, 63, 127, 129, 133])
@pytest.mark.parametrize("prec,tol", [(1, 1e-5), (2, 2e-2)])
def test_padded_rows_match_fp64(fdtd, nz, prec, tol):
    shape = (40, 37, nz)
    rng = np.random.default_rng(nz)
    # noise resumed at t = 30, with values FP16 storage holds exactly
    fields = {c: np.zeros(shape) for c in COMPS}
    for c in COMPS:
        v = rng.standard_normal(tuple(n - 2 for n in shape)).astype(np.float16).astype(np.float64)
        fields[c][1:-1, 1:-1, 1:-1] = v / (1.0 if c[0] == "E" else ETA0)
    eps = 1.0 + np.kron(rng.uniform(0, 3, (7, 7, nz // 6 + 1)), np.ones((6, 6, 6)))[:40, :37, :nz].astype(np.float32)
    kw = dict(mode=3, size=shape, use_pml=True, pml=4, use_tfsf=True, tfsf_left=13, tfsf_right=13, teta=30, phi=45,
              psi=20)
    out, spectrum, energy = {}, {}, {}
    for p in (0, prec):
        with fdtd.Simulation(materials={"eps": eps}, precision=p, **kw) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
                if p == 1:
                    np.testing.assert_allclose(sim.field(c), v, rtol=1e-6, atol=0)
            sim.step(12, t_start=30)
            sim.dft_setup("Ey", 1, 17, [15e9, 9e9])
            sim.step(3)
            out[p] = {c: sim.field(c) for c in COMPS}
            spectrum[p], energy[p] = sim.dft(), sim.reduce()[0]
            if p:
                unit = 8 if p == 2 else 4
                want = "fused3d_regblock" if nz < 32 and nz % unit else "sweep3d_tma"
                assert sim.step_kernel == want, sim.step_kernel
    for fam in "EH":
        assert _family(out[prec], out[0], fam) <= tol, (nz, fam, _family(out[prec], out[0], fam))
    assert np.linalg.norm(spectrum[prec] - spectrum[0]) <= tol * np.linalg.norm(spectrum[0])
    assert abs(energy[prec] / energy[0] - 1) <= tol


# a mu map takes the per-cell kernels: rows of nz cells and padded ones, grids
# that four CTAs an SM hold at once (up to 151 552 updated cells on 148) and
# larger ones
@pytest.mark.parametrize("shape", [(18, 15, 31), (18, 15, 36), (18, 15, 37), (18, 15, 40), (18, 15, 63), (66, 39, 66),
                                   (66, 40, 66), (61, 62, 63)])
@pytest.mark.parametrize("prec,tol", [(1, 1e-5), (2, 2e-2)])
def test_per_cell_kernels_on_either_row(fdtd, shape, prec, tol):
    nz = shape[2]
    rng = np.random.default_rng(nz)
    fields = {c: np.zeros(shape) for c in COMPS}
    for c in COMPS:
        fields[c][1:-1, 1:-1, 1:-1] = rng.standard_normal(tuple(n - 2 for n in shape)) / (1 if c[0] == "E" else ETA0)
    maps = {m: 1 + np.kron(rng.uniform(0, 3, [n // 5 + 1 for n in shape]), np.ones((5, 5, 5))) for m in ("eps", "mu")}
    maps = {m: v[:shape[0], :shape[1], :nz] for m, v in maps.items()}
    maps = {m: v.astype(np.float32).astype(np.float64) for m, v in maps.items()}
    out = {}
    for p in (0, prec):
        with fdtd.Simulation(materials=maps, precision=p, mode=3, size=shape, use_pml=True, pml=3) as sim:
            for c, v in fields.items():
                sim.set_field(c, v)
            sim.step(12, t_start=30)
            out[p] = {c: sim.field(c) for c in COMPS}
            assert not p or sim.step_kernel == "per_cell", sim.step_kernel
    for fam in "EH":
        assert _family(out[prec], out[0], fam) <= tol, (nz, fam, _family(out[prec], out[0], fam))


# fields to the device and back: rows of nz cells below and above the line of
# the four-cell form (8 M cells; the last one not a multiple of four), padded rows
@pytest.mark.parametrize("shape", [(20, 21, 40), (200, 200, 200), (201, 199, 200), (250, 181, 177), (21, 20, 33), (251, 252, 129)])
@pytest.mark.parametrize("prec", [1, 2])
def test_fields_come_back_as_they_went(fdtd, shape, prec):
    import torch

    rng = np.random.default_rng(1)
    v = rng.integers(-1000, 1001, shape) / 8.0   # (values that 11 bits hold)
    with fdtd.Simulation(mode=3, size=shape, precision=prec) as sim:
        sim.set_field("Ey", v)
        assert np.array_equal(sim.field("Ey"), v)
        out = torch.empty(v.size + 1, dtype=torch.float64, device="cuda")
        sim.field_device("Ey", out.data_ptr() + 8)   # off the 16-byte boundary
        sim.sync()
        assert np.array_equal(out[1:].cpu().numpy().reshape(shape), v)
        assert not np.any(sim.field("Ex"))
