"""The batch's tiles at their edges: an own area of 18 cells (32-cell tiles) or
50 (64-cell tiles) per side; rounds of seven steps with remainders."""
import numpy as np
import pytest

from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 6, 7, 8, 30])
def test_batch_at_tile_edges(fdtd, steps):
    phys = dict(use_pml=True, pml=4, dx=0.0005, wavelength=0.02, courant=0.5, teta=90, phi=0, psi=90,
                point_source_mask=4, point_source_kind=1, point_source_bandwidth=0.5)
    sizes = [(18, 18), (19, 50), (50, 50), (51, 51), (100, 37), (17, 101)]
    eps = [np.random.default_rng(i).uniform(1, 4, s).astype(np.float32).astype(np.float64)
           for i, s in enumerate(sizes)]
    with fdtd.Batch(sizes, **phys) as b:
        for i, e in enumerate(eps):
            b.set_eps(i, e)
        b.step(steps)
        b.sync()
        for i, (s, e) in enumerate(zip(sizes, eps)):
            o = Oracle(mode=2, size=s, point_source=(s[0] // 2, s[1] // 2), materials={"eps": e}, **phys)
            o.step(steps)
            for fam in (("Ez",), ("Hx", "Hy")):
                got = np.concatenate([b.field(i, c).ravel() for c in fam])
                want = np.concatenate([np.asarray(o.field(c)).ravel() for c in fam])
                # the bound of the 60-step comparison of the other batch tests
                assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want), (s, fam)
            o.close()


# calls of up to three steps go by cells, longer ones by tiles; 33, 34 columns
# and 34, 35 rows: a patch filled (31 x 32 cells) and one more
@pytest.mark.parametrize("pml", [0, 4])
@pytest.mark.parametrize("calls", [[1] * 14, [2, 3, 1, 8], [7, 1, 3, 3], [3, 4, 7]])
def test_short_calls_match_long_ones(fdtd, pml, calls):
    sizes = [(34, 33), (35, 34), (34, 65), (3, 3), (67, 95), (40, 1500)]
    if pml:
        sizes[3] = (12, 11)
    kw = dict(use_pml=bool(pml), pml=pml, dx=0.0005, wavelength=0.02, courant=0.5, teta=90, phi=0, psi=90,
              point_source_mask=1 << 2)
    rng = np.random.default_rng(6)
    maps = [1 + np.kron(rng.integers(0, 6, [v // 4 + 1 for v in s]), np.ones((4, 4)))[: s[0], : s[1]] for s in sizes]
    out = []
    for steps in (calls, [14]):
        with fdtd.Batch(sizes, **kw) as b:
            for i, m in enumerate(maps):
                b.set_eps(i, m)
            for n in steps:
                b.step(n)
            b.sync()
            out.append([{c: b.field(i, c) for c in ("Ez", "Hx", "Hy")} for i in range(len(sizes))])
    for i, (got, want) in enumerate(zip(*out)):
        for c in want:
            # (the same operations in the same order, contracted by the compiler in two kernels)
            assert np.linalg.norm(got[c] - want[c]) <= 1e-6 * np.linalg.norm(want[c]), (i, c)
        assert np.any(want["Ez"] != 0), i


def test_tuning_over_few_steps_times_the_tiles(fdtd):
    """tune () measures the tile shapes whatever the number of steps, and leaves the fields at 0."""
    kw = dict(use_pml=True, pml=4, dx=0.0005, wavelength=0.02, courant=0.5, teta=90, phi=0, psi=90, point_source_mask=4)
    out = []
    for tuned in (None, 1, 3, 8):
        with fdtd.Batch([(120, 90), (50, 61)], **kw) as b:
            if tuned:
                assert b.tune(tuned)[0] in (32, 64)
            b.step(20)
            out.append([b.field(i, "Ez") for i in range(2)])
    for got in out[1:]:
        for g, w in zip(got, out[0]):
            assert np.any(w != 0) and np.linalg.norm(g - w) <= 1e-6 * np.linalg.norm(w)
