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
