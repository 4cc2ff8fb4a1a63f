"""The adjoint's tiles at their edges: an own area of 18 cells
(32-cell tiles) or 50 (64-cell tiles) per side, grids of exactly one, one cell
more, ragged, and large enough for the larger tile; rounds of seven steps with
remainders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the last one is more than half the SMs' worth of small tiles
GRIDS = [(18, 18), (19, 37), (36, 19), (55, 18), (90, 111), (190, 205)]


def _grid(size):
    c = tuple(n // 2 for n in size)
    kw = dict(mode=2, size=size, use_pml=True, pml=4, teta=90, phi=0, psi=90, point_source=(c[0] - 3, c[1], 0),
              point_source_mask=4, point_source_kind=1, point_source_bandwidth=0.5)
    rng = np.random.default_rng(size[0] * 1000 + size[1])
    eps = rng.uniform(1.0, 4.0, size).astype(np.float32).astype(np.float64)
    return kw, eps, (c[0] + 1, c[1] - 2), (c[0] + 3, c[1] + 1)


@pytest.mark.parametrize("size", GRIDS)
def test_gradient_matches_central_differences(fdtd, size):
    kw, eps, lo, hi = _grid(size)
    steps = 44   # six rounds and a remainder of two

    def objective(e):
        with fdtd.Simulation(materials={"eps": e}, precision=0, **kw) as sim:   # (a 64-bit eps map)
            return sim.objective(steps, lo, hi, 0)

    with fdtd.Simulation(materials={"eps": eps}, precision=1, **kw) as sim:
        j, g = sim.backward(steps, 10, lo, hi, 0)       # segments of a round and a remainder of three
        j1, g1 = sim.backward(steps, 44, lo, hi, 0)
        j32, g32 = sim.backward(steps, 10, lo, hi, 1)
    assert j > 0 and j == j1 and np.array_equal(g, g1)
    # 44 steps in 32 bits: the bound of the FP32 adjoint's own test
    assert abs(j32 - j) <= 1e-4 * j
    assert np.linalg.norm(g32 - g) <= 1e-3 * np.linalg.norm(g)
    # second-order differences of 64-bit objectives: h^2 J'''/6 + 2^-53 J/h
    h = 1e-4
    order = np.argsort(-np.abs(g).ravel())
    for q in order[[0, 3, 17, 40]]:
        x, y = divmod(int(q), size[1])
        ep, em = eps.copy(), eps.copy()
        ep[x, y] += h
        em[x, y] -= h
        fd = (objective(ep) - objective(em)) / (2 * h)
        assert abs(fd - g[x, y]) <= 2e-6 * np.max(np.abs(g)), ((x, y), fd, g[x, y])
