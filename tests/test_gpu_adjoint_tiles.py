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


@pytest.mark.parametrize("every", [200, 100, 67, 30, 7, 1])
@pytest.mark.parametrize("whole", [False, True])
def test_memory_of_a_run(fdtd, every, whole):
    """Device memory of a backward run, against the run with single buffers: state 6 N, adjoint 9 N, checkpoints 6 N
    each, two segments' per-step data (K N values, and the K probe fields in FP64), im in both precisions, the
    gradient twice.  With a probe of a few cells, and one that covers the grid."""
    import torch

    size, steps = (1200, 1100), 200
    cells = size[0] * size[1]
    probe = ((1, 1), (size[0] - 1, size[1] - 1)) if whole else ((700, 600), (704, 603))
    npr = (probe[1][0] - probe[0][0]) * (probe[1][1] - probe[0][1])
    kw = dict(mode=2, size=size, use_pml=True, pml=8, teta=90, phi=0, psi=90, point_source=(500, 500, 0),
              point_source_mask=4, precision=1)
    segments = -(-steps // every)
    single = cells * (4 * (6 + 9 + 6 * segments + 2 * every + 1) + 8 * 3) + 16 * every * npr
    with fdtd.Simulation(**kw) as sim:
        sim.step(1)
        sim.sync()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info(0)[0]
        sim.backward(steps, every, *probe, 1)
        used = before - torch.cuda.mem_get_info(0)[0]
    assert used <= single + (8 << 20), (used / single)


@pytest.mark.parametrize("every", [44, 22, 21, 15, 7, 1])
def test_segments_agree_whatever_their_number(fdtd, every):
    """One segment, two (neither is stored as a checkpoint), three and more: the same gradient, bit for bit, from the
    same forward run, with a probe over several tiles."""
    kw, eps, _, _ = _grid((90, 111))
    with fdtd.Simulation(materials={"eps": eps}, precision=1, **kw) as sim:
        j, g = sim.backward(44, 1000, (20, 30), (70, 90), 0)
        j1, g1 = sim.backward(44, every, (20, 30), (70, 90), 0)
        assert sim.objective(44, (20, 30), (70, 90), 0) == j
    assert j > 0 and j1 == j and np.array_equal(g1, g)
