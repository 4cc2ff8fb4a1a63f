"""The batch read-out goes through a bounded staging buffer in pieces of rows:
instances of several pieces, and one of more than 2^31 cells."""
import numpy as np
import psutil
import pytest
import torch

pytestmark = pytest.mark.gpu

PHYS = dict(dx=0.0005, wavelength=0.02, courant=0.5, teta=90, phi=0, psi=90, point_source_mask=1 << 2,
            point_source_kind=1, point_source_bandwidth=0.5)


def _middle(field, reach):
    c = [n // 2 for n in field.shape]
    return field[c[0] - reach:c[0] + reach + 1, c[1] - reach:c[1] + reach + 1]


# 2^23 cells a piece: 2896 x 2897 fits in one, 2900 x 2901 ends on a short
# second one, 9 x 2^20 takes rows that are no group of four
@pytest.mark.parametrize("size", [(2896, 2897), (2900, 2901), (9, 1 << 20)])
def test_pieces_of_an_instance(fdtd, size):
    kw = dict(use_pml=min(size) > 20, pml=8, **PHYS)
    fields = {}
    with fdtd.Batch([(60, 50), size], **kw) as b:
        b.step(30)
        for i in (1, 0):
            fields[i] = {c: b.field(i, c) for c in ("Ez", "Hx", "Hy")}
    for i, n in enumerate([(60, 50), size]):
        with fdtd.Simulation(mode=2, size=n, precision=fdtd.PREC_FP32, point_source=tuple(v // 2 for v in n), **kw) as s:
            s.step(30)
            for c, v in fields[i].items():
                assert np.linalg.norm(v - s.field(c)) <= 1e-5 * np.linalg.norm(v) and np.any(v != 0), (i, c)


def test_instance_of_more_cells_than_an_int_holds(fdtd):
    size = (2050, 1 << 20)
    cells = size[0] * size[1]
    assert cells > 2 ** 31
    if torch.cuda.mem_get_info()[0] < 30 * cells or psutil.virtual_memory().available < 24 * cells:
        pytest.skip("needs 65 GB of device and 52 GB of host memory")
    got = {}
    for name, n in (("small", (101, 101)), ("large", size)):
        with fdtd.Batch([n], **PHYS) as b:
            b.step(30)
            # the wave has not reached the small grid's faces: the same cells around the source
            got[name] = {c: _middle(b.field(0, c), 40).copy() for c in ("Ez", "Hy")}
    for c in ("Ez", "Hy"):
        assert np.any(got["small"][c] != 0)
        assert np.array_equal(got["small"][c], got["large"][c]), c
