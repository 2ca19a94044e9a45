"""GPU: the float distance-driven pair over the widths of z footprint its
kernel tells apart (under one voxel with merged neighbouring rows, across one
voxel within a column, one to two, wider), at partial row tiles, with rows
falling in z, rows leaving the grid, wide transverse footprints, and values
that are not finite -- against the double build.

Tolerance: the parity bar (rel-L2 1e-5, max-abs 1e-4 x max).  Positions round
to about 1e-6 voxel on these grids, a share to that over the footprint's
width, i.e. ~1e-6 of a result.
"""
import numpy as np
import pytest
import torch

from nefct_b200 import _lib, ops
from tests.test_gpu_siddon import assert_parity

pytestmark = pytest.mark.gpu

ANGLES = np.array([0.0, 0.4, np.pi / 4 + 1e-3, 1.3, 2.9, 4.4, 5.6], np.float32)
# rows, row pitch, column pitch (magnification 2), z offset, source-axis distance
CASES = [(1, 1.1, 1.1, 0.0, 70.0), (33, 0.5, 1.3, 0.0, 70.0), (64, 1.2, 1.2, 2.0, 70.0), (65, 1.2, 0.4, -9.0, 70.0),
         (41, -1.1, 1.1, 0.0, 70.0), (30, 1.6, 1.2, 0.0, 40.0), (30, 2.0, 2.4, 0.0, 70.0), (30, 2.9, 6.5, 1.0, 70.0),
         (20, 5.0, 1.2, 0.0, 70.0), (9, 13.0, 9.0, 0.0, 70.0)]


def _geom(rows, db, da, off, sad, kind="flat"):
    return ops.DDGeometry((26, 21, 19), ANGLES, sad, 2 * sad, 35, da if kind == "flat" else da / (2 * sad), rows, db, 0.2,
                          -0.3, kind, np.linspace(off - 0.5, off + 0.5, ANGLES.size).astype(np.float32))


@pytest.mark.parametrize("kind", ["flat", "cyl"])
@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}x{c[1]}-da{c[2]}" for c in CASES])
def test_footprints(cuda, case, kind):
    g = _geom(*case, kind)
    gen = torch.Generator(device=cuda).manual_seed(case[0])
    x = torch.rand(g.vol_shape, device=cuda, generator=gen)
    y = torch.rand(g.proj_shape, device=cuda, generator=gen)
    y[2, :, 5] = 0
    y[3, : case[0] // 2, 7:12] = 0
    for flags in (0, _lib.FDK_NO_WEIGHT):
        assert_parity(ops.dd_forward(x, g, flags).cpu().numpy(), ops.dd_forward(x.double(), g, flags).cpu().numpy())
        assert_parity(ops.dd_backward(y, g, flags).cpu().numpy(), ops.dd_backward(y.double(), g, flags).cpu().numpy())


@pytest.mark.parametrize("db", [1.2, 2.4, 5.0])
def test_values_that_are_not_finite_stay_in_their_footprints(cuda, db):
    g = _geom(40, db, 1.2, 0.0, 70.0)
    gen = torch.Generator(device=cuda).manual_seed(3)
    x = torch.rand(g.vol_shape, device=cuda, generator=gen)
    y = torch.rand(g.proj_shape, device=cuda, generator=gen)
    x[9, 11, 13] = float("inf")
    y[4, 21, 18] = float("nan")
    for f, v in ((ops.dd_forward, x), (ops.dd_backward, y)):
        out, ref = f(v, g), f(v.double(), g)
        fine = torch.isfinite(ref)
        assert 0 < int((~fine).sum()) < ref.numel() // 10
        assert torch.equal(torch.isfinite(out), fine)
        assert_parity(torch.where(fine, out, 0.0).cpu().numpy(), torch.where(fine, ref, 0.0).cpu().numpy())


def test_pairs_of_rows_in_a_tall_grid(cuda):
    """10^6 slices and footprints just under a voxel wide: neighbouring rows'
    positions, rounded at that height, can lie more than a voxel apart.  Pairing
    the rows the other way round (one more row in front, without a value) moves no
    contribution.  The rows' places are exact in float, so both calls have the same
    footprints."""
    nz, nb_, db = 1_000_000, 4096, 2.0

    def back(rows, y):
        # row i of the first call is row i + 1 of the second
        first = 800_000.0 - (rows - nb_) * db
        g = ops.DDGeometry((6, 2, nz), np.zeros(1, np.float32), 600.0, 1207.2, 6, 1.0, rows, db,
                           b_offset=first + rows * db / 2)
        return ops.dd_backward(y, g, _lib.FDK_NO_WEIGHT)

    y = torch.rand((1, nb_, 6), device=cuda, generator=torch.Generator(device=cuda).manual_seed(2))
    a = back(nb_, y)
    b = back(nb_ + 1, torch.cat([torch.zeros((1, 1, 6), device=cuda), y], 1))
    assert float((a != 0).float().sum()) > 1e4
    # sums of a few products each: a few roundings of 6e-8
    assert float((a - b).abs().max()) < 1e-6 * float(a.abs().max())
