"""GPU: the column-warp kernels at the edges of their row tiles and dispatch
rules -- row counts around the tiles of one, two and three rows per lane, row
pitches on both sides of the rule for merged reductions (and pairs that drift
more than a voxel apart inside it), rows falling in z, warps with rising and
falling rays, cone angles beyond 45 degrees, voxels that are not cubic,
rounding rules, infinities -- against the CPU restatement, and against the
thread walk, whose forward has the same bits.

Tolerance: the parity bar of the other tests (rel-L2 1e-5, max-abs 1e-4 x max).
The walk's z positions differ from the restatement's by at most two roundings
of about 1e-6 voxel on these grids, i.e. ~1e-6 of a result.
"""
import numpy as np
import pytest
import torch

import nefct_b200 as nb
from nefct_b200 import _lib, autotune, ops
from tests.test_gpu_siddon import assert_parity

pytestmark = pytest.mark.gpu

ANGLES = np.array([0.1, 0.7, np.pi / 2, 2.2, 3.6, 5.3], np.float32)

# rows; row pitch (detector, magnification 2); z voxel; z offset of the views
CASES = [
    (1, 1.2, 1.0, 0.0), (31, 1.2, 1.0, 0.0), (32, 1.0, 1.0, 0.4), (33, 1.2, 1.0, 0.0), (63, 0.6, 1.0, 0.0),
    (64, 1.2, 1.0, -6.0), (65, 1.2, 1.0, 6.0), (96, 0.7, 1.0, 0.0), (97, 0.7, 1.0, 0.0), (129, 0.4, 1.0, 3.0),
    (45, -1.1, 1.0, 0.0),                   # rows falling in z
    (40, 1.75, 1.0, 0.0),                   # pairs under the rule at the axis, over a voxel apart behind it
    (40, 1.9, 1.0, 0.0), (40, 3.1, 1.0, 0.0),          # single rows
    (50, 1.2, 0.7, 0.0), (50, 1.2, 1.6, 1.0),          # voxels that are not cubic
    # three and four rows per lane (thick slices), full and partial groups, rows
    # falling in z, and groups that drift over a voxel
    (77, 0.7, 1.0, 0.0), (96, 0.7, 1.0, 2.0), (70, -0.7, 1.0, -3.0), (127, 0.5, 1.0, 0.0), (128, 0.45, 1.0, 5.0),
    (101, -0.5, 1.0, 0.0), (90, 1.3, 2.5, 0.0), (91, 0.88, 1.0, 0.0),
    # last rows in a launch of their own: three and four rows per lane, then one
    # and three
    (193, 0.4, 1.0, 2.0),
]


def _geom(rows, pitch, vz, off, src_iso=70.0):
    shape = (26, 22, 24)
    return nb.ConeBeam(shape, ANGLES, src_iso, 2 * src_iso, 37, 1.5, rows, pitch, size=(26.0, 24.2, 24.0 * vz),
                       center=(0.3, -0.2, 0.1), z_offsets=np.linspace(off - 0.5, off + 0.5, ANGLES.size))


def _oracle(oracle_lib, g, vol, y, flags):
    og = oracle_lib.grid(g.shape, g.center, g.size)
    args = (g.angles, g.src_iso, g.src_det, g.na, g.da, 0.5, g.nb, g.db, 0.5)
    of = (0 if flags & _lib.TIE_GT else oracle_lib.TIE_GE) | (0 if flags & _lib.NO_INV_L2 else oracle_lib.INV_L2)
    of |= oracle_lib.SKIP_SHORT if flags & _lib.SKIP_SHORT else 0
    fwd = oracle_lib.cb_forward(og, vol, *args, off=g.z_offsets, flags=of)[0]
    return fwd, oracle_lib.cb_backward(og, y, *args, off=g.z_offsets, flags=of)


def _both(g, vol, y, flags, walk):
    saved = autotune.current()
    try:
        autotune.apply(saved["rows"], saved["order"], walk)
        return ops.cb_forward(vol, g, flags), ops.cb_backward(y, g, flags)
    finally:
        autotune.apply(saved["rows"], saved["order"], saved["walk"])


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}x{c[1]}-dz{c[2]}-off{c[3]}" for c in CASES])
def test_row_tiles_and_dispatch(cuda, oracle_lib, case, flags):
    g = _geom(*case)
    rng = np.random.default_rng(case[0])
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    y[1, : case[0] // 3] = 0                       # rays that take no part
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, flags)
    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    f, b = _both(g, v, s, flags, 3)
    assert_parity(f.cpu().numpy(), ref_f)
    assert_parity(b.cpu().numpy(), ref_b)
    ft, bt = _both(g, v, s, flags, 0)
    assert torch.equal(f, ft)
    assert_parity(b.cpu().numpy(), bt.cpu().numpy(), rel=1e-6, mabs=1e-5)
    det = [ops.cb_backward(s, g, flags | _lib.DETERMINISTIC) for _ in range(2)]
    assert torch.equal(det[0], det[1])
    assert_parity(det[0].cpu().numpy(), b.cpu().numpy(), rel=1e-6, mabs=1e-5)


def test_deterministic_flag_leaves_the_forward_alone(cuda):
    g = _geom(65, 1.2, 1.0, 0.0)
    vol = torch.rand(g.vol_shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(1))
    assert torch.equal(ops.cb_forward(vol, g, _lib.DETERMINISTIC), ops.cb_forward(vol, g, 0))


@pytest.mark.parametrize("pitch", [1.2, 3.0], ids=["pairs", "single-rows"])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_values_that_are_not_finite_stay_on_their_rays(cuda, oracle_lib, value, pitch):
    """A voxel that is not finite reaches the rays that pass it and no other;
    a sinogram value that is not finite the voxels on its ray."""
    g = _geom(45, pitch, 1.0, 0.0)
    rng = np.random.default_rng(7)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    vol[11, 9, 14] = value
    y[2, 21, 17] = value
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, 0)
    f, b = (t.cpu().numpy() for t in _both(g, torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda), 0, 3))
    for out, ref in ((f, ref_f), (b, ref_b)):
        fine = np.isfinite(ref)
        assert 0 < (~fine).sum() < ref.size // 10
        np.testing.assert_array_equal(np.isfinite(out), fine)
        np.testing.assert_array_equal(np.isnan(out), np.isnan(ref))
        assert_parity(np.where(fine, out, 0), np.where(fine, ref, 0))


def _thread_walk(g, vol, y, flags):
    """The thread walk with and without its y-fastest copy."""
    return _both(g, vol, y, flags, 0), _both(g, vol, y, flags | _lib.NO_TRANSPOSE, 3)


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("ratio", [0.91, 0.5, 0.25])
def test_rows_thinner_than_columns(cuda, oracle_lib, ratio, flags):
    """Grids whose y pitch is below the x pitch: a slab of an x-driven ray moves
    over a voxel in y, so its high column is not the one above its low column."""
    g = nb.ConeBeam((26, 22, 24), ANGLES, 70.0, 140.0, 37, 1.5, 65, 1.2, size=(26.0, 22.0 * ratio, 24.0),
                    center=(0.3, -0.2, 0.1), z_offsets=np.linspace(-0.5, 0.5, ANGLES.size))
    rng = np.random.default_rng(11)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, flags)
    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    f, b = _both(g, v, s, flags, 3)
    assert_parity(f.cpu().numpy(), ref_f)
    assert_parity(b.cpu().numpy(), ref_b)
    for ft, bt in _thread_walk(g, v, s, flags):
        assert torch.equal(f, ft)
        assert_parity(bt.cpu().numpy(), ref_b)
    fixed = [ops.cb_backward(s, g, flags | _lib.DETERMINISTIC | extra) for extra in (0, _lib.NO_TRANSPOSE)]
    assert torch.equal(*fixed)
    assert_parity(fixed[0].cpu().numpy(), ref_b)


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("rows", [20, 33, 70])
def test_two_slices_and_lanes_without_a_ray(cuda, oracle_lib, rows, flags):
    """nz = 2, rays that stay in the lower slice (slabs without range checks) and
    warps with lanes past the last row, which walk row 0."""
    g = nb.ConeBeam((26, 22, 2), ANGLES, 70.0, 140.0, 37, 1.5, rows, 0.02, size=(26.0, 22.0, 8.0),
                    center=(0.3, -0.2, 2.0), z_offsets=np.linspace(-0.1, 0.1, ANGLES.size))
    rng = np.random.default_rng(rows)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, flags)
    f, b = _both(g, torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda), flags, 3)
    assert_parity(f.cpu().numpy(), ref_f)
    assert_parity(b.cpu().numpy(), ref_b)


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("shape,angle", [((65600, 3, 2), np.pi / 2), ((3, 65600, 2), 0.0)], ids=["wide", "deep"])
def test_grids_wider_than_65536(cuda, oracle_lib, shape, angle, flags):
    """Rays that pass the far end of an axis of 65600 voxels, across it (the
    thread walk: column warps take at most 65535)."""
    ang = np.array([angle, angle + 5e-4, angle + np.pi, angle + np.pi + 5e-4], np.float32)
    g = nb.ConeBeam(shape, ang, 1e5, 2e5, 40, 10.0, 3, 0.4, a_shift=6560.0)
    og = oracle_lib.grid(g.shape, g.center, g.size)
    args = (g.angles, g.src_iso, g.src_det, g.na, g.da, g.a_shift, g.nb, g.db, g.b_shift)
    of = oracle_lib.CB_BP if flags else oracle_lib.CB_FWD
    rng = np.random.default_rng(2)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    ref_f = oracle_lib.cb_forward(og, vol, *args, flags=of)[0]
    ref_b = oracle_lib.cb_backward(og, y, *args, flags=of)
    assert 0.3 < (ref_f != 0).mean() < 0.9             # rays on both sides of the end
    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    for extra in (0, _lib.NO_TRANSPOSE):
        assert_parity(ops.cb_forward(v, g, flags | extra).cpu().numpy(), ref_f)
        assert_parity(ops.cb_backward(s, g, flags | extra).cpu().numpy(), ref_b)
        assert_parity(ops.cb_backward(s, g, flags | extra | _lib.DETERMINISTIC).cpu().numpy(), ref_b)


@pytest.mark.parametrize("walk", [0, 3], ids=["thread", "columns"])
@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT, _lib.NO_TRANSPOSE, _lib.DETERMINISTIC],
                         ids=["default", "reference-rounding", "direct", "deterministic"])
@pytest.mark.parametrize("rows", [1, 9])
@pytest.mark.parametrize("nz", [1, 2])
def test_nothing_outside_the_buffers_is_touched(cuda, nz, rows, flags, walk):
    """Volume, sinogram and workspace between NaN (inputs) or a mark (outputs):
    rays in the grid's last slice touch no voxel above it, whatever the rounding
    of their crossing ratios."""
    import ctypes as C
    g = nb.ConeBeam((200, 200, nz), np.linspace(0, 2 * np.pi, 90, endpoint=False), 300.0, 600.0, 310, 1.0, rows, 0.05,
                    z_offsets=np.full(90, 0.5 * nz - 0.5))
    pad, s, lib = 1 << 17, g.struct(), _lib.load()
    stream = torch.cuda.current_stream(cuda).cuda_stream
    wn = lib.nefct_cb_workspace_bytes(C.byref(s), flags)
    assert wn % 4 == 0

    def inside(n, fill):
        t = torch.full((n + 2 * pad,), fill, device=cuda)
        return t, t[pad:pad + n]

    vol_all, vol = inside(200 * 200 * nz, np.nan)
    ws_all, ws = inside(max(wn // 4, 1), np.nan)
    out_all, out = inside(90 * 310 * rows, 7.0)
    vol.copy_(torch.rand(vol.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(4)))
    back_all, back = inside(vol.numel(), 7.0)
    y = torch.rand(out.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(5))
    saved = autotune.current()
    try:
        autotune.apply(saved["rows"], saved["order"], walk)
        _lib.check(lib.nefct_cb_forward(C.byref(s), vol.data_ptr(), out.data_ptr(), flags, ws.data_ptr(), wn, stream))
        assert torch.isfinite(out).all() and out.any()
        ws_all.fill_(7.0)
        _lib.check(lib.nefct_cb_backward(C.byref(s), y.data_ptr(), back.data_ptr(), flags, ws.data_ptr(), wn, stream))
    finally:
        autotune.apply(saved["rows"], saved["order"], saved["walk"])
    assert torch.isfinite(back).all() and back.any()
    for t in (ws_all, out_all, back_all):
        assert (t[:pad] == 7.0).all() and (t[-pad:] == 7.0).all()


# rows, row pitch, z voxel, z offset: one to three rows per lane (forward), one to
# four that share reductions (transpose), rows falling in z, with rays that move
# over a voxel in z per slab
STEEP = [(24, 6.0, 1.0, 0.0), (120, 1.2, 1.0, 0.0), (120, -1.2, 1.0, 2.0), (129, 0.8, 0.7, 0.0), (161, 0.7, 0.8, 1.0),
         (200, 0.7, 0.5, -1.0)]


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("case", STEEP, ids=[f"{c[0]}x{c[1]}-dz{c[2]}-off{c[3]}" for c in STEEP])
def test_steep_rays(cuda, oracle_lib, case, flags):
    """Cone angles beyond 45 degrees (rays that cross a z plane in every slab and
    two in some), alone and in warps with others that are not steep; one value
    that is not finite in such a warp."""
    rows, pitch, vz, off = case
    g = nb.ConeBeam((20, 18, 60), ANGLES, 25.0, 50.0, 37, 1.0, rows, pitch, size=(20.0, 18.0, 60.0 * vz),
                    center=(0.3, -0.2, 0.1), z_offsets=np.linspace(off - 0.5, off + 0.5, ANGLES.size))
    # voxel rows per slab, at least, of each detector row's rays
    slope = np.abs((np.arange(rows) + 0.5) * pitch - rows * pitch / 2) / 50.0 / vz
    rng = np.random.default_rng(rows)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    y[2, rows // 2:, 5] = 0
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, flags)
    hit = slope[(ref_f != 0).any(axis=(0, 2))]
    assert hit.max() > 1.05 and hit.min() < 0.5
    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    f, bw = _both(g, v, s, flags, 3)
    assert_parity(f.cpu().numpy(), ref_f)
    assert_parity(bw.cpu().numpy(), ref_b)
    for ft, bt in _thread_walk(g, v, s, flags):
        assert torch.equal(f, ft)
        assert_parity(bt.cpu().numpy(), ref_b)
    fixed = [ops.cb_backward(s, g, flags | _lib.DETERMINISTIC | extra) for extra in (0, _lib.NO_TRANSPOSE)]
    assert torch.equal(*fixed)
    assert_parity(fixed[0].cpu().numpy(), ref_b)
    y[3, np.flatnonzero(ref_f[3, :, 18])[-1], 18] = np.inf
    ref_i = _oracle(oracle_lib, g, vol, y, flags)[1]
    out = ops.cb_backward(torch.from_numpy(y).to(cuda), g, flags).cpu().numpy()
    fine = np.isfinite(ref_i)
    assert 0 < (~fine).sum() < ref_i.size // 10
    np.testing.assert_array_equal(np.isfinite(out), fine)
    assert_parity(np.where(fine, out, 0), np.where(fine, ref_i, 0))


@pytest.mark.parametrize("nz,vz,off,rows,pitch", [(600, 0.1, 25.0, 65, 0.2), (300, 1.0, 120.3, 33, 0.3),
                                                  (120, 0.71, 35.0, 33, 0.4)])
def test_error_against_double_is_no_larger_than_the_reference_walks(cuda, oracle_lib, nz, vz, off, rows, pitch):
    """Nearly level rays far from row 0, whose shares divide the error of a z
    position by a small slope: the rel-L2 error against the double walk is at most
    1.1 times that of the reference's operations in float (0.2 to 0.8 times on a
    host build of the walk; positions held as row numbers: 1.5 to 1.8 times)."""
    g = nb.ConeBeam((26, 22, nz), ANGLES, 70.0, 140.0, 37, 1.5, rows, float(np.float32(pitch)),
                    size=tuple(float(np.float32(s)) for s in (26.0, 24.2, nz * vz)),
                    center=tuple(float(np.float32(c)) for c in (0.3, -0.2, 0.1)),
                    z_offsets=np.linspace(off - 0.05, off + 0.05, ANGLES.size, dtype=np.float32))
    og = oracle_lib.grid(g.shape, g.center, g.size)
    args = (g.angles, g.src_iso, g.src_det, g.na, g.da, 0.5, g.nb, g.db, 0.5)
    rng = np.random.default_rng(1)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    f64 = oracle_lib.cb_forward(og, vol, *args, off=g.z_offsets, f64=True)[0]
    b64 = oracle_lib.cb_backward(og, y, *args, off=g.z_offsets, flags=oracle_lib.CB_FWD, f64=True)
    f32 = oracle_lib.cb_forward(og, vol, *args, off=g.z_offsets)[0]
    b32 = oracle_lib.cb_backward(og, y, *args, off=g.z_offsets, flags=oracle_lib.CB_FWD)

    def err(a, ref):
        return np.linalg.norm(np.asarray(a, np.float64) - ref) / np.linalg.norm(ref)

    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    for walk in (3, 0):
        f, b = (t.cpu().numpy() for t in _both(g, v, s, 0, walk))
        assert err(f, f64) <= 1.1 * err(f32, f64), (err(f, f64), err(f32, f64))
        assert err(b, b64) <= 1.1 * err(b32, b64), (err(b, b64), err(b32, b64))


@pytest.mark.parametrize("flags", [0, _lib.TIE_GT], ids=["default", "reference-rounding"])
def test_pairs_of_rows_in_a_tall_grid(cuda, flags):
    """65535 slices and neighbouring rows just under a voxel apart, whose
    positions round by some thousandths of a voxel at that height: pairing the rows
    the other way round (one more row in front, without a value) moves no
    contribution.  The rows' places are exact in float in both calls."""
    nv, rows, db = 1000, 18, 113 / 64
    off = np.floor(np.random.default_rng(3).random(nv) * 64000) / 2 - 16000 + np.arange(nv) / 1024

    def back(nb_, y):
        g = nb.ConeBeam((3, 3, 65535), np.linspace(0, 2 * np.pi, nv, endpoint=False), 12.0, 24.0, 8, 0.5, nb_, db,
                        b_shift=0.5 + nb_ / 2 - (nb_ - rows) - rows / 2, z_offsets=off.astype(np.float32))
        return ops.cb_backward(y, g, flags)

    y = torch.rand((nv, rows, 8), device=cuda, generator=torch.Generator(device=cuda).manual_seed(2))
    a = back(rows, y)
    b = back(rows + 1, torch.cat([torch.zeros((nv, 1, 8), device=cuda), y], 1))
    assert int((a != 0).sum()) > 10000
    # sums of up to a few hundred terms in another order
    assert float((a - b).abs().max()) < 3e-6 * float(a.abs().max())


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("rows", [7, 8, 9])
def test_few_detector_rows(cuda, oracle_lib, rows, flags):
    """Both sides of the line below which the thread walk takes the rows, alone and
    in a batch plan (column warps at any number of rows)."""
    from nefct_b200.batch import BatchProjector
    g = _geom(rows, 1.2, 1.0, 1.0)
    rng = np.random.default_rng(rows)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, flags)
    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    f, b = _both(g, v, s, flags, 3)
    assert_parity(f.cpu().numpy(), ref_f)
    assert_parity(b.cpu().numpy(), ref_b)
    plan = BatchProjector([g], [v], grads=[s], flags=flags, strategy="persistent")
    plan.step()
    assert torch.equal(plan.sinos[0], f)
    assert_parity(plan.backs[0].cpu().numpy(), ref_b)
    fixed = [ops.cb_backward(s, g, flags | _lib.DETERMINISTIC | extra) for extra in (0, _lib.NO_TRANSPOSE)]
    assert torch.equal(*fixed)


@pytest.mark.parametrize("flags", [0, _lib.REF_BACKPROJECT], ids=["default", "reference-rounding"])
@pytest.mark.parametrize("bound", [0.97, 0.99, 1.3])
def test_both_sides_of_the_steep_line(cuda, oracle_lib, bound, flags):
    """Transposes are launched without the code for steep rays while sqrt(2) max |b|
    / src_det stays under 0.98 voxel rows per slab; views along the diagonals have
    rays that come close to that bound."""
    rows, vz = 58, 0.8
    pitch = bound * vz * 50.0 / np.sqrt(2.0) / (rows / 2 - 0.5)
    ang = np.array([np.pi / 4, 3 * np.pi / 4 + 0.01, 4.0, 5.49], np.float32)
    g = nb.ConeBeam((20, 18, 60), ang, 25.0, 50.0, 37, 0.7, rows, float(np.float32(pitch)), size=(20.0, 18.0, 60.0 * vz))
    rng = np.random.default_rng(4)
    vol = rng.random(g.vol_shape, dtype=np.float32)
    y = rng.random(g.sino_shape, dtype=np.float32)
    ref_f, ref_b = _oracle(oracle_lib, g, vol, y, flags)
    v, s = torch.from_numpy(vol).to(cuda), torch.from_numpy(y).to(cuda)
    f, b = _both(g, v, s, flags, 3)
    assert_parity(f.cpu().numpy(), ref_f)
    assert_parity(b.cpu().numpy(), ref_b)
    fixed = [ops.cb_backward(s, g, flags | _lib.DETERMINISTIC | extra) for extra in (0, _lib.NO_TRANSPOSE)]
    assert torch.equal(*fixed)
