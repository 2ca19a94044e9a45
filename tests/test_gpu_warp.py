"""GPU parity of the cpp/deform warp and its derivatives."""
import numpy as np
import pytest
import torch

import nefct_b200 as nb
from nefct_b200 import ops
from tests.test_gpu_siddon import assert_parity

pytestmark = pytest.mark.gpu


def test_warp_vs_reference_fixture(cuda, golden):
    t = [torch.from_numpy(golden[k]).to(cuda) for k in ("deform/img", "deform/mx", "deform/my", "deform/mz")]
    out = ops.warp_forward(*t).cpu().numpy()
    assert_parity(out, golden["deform/out"], rel=1e-6, mabs=1e-6)
    # the op-level mirror of Deform(image, mx, my, mz, grid)
    out2 = nb.cc.deform.deform(*t, [22, 20, 18]).cpu().numpy()
    np.testing.assert_array_equal(out, out2)


def _field(shape, amp, seed, dev, dtype):
    g = torch.Generator(device=dev).manual_seed(seed)
    return [(torch.rand(shape, dtype=dtype, device=dev, generator=g) * 2 - 1) * amp for _ in range(3)]


def test_warp_adjoint_identity_f64(cuda):
    shape = (20, 22, 24)
    m = _field(shape, 3.0, 1, cuda, torch.float64)
    g = torch.Generator(device=cuda).manual_seed(2)
    x = torch.randn(shape, dtype=torch.float64, device=cuda, generator=g)
    y = torch.randn(shape, dtype=torch.float64, device=cuda, generator=g)
    lhs = float((ops.warp_forward(x, *m) * y).sum())
    rhs = float((x * ops.warp_adjoint(y, *m)).sum())
    assert abs(lhs - rhs) <= 1e-12 * abs(lhs)


def test_warp_dvf_gradient_finite_difference_f64(cuda):
    shape = (16, 18, 20)
    m = _field(shape, 2.5, 3, cuda, torch.float64)
    g = torch.Generator(device=cuda).manual_seed(4)
    img = torch.rand(shape, dtype=torch.float64, device=cuda, generator=g)
    w = torch.randn(shape, dtype=torch.float64, device=cuda, generator=g)
    d = [torch.randn(shape, dtype=torch.float64, device=cuda, generator=g) for _ in range(3)]
    gx, gy, gz = ops.warp_grad_dvf(img, *m, w)
    an = float((gx * d[0] + gy * d[1] + gz * d[2]).sum())
    h = 1e-7
    fp = float((ops.warp_forward(img, *[a + h * b for a, b in zip(m, d)]) * w).sum())
    fm = float((ops.warp_forward(img, *[a - h * b for a, b in zip(m, d)]) * w).sum())
    fd = (fp - fm) / (2 * h)
    assert abs(fd - an) <= 1e-5 * abs(an)


def test_warp_then_project_autograd(cuda):
    """Gradients w.r.t. image and displacement field through warp -> project,
    checked by central differences in FP64."""
    shape = (24, 24, 24)
    geom = nb.ConeBeam((24, 24, 24), np.linspace(0, 2 * np.pi, 24, endpoint=False), 100.0, 200.0, 40, 1.5, 32, 1.5)
    gen = torch.Generator(device=cuda).manual_seed(6)
    img = torch.rand(shape, dtype=torch.float64, device=cuda, generator=gen).requires_grad_()
    m = [t.requires_grad_() for t in _field(shape, 2.0, 7, cuda, torch.float64)]
    b = torch.rand(geom.sino_shape, dtype=torch.float64, device=cuda, generator=gen)
    loss = ((nb.project(nb.warp(img, *m), geom) - b) ** 2).sum()
    loss.backward()
    di = torch.randn(shape, dtype=torch.float64, device=cuda, generator=gen)
    dm = [torch.randn(shape, dtype=torch.float64, device=cuda, generator=gen) for _ in range(3)]
    an = float((img.grad * di).sum() + sum((t.grad * dd).sum() for t, dd in zip(m, dm)))
    h = 1e-6

    def f(s):
        with torch.no_grad():
            w = ops.warp_forward(img + s * di, *[t + s * dd for t, dd in zip(m, dm)])
            return float(((ops.cb_forward(w, geom) - b) ** 2).sum())

    fd = (f(h) - f(-h)) / (2 * h)
    assert abs(fd - an) <= 1e-5 * abs(an)


def test_warp_invert_vs_oracle(cuda, oracle_lib):
    """A smooth field (|grad m| < 1, so the fixed point is contractive and
    FP32 rounding differences do not grow over the iterations)."""
    rng = np.random.default_rng(12)
    shape = (18, 20, 22)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape], indexing="ij")
    m = []
    for _ in range(3):
        a, ph = rng.uniform(0.8, 1.6), rng.uniform(0, 2 * np.pi, 3)
        m.append((a * np.sin(2 * np.pi * x / 22 + ph[0]) * np.cos(2 * np.pi * y / 20 + ph[1])
                  + 0.5 * a * np.sin(2 * np.pi * z / 18 + ph[2])).astype(np.float32))
    out = [t.cpu().numpy() for t in ops.warp_invert(*[torch.from_numpy(a).to(cuda) for a in m], iters=30)]
    ref = oracle_lib.warp_invert(*m, iters=30)
    for o, r in zip(out, ref):
        assert_parity(o, r, rel=1e-5, mabs=1e-4)


@pytest.mark.skipif("not __import__('oracle').have_ref_tex()")
@pytest.mark.parametrize("case", ["small", "motion"])
def test_warp_invert_vs_reference_texture_kernel(cuda, oracle_lib, case):
    """nefct_warp_invert against the reference's own DeformInvertKernel
    (deform_tex.cu.cc:78-99, run on this GPU through its texture units).
    Both iterate the same 30 Gauss-Seidel passes from 0 with clamp-to-edge
    trilinear sampling at the same points; the texture unit keeps 8
    fractional bits of each interpolation weight, this library samples in
    FP32.  A weight quantised by <= 2^-8 moves a sample by <= 2^-8 x the
    largest difference of neighbouring field values (here <= 0.6 voxel, so
    <= 0.0025 voxel), and the contraction (|grad m| <= 0.6) amplifies it by
    <= 1 / (1 - 0.6): the two inverses may differ by up to ~0.006 voxel
    (measured on B200: at most 5.7e-3 voxel, 5.2e-4 on average).  The bound
    asserted is 0.015 voxel at any voxel and 0.002 voxel on average; the
    same field shifted by one voxel moves the inverse by 0.8-0.9 voxel."""
    rng = np.random.default_rng(31 if case == "small" else 32)
    shape = (18, 20, 22) if case == "small" else (40, 48, 56)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape], indexing="ij")
    amp, lam = (1.6, 22.0) if case == "small" else (5.0, 56.0)
    m = []
    for _ in range(3):
        a, ph = rng.uniform(0.5, 1.0) * amp, rng.uniform(0, 2 * np.pi, 3)
        m.append((a * np.sin(2 * np.pi * x / lam + ph[0]) * np.cos(2 * np.pi * y / lam + ph[1])
                  + 0.5 * a * np.sin(2 * np.pi * z / lam + ph[2])).astype(np.float32))
    dm = [torch.from_numpy(a).to(cuda) for a in m]
    ours = ops.warp_invert(*dm, iters=30)
    ref = oracle_lib.ref_tex_invert(*dm)
    torch.cuda.synchronize()
    for o, r, f in zip(ours, ref, dm):
        d = (o - r).abs()
        assert float(r.abs().max()) > 0.3 * float(f.abs().max())       # a real inverse, not zeros
        assert float(d.max()) <= 0.015, float(d.max())
        assert float(d.mean()) <= 0.002, float(d.mean())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["zero", "smooth", "rough", "steps"])
@pytest.mark.parametrize("shape", [(3, 5, 4), (4, 8, 32), (5, 9, 33), (18, 7, 70)])
def test_warp_and_derivatives_share_corners(cuda, shape, kind, dtype):
    """The warp, its adjoint and its field gradient against sums over the eight
    corners in double precision, where neighbouring samples share corners
    (zero, smooth), do not (rough) and do so here and there (steps), for
    partial z groups and row tails; zeros in the cotangent take no part.

    Tolerance: a float32 result is a sum of rounded products of up to a few
    dozen terms, 2e-6 of the largest."""
    rng = np.random.default_rng(shape[0])
    nz, ny, nx = shape
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    if kind == "rough":
        m = [rng.uniform(-2.5, 2.5, shape) for _ in range(3)]
    elif kind == "steps":
        m = [rng.integers(-1, 2, shape) * (rng.random(shape) < 0.3) + 0.25 for _ in range(3)]
    else:
        amp = 0.0 if kind == "zero" else 1.3
        m = [amp * np.sin(0.21 * x + 0.17 * y + 0.4 * z + i) for i in range(3)]
    m = [a.astype(dtype) for a in m]
    img, g = rng.random(shape).astype(dtype), rng.standard_normal(shape).astype(dtype)
    g[rng.random(shape) < 0.1] = 0
    p = [(c.astype(dtype) + a) for c, a in zip((x, y, z), m)]
    f = [np.floor(a) for a in p]
    ok = np.ones(shape, bool)
    for a, n in zip(f, (nx, ny, nz)):
        ok &= (a > 0) & (a + 1 < n)
    w = [(a - b).astype(np.float64)[ok] for a, b in zip(p, f)]
    i = [a.astype(int)[ok] for a in f]
    out, adj = np.zeros(shape), np.zeros(shape)
    grad = [np.zeros(shape) for _ in range(3)]
    g64, acc, dacc = g.astype(np.float64)[ok], np.zeros(ok.sum()), [np.zeros(ok.sum()) for _ in range(3)]
    for c in range(8):
        b = [c & 1, c >> 1 & 1, c >> 2]
        at = (i[2] + b[2], i[1] + b[1], i[0] + b[0])
        part = [u if s else 1 - u for u, s in zip(w, b)]
        v = img[at].astype(np.float64)
        acc += v * part[0] * part[1] * part[2]
        np.add.at(adj, at, g64 * part[0] * part[1] * part[2])
        for k in range(3):
            o = [part[j] for j in range(3) if j != k]
            dacc[k] += (1 if b[k] else -1) * v * o[0] * o[1]
    out[ok] = acc
    for k in range(3):
        grad[k][ok] = dacc[k] * g64
    t = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (img, *m, g)]
    tol = 2e-6 if dtype == np.float32 else 1e-13
    for got, ref in ((ops.warp_forward(*t[:4]), out), (ops.warp_adjoint(t[4], *t[1:4]), adj),
                     *zip(ops.warp_grad_dvf(*t), grad)):
        np.testing.assert_allclose(got.cpu().numpy(), ref, rtol=0, atol=tol * max(np.abs(ref).max(), 1.0))
