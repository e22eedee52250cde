"""FP64 near field at the edges of its tiles (groups of 8 targets, teams of warps, items of 128 targets, runs of 32 and
chunks of 512 sources).

All points lie in the eight mutually neighbouring leaves around (0.25, 0.25, 0.25) of a depth-2 tree, so the matvec is
the near field alone and equals the direct sum.  Bound: each term carries a few roundings and at most n of one sign add
up, so the error is below (n + 8) 2^-53 of the sum of the terms' magnitudes."""
import numpy as np
import pytest

import old_fmm_bem_b200 as ob

pytestmark = pytest.mark.gpu


def _direct(kernel, xt, xs, tn, sn, q, ref, excl):
    """FP64 sums, and the same sums of magnitudes: (4, ni) each (potential, gradient)."""
    d = (xt[:, :, None] - xs[:, None, :]).astype(np.float64) if ref else \
        xt.astype(np.float64)[:, :, None] - xs.astype(np.float64)[:, None, :]
    r2 = (d ** 2).sum(0) + (float(np.float32(1e-6)) if ref else 0.0)
    skip = (d == 0).all(0) & excl
    ri = np.where(skip, 0.0, 1.0 / np.sqrt(np.where(skip, 1.0, r2)))
    qc = q.astype(np.float64)[None] * (0.25 / (float(np.float32(np.pi)) if ref else np.pi))
    if kernel == ob.LAPLACE_G:
        t = [qc * ri] + [-qc * ri ** 3 * d[k] for k in range(3)]
        m = [abs(v) for v in t]
    else:
        n = (tn[:, :, None] if kernel == ob.LAPLACE_GNI else sn[:, None, :]).astype(np.float64)
        dot, mag = (d * n).sum(0), abs(d * n).sum(0)
        t = [qc * ri ** 3 * dot] + [qc * ri ** 3 * (n[k] - 3 * dot * ri ** 2 * d[k]) for k in range(3)]
        m = [abs(qc) * ri ** 3 * mag] + [abs(qc) * ri ** 3 * (abs(n[k]) + 3 * mag * ri ** 2 * abs(d[k])) for k in range(3)]
    return np.array([v.sum(1) for v in t]), np.array([v.sum(1) for v in m])


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI, ob.LAPLACE_GNJ])
@pytest.mark.parametrize("ref", [False, True])
@pytest.mark.parametrize("ni,nj", [(1, 1), (7, 31), (9, 33), (33, 513), (65, 100), (128, 4100), (129, 65), (1300, 2047)])
def test_near_field_equals_direct(kernel, ref, ni, nj):
    rng = np.random.default_rng(ni * 10007 + nj)
    # most points in the first leaf, so that it holds more than one item of 128 targets at the larger sizes
    xt = (rng.random((3, ni)) * np.where(rng.random(ni) < 0.7, 0.24, 0.49)).astype(np.float32)
    xs = (rng.random((3, nj)) * np.where(rng.random(nj) < 0.7, 0.24, 0.49)).astype(np.float32)
    k = min(ni, nj) // 2
    xs[:, :k] = xt[:, :k]  # coincident pairs
    tn, sn = rng.standard_normal((3, ni)).astype(np.float32), rng.standard_normal((3, nj)).astype(np.float32)
    q = rng.standard_normal(nj).astype(np.float32)
    with ob.Plan(kernel=kernel, p=4, lmax=2, precision=ob.FP64, semantics=ob.SEM_REFERENCE if ref else ob.SEM_ACCURATE,
                 exclude_self=not ref) as pl:
        pl.set_geometry(xt, xs, tn if kernel == ob.LAPLACE_GNI else None, sn if kernel == ob.LAPLACE_GNJ else None,
                        bbox=(0, 0, 0, 1))
        grad = np.zeros(3 * ni) if kernel == ob.LAPLACE_G or not ref else None
        pot, grad = pl.evaluate(q, np.zeros(ni), grad, f64=True)
    want, mag = _direct(kernel, xt, xs, tn, sn, q, ref, not ref)
    tol = (nj + 8) * 2.0 ** -53 * mag
    assert np.all(abs(pot - want[0]) <= tol[0])
    if grad is not None:
        assert np.all(abs(grad.reshape(3, -1) - want[1:]) <= tol[1:])


def test_included_coincident_pair_is_infinite():
    x = np.array([[0.1, 0.2], [0.1, 0.1], [0.1, 0.1]], np.float32)
    with ob.Plan(kernel=ob.LAPLACE_G, p=4, lmax=2, precision=ob.FP64, semantics=ob.SEM_ACCURATE) as pl:
        pl.set_geometry(x, x, bbox=(0, 0, 0, 1))
        pot, _ = pl.evaluate(np.ones(2, np.float32), f64=True)
    assert np.all(np.isposinf(pot))


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI, ob.LAPLACE_GNJ])
def test_any_coordinates(kernel):
    # no coordinates a caller can give meet the padding of the source lists: targets around 1e18, which FP32 holds to
    # 2^36.  Bounds as above
    rng = np.random.default_rng(2)
    x = (rng.random((3, 70)) * 1.9e18).astype(np.float32)
    x[:, 5] = 1e18
    s = x[:, 20:57].copy()
    tn, sn = rng.standard_normal((3, 70)).astype(np.float32), rng.standard_normal((3, 37)).astype(np.float32)
    q = rng.standard_normal(37).astype(np.float32)
    with ob.Plan(kernel=kernel, p=4, lmax=2, precision=ob.FP64, semantics=ob.SEM_ACCURATE, exclude_self=True) as pl:
        pl.set_geometry(x, s, tn if kernel == ob.LAPLACE_GNI else None, sn if kernel == ob.LAPLACE_GNJ else None,
                        bbox=(0, 0, 0, 4e18))
        pot, grad = pl.evaluate(q, np.zeros(70), np.zeros(210), f64=True)
    want, mag = _direct(kernel, x, s, tn, sn, q, False, True)
    tol = (37 + 8) * 2.0 ** -53 * mag
    assert np.all(abs(pot - want[0]) <= tol[0]) and np.all(abs(grad.reshape(3, -1) - want[1:]) <= tol[1:])
