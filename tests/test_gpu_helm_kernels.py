"""Helmholtz and Yukawa near field, P2M and L2P at the edges of their tiles (8-target groups, items of 128 targets, runs of
32 and chunks of 512 sources, groups of 32 and blocks of 128 points)."""
import numpy as np
import pytest

import old_fmm_bem_b200 as ob

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (7, 31), (9, 33), (33, 513), (65, 100), (128, 2100), (129, 65), (300, 129)]


def _plan(kernel, precision, k, p=4):
    return ob.Plan(kernel=kernel, p=p, lmax=2, precision=precision, semantics=ob.SEM_ACCURATE, exclude_self=True,
                   wavenumber=k)


def _charges(rng, kernel, n):
    q = rng.standard_normal(n).astype(np.float32)
    return (q + 1j * rng.standard_normal(n)).astype(np.complex64) if kernel == ob.HELMHOLTZ_G else q


def _direct(kernel, xt, xs, q, k):
    """Sums and sums of the terms' magnitudes."""
    d = xt.astype(np.float64)[:, :, None] - xs.astype(np.float64)[:, None, :]
    r = np.sqrt((d ** 2).sum(0))
    ri = np.where(r > 0, 1.0 / np.where(r > 0, r, 1.0), 0.0)
    if kernel == ob.HELMHOLTZ_G:
        kv = np.exp(1j * k * r) * ri / (4 * np.pi)
    else:
        kv = 0.5 * np.pi * np.exp(-k * r) * ri / k
    t = kv * q.astype(np.complex128 if kernel == ob.HELMHOLTZ_G else np.float64)[None]
    return t.sum(1), abs(t).sum(1)


@pytest.mark.parametrize("kernel,k", [(ob.HELMHOLTZ_G, 1.0), (ob.HELMHOLTZ_G, 60.0), (ob.YUKAWA, 4.0)])
@pytest.mark.parametrize("precision", [ob.FP64, ob.MIXED])
@pytest.mark.parametrize("ni,nj", SIZES)
def test_near_field_equals_direct(kernel, k, precision, ni, nj):
    # all points in eight mutually neighbouring leaves: no far field.  Bounds, per sum of magnitudes: FP64 (n + 16)
    # roundings; mixed: 2^-20 of the hardware sine and cosine, 2^-24 k r of the phase (k r up to 52 here), 2^-22 of the
    # inverse root, the sums of 32 in FP32
    rng = np.random.default_rng(ni * 10007 + nj)
    xt = (rng.random((3, ni)) * np.where(rng.random(ni) < 0.7, 0.24, 0.49)).astype(np.float32)
    xs = (rng.random((3, nj)) * np.where(rng.random(nj) < 0.7, 0.24, 0.49)).astype(np.float32)
    m = min(ni, nj) // 2
    xs[:, :m] = xt[:, :m]  # coincident pairs
    q = _charges(rng, kernel, nj)
    with _plan(kernel, precision, k) as pl:
        pl.set_geometry(xt, xs, bbox=(0, 0, 0, 1))
        pot = np.asarray(pl.evaluate(q, f64=True)[0])
    want, mag = _direct(kernel, xt, xs, q, k)
    # FP64: the phase carries k r 2^-52 besides the sums
    tol = (nj + 16 + 2 * 0.87 * k) * 2.0 ** -53 if precision == ob.FP64 else 2.0 ** -19 + (32 + 0.87 * k) * 2.0 ** -23
    assert np.all(abs(pot - want) <= tol * mag)


@pytest.mark.parametrize("kernel", [ob.HELMHOLTZ_G, ob.YUKAWA])
@pytest.mark.parametrize("p", [3, 8, 16, 20])
@pytest.mark.parametrize("ni,nj", SIZES)
def test_far_field_of_one_pair_of_leaves(kernel, p, ni, nj):
    # sources in one corner leaf, targets in the opposite one: P2M, one M2L, L2P.  Boxes of side 1/4 at distance
    # 0.75 sqrt(3): the truncation error falls as (0.217 / (1.3 - 0.217))^(p + 1) = 0.2^(p + 1), of fields of this size
    # with a factor of about 10
    rng = np.random.default_rng(p * 977 + ni + nj)
    xs = (rng.random((3, nj)) * 0.249).astype(np.float32)
    xt = (0.751 + rng.random((3, ni)) * 0.248).astype(np.float32)
    q = abs(_charges(rng, kernel, nj).real) + 0.1
    q = q.astype(np.complex64 if kernel == ob.HELMHOLTZ_G else np.float32)
    with _plan(kernel, ob.FP64, 2.0, p) as pl:
        pl.set_geometry(xt, xs, bbox=(0, 0, 0, 1))
        pot = np.asarray(pl.evaluate(q, f64=True)[0])
    want, mag = _direct(kernel, xt, xs, q, 2.0)
    assert np.all(abs(pot - want) <= max(10 * 0.2 ** (p + 1), 1e-12) * mag)


def test_a_plan_of_lower_order_in_between():
    # the shared-memory limits of the kernels are process-wide: a plan of order 4 made after one of order 16 leaves the
    # first one's evaluates (its first, launched directly, included) as they are
    rng = np.random.default_rng(8)
    x = rng.random((3, 700)).astype(np.float32)
    q = (rng.standard_normal(700) + 1j * rng.standard_normal(700)).astype(np.complex64)
    kw = dict(kernel=ob.HELMHOLTZ_G, lmax=2, precision=ob.FP64, semantics=ob.SEM_ACCURATE, exclude_self=True, wavenumber=2.0)
    with ob.Plan(p=16, **kw) as a, ob.Plan(p=4, **kw) as b:
        a.set_geometry(x, x, bbox=(0, 0, 0, 1))
        b.set_geometry(x, x, bbox=(0, 0, 0, 1))
        got = np.asarray(a.evaluate(q, f64=True)[0])
        want = np.asarray(a.direct(q)[0])
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("kernel", [ob.HELMHOLTZ_G, ob.YUKAWA])
@pytest.mark.parametrize("precision", [ob.FP64, ob.MIXED])
@pytest.mark.parametrize("where", ["one leaf", "across leaves", "softened"])
def test_squared_distances_below_the_normal_range(kernel, precision, where):
    # r^2 is subnormal in FP32 (r of 5e-21 and more, so 2^-14 of r^2 and less is lost): two close points, a whole domain
    # of that size, and a softening of that size
    rng = np.random.default_rng(11)
    eps2 = 0.0
    if where == "across leaves":
        cells = np.array(np.unravel_index(rng.permutation(512)[:300], (8, 8, 8)))
        x = (1e-20 * (cells + 0.1 + 0.2 * rng.random((3, 300)))).astype(np.float32)
        side = np.float32(16e-20)
    else:
        x, side = (rng.random((3, 40)) * 0.4).astype(np.float32), 1.0
        x[:, 7], x[:, 8] = (0.3, 0, 0.1), (0.3, 2e-20, 0.1)
        if where == "softened":
            eps2 = 1e-40
            x[:, 8] = x[:, 7]
    q = _charges(rng, kernel, x.shape[1])
    with ob.Plan(kernel=kernel, p=4, lmax=2, precision=precision, semantics=ob.SEM_ACCURATE, exclude_self=where != "softened",
                 eps2=eps2, wavenumber=1.0) as pl:
        pl.set_geometry(x, x, bbox=(0, 0, 0, side))
        pot = np.asarray(pl.evaluate(q, f64=True)[0])
        want = np.asarray(pl.direct(q)[0])
    assert np.all(np.isfinite(pot)) and np.linalg.norm(pot - want) <= 2.0 ** -12 * np.linalg.norm(want)
