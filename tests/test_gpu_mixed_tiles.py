"""Mixed form at the edges of its tiles: the many-right-hand-side near field (tiles of 16 targets, teams of 8 warps, groups
of 8 / 4 / 2 / 1 right-hand sides) and the FP32 P2M and L2P (items of 64 sources and 128 targets, 16 staged rows)."""
import numpy as np
import pytest

import old_fmm_bem_b200 as ob

pytestmark = pytest.mark.gpu


def _unit(rng, n):
    v = rng.standard_normal((3, n))
    return (v / np.linalg.norm(v, axis=0)).astype(np.float32)


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI, ob.LAPLACE_GNJ])
@pytest.mark.parametrize("nrhs", [2, 5, 8, 15])
@pytest.mark.parametrize("ni,nj", [(1, 1), (9, 33), (17, 513), (33, 100), (65, 65), (129, 1100), (700, 31)])
def test_many_rhs_near_field_equals_direct(kernel, nrhs, ni, nj):
    # eight mutually neighbouring leaves: no far field.  Bound: at most 67 roundings of an FP32 sum and 13 of a term,
    # 2^-24 each, of the sum of the terms' magnitudes
    rng = np.random.default_rng(ni * 10007 + nj)
    xt = (rng.random((3, ni)) * np.where(rng.random(ni) < 0.7, 0.24, 0.49)).astype(np.float32)
    xs = (rng.random((3, nj)) * np.where(rng.random(nj) < 0.7, 0.24, 0.49)).astype(np.float32)
    m = min(ni, nj) // 2
    xs[:, :m] = xt[:, :m]  # coincident pairs
    tn, sn = _unit(rng, ni), _unit(rng, nj)
    q = rng.standard_normal((nrhs, nj)).astype(np.float32)
    with ob.Plan(kernel=kernel, p=4, lmax=2, precision=ob.MIXED, semantics=ob.SEM_ACCURATE, exclude_self=True,
                 nrhs=nrhs) as pl:
        pl.set_geometry(xt, xs, tn if kernel == ob.LAPLACE_GNI else None, sn if kernel == ob.LAPLACE_GNJ else None,
                        bbox=(0, 0, 0, 1))
        pot, grad = pl.evaluate(q.reshape(-1), f64=True)
    d = xt.astype(np.float64)[:, :, None] - xs.astype(np.float64)[:, None, :]
    r2 = (d ** 2).sum(0)
    ri = np.where(r2 > 0, 1.0 / np.sqrt(np.where(r2 > 0, r2, 1.0)), 0.0)
    qd, c, tol = q.astype(np.float64).T, 0.25 / np.pi, 80 * 2.0 ** -24
    if kernel == ob.LAPLACE_G:
        t = [ri] + [-d[k] * ri ** 3 for k in range(3)]
        mag = [abs(v) for v in t]
    else:
        n = (tn[:, :, None] if kernel == ob.LAPLACE_GNI else sn[:, None, :]).astype(np.float64)
        t, mag = [(d * n).sum(0) * ri ** 3], [abs(d * n).sum(0) * ri ** 3]
    assert np.all(abs(pot.reshape(nrhs, ni).T - c * t[0] @ qd) <= tol * c * (mag[0] @ abs(qd)))
    if grad is not None:
        g = grad.reshape(nrhs, 3, ni)
        for k in range(3):
            assert np.all(abs(g[:, k].T - c * t[1 + k] @ qd) <= tol * c * (mag[1 + k] @ abs(qd)))


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI, ob.LAPLACE_GNJ])
@pytest.mark.parametrize("p", [1, 4, 5, 8, 9, 10, 11, 12, 14, 16])
@pytest.mark.parametrize("ni,nj", [(1, 1), (31, 33), (64, 63), (65, 129), (300, 257)])
def test_mixed_expansions_match_fp64(kernel, p, ni, nj):
    # sources in one corner leaf, targets in the opposite one: P2M, one M2L, L2P.  2e-6 of the sum of magnitudes: FP32
    # terms and sums of up to 64 points, 22-bit operators, FP32 sums of up to p + 1 terms
    rng = np.random.default_rng(p * 977 + ni + 7 * nj)
    xs = (rng.random((3, nj)) * 0.249).astype(np.float32)
    xt = (0.751 + rng.random((3, ni)) * 0.248).astype(np.float32)
    tn, sn = _unit(rng, ni), _unit(rng, nj)
    q = (rng.random(nj) + 0.1).astype(np.float32)
    out = []
    for prec in (ob.MIXED, ob.FP64):
        with ob.Plan(kernel=kernel, p=p, lmax=2, precision=prec, semantics=ob.SEM_ACCURATE, exclude_self=True) as pl:
            pl.set_geometry(xt, xs, tn if kernel == ob.LAPLACE_GNI else None, sn if kernel == ob.LAPLACE_GNJ else None,
                            bbox=(0, 0, 0, 1))
            out.append(pl.evaluate(q, f64=True))
    r = np.linalg.norm(xt.astype(np.float64)[:, :, None] - xs[:, None, :], axis=0)
    mag = (q / (4 * np.pi * (r if kernel == ob.LAPLACE_G else r ** 2))).sum(1)
    assert np.all(abs(out[0][0] - out[1][0]) <= 2e-6 * mag)
    if kernel == ob.LAPLACE_G:
        gm = (q / (4 * np.pi * r ** 2)).sum(1)
        assert np.all(abs(out[0][1] - out[1][1]).reshape(3, -1) <= 2e-6 * gm)


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI, ob.LAPLACE_GNJ])
@pytest.mark.parametrize("precision", [ob.FP64, ob.MIXED])
@pytest.mark.parametrize("nrhs", [1, 2, 8])
def test_excluded_pairs_with_softening(kernel, precision, nrhs):
    # pairs at zero distance are left out whatever the softening; distinct points whose squared distance underflows in
    # FP32 (1e-24 apart) are not.  All points in one leaf; bounds as above
    rng = np.random.default_rng(nrhs)
    n, eps2 = 203, 1e-3
    x = (rng.random((3, n)) * 0.24).astype(np.float32)
    x[:, 50:60] = x[:, 40:50]
    x[:, 0], x[:, 1] = (0.1, 0, 0), (0.1, 1e-24, 0)
    nrm = _unit(rng, n)
    q = rng.standard_normal((nrhs, n)).astype(np.float32)
    with ob.Plan(kernel=kernel, p=4, lmax=2, precision=precision, semantics=ob.SEM_ACCURATE, exclude_self=True, eps2=eps2,
                 nrhs=nrhs) as pl:
        pl.set_geometry(x, x, nrm if kernel == ob.LAPLACE_GNI else None, nrm if kernel == ob.LAPLACE_GNJ else None,
                        bbox=(0, 0, 0, 1))
        pot, grad = pl.evaluate(q.reshape(-1), np.zeros(n * nrhs), np.zeros(3 * n * nrhs), f64=True)
    d = x.astype(np.float64)[:, :, None] - x.astype(np.float64)[:, None, :]
    ri = np.where((d == 0).all(0), 0.0, 1.0 / np.sqrt((d ** 2).sum(0) + eps2))
    if kernel == ob.LAPLACE_G:
        t = [ri] + [-d[k] * ri ** 3 for k in range(3)]
        mag = [abs(v) for v in t]
    else:
        v = (nrm[:, :, None] if kernel == ob.LAPLACE_GNI else nrm[:, None, :]).astype(np.float64)
        dot, m = (d * v).sum(0), abs(d * v).sum(0)
        t = [dot * ri ** 3] + [ri ** 3 * (v[k] - 3 * dot * ri ** 2 * d[k]) for k in range(3)]
        mag = [m * ri ** 3] + [ri ** 3 * (abs(v[k]) + 3 * m * ri ** 2 * abs(d[k])) for k in range(3)]
    qd, c, tol = q.astype(np.float64).T, 0.25 / np.pi, 80 * 2.0 ** -24
    out = [pot.reshape(nrhs, n)] + list(np.moveaxis(grad.reshape(nrhs, 3, n), 1, 0))
    for a, tt, mm in zip(out, t, mag):
        assert np.all(abs(a.T - c * tt @ qd) <= tol * c * (mm @ abs(qd)))


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI])
@pytest.mark.parametrize("p", [4, 8, 11, 12, 16])
def test_fp32_l2p_rounding(kernel, p):
    # the L2P alone: point sources at leaf centres (their multipoles are exact), no near field, the FP64 M2L.  The terms
    # of degree 0 are added in FP64; what is left, FP32 terms of relative size 1/3 and less, carries coordinates, tables
    # and recurrences of 2^-24 each and p + 1 sums of up to p + 1 terms, at random: 2^-24 of the field in the 2-norm
    rng = np.random.default_rng(p)
    far = np.array([(a, b, c) for a in range(8) for b in range(8) for c in range(8) if max(a, b, c) >= 5])
    pick = far[rng.permutation(len(far))[:80]]
    xs = ((pick.T + 0.5) / 8).astype(np.float32)
    xt = (rng.random((3, 4000)) * 0.374).astype(np.float32)
    tn = _unit(rng, 4000)
    q = rng.standard_normal(80).astype(np.float32)
    out = []
    for prec in (ob.MIXED, ob.FP64):
        with ob.Plan(kernel=kernel, p=p, lmax=3, precision=prec, semantics=ob.SEM_ACCURATE, exclude_self=True) as pl:
            pl.set_geometry(xt, xs, tn if kernel == ob.LAPLACE_GNI else None, bbox=(0, 0, 0, 1))
            out.append(pl.evaluate(q, f64=True))
            assert pl.stats()["p2p_pairs"] == 0
    for a, b in zip(*out):
        if a is not None:
            err = np.linalg.norm(a - b) / np.linalg.norm(b)
            print(kernel, p, err)
            assert err <= 2.0 ** -24


@pytest.mark.parametrize("n", [33, 40, 100])
def test_many_rhs_near_field_rounding(n):
    # potentials of equal charges of one sign, n in each of 27 leaves.  A FP32 chain of c terms is off by
    # 0.4 2^-24 sqrt(c / 3) of its sum, M chains by that over sqrt(M) of the total: 0.7e-8 with c = 16 and n = 33, 0.6e-8
    # with c = 32 and n = 100, and the terms' own roundings; chains of 64 terms and sums of several chains in FP32, 2e-8
    err = []
    for seed in range(8):
        rng = np.random.default_rng(seed)
        cells = np.array(np.unravel_index(np.arange(27), (3, 3, 3))).T
        xs = np.concatenate([(c + rng.random((n, 3))) / 4 for c in cells]).T.astype(np.float32)
        xt = ((1 + rng.random((n, 3))) / 4).T.astype(np.float32)
        q = rng.random((4, 27 * n)).astype(np.float32)
        with ob.Plan(kernel=ob.LAPLACE_G, p=4, lmax=2, precision=ob.MIXED, semantics=ob.SEM_ACCURATE, exclude_self=True,
                     nrhs=4) as pl:
            pl.set_geometry(xt, xs, bbox=(0, 0, 0, 1))
            pot, _ = pl.evaluate(q.reshape(-1), f64=True)
        r = np.linalg.norm(xt.astype(np.float64)[:, :, None] - xs[:, None, :], axis=0)
        want = q.astype(np.float64) @ (0.25 / (np.pi * r)).T
        err.append(np.linalg.norm(pot.reshape(4, n) - want) / np.linalg.norm(want))
    err = np.exp(np.mean(np.log(err)))
    print(n, err)
    assert err <= 1.6e-8
