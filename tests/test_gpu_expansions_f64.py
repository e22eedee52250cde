"""FP64 P2M and L2P at the edges of their tiles (groups of 32 and blocks of 128 points, items of 128 targets, row tiles of
8 orders' terms), both semantics, against the CPU restatement."""
import numpy as np
import pytest

import old_fmm_bem_b200 as ob
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [ob.LAPLACE_G, ob.LAPLACE_GNI, ob.LAPLACE_GNJ])
@pytest.mark.parametrize("ref", [False, True])
@pytest.mark.parametrize("p", [1, 2, 7, 8, 12, 16])
@pytest.mark.parametrize("ni,nj", [(1, 1), (31, 33), (64, 32), (65, 128), (129, 129), (300, 257)])
def test_one_pair_of_leaves(kernel, ref, p, ni, nj):
    # sources in one corner leaf, targets in the opposite one: no near field.  Expansions within (p + 1)^2 + n roundings
    # of 2^-53, growth of the recurrences below 100; outputs likewise (the oracle sums them in float in reference
    # semantics)
    rng = np.random.default_rng(p * 977 + ni + 7 * nj)
    xs = (rng.random((3, nj)) * 0.249).astype(np.float32)
    xt = (0.751 + rng.random((3, ni)) * 0.248).astype(np.float32)
    unit = lambda n: (lambda v: (v / np.linalg.norm(v, axis=0)).astype(np.float32))(rng.standard_normal((3, n)))
    tn, sn, q = unit(ni), unit(nj), rng.standard_normal(nj).astype(np.float32)
    with ob.Plan(kernel=kernel, p=p, lmax=2, precision=ob.FP64, semantics=ob.SEM_REFERENCE if ref else ob.SEM_ACCURATE,
                 exclude_self=not ref) as pl:
        pl.set_geometry(xt, xs, tn if kernel == ob.LAPLACE_GNI else None, sn if kernel == ob.LAPLACE_GNJ else None,
                        bbox=(0, 0, 0, 1))
        pot, grad = pl.evaluate(q, f64=True)
        M = pl.expansions(0)
    po, go = pyoracle.oracle_fmm(xt, xs, q, neq=kernel, p=p, lmax=2, ref_semantics=ref, exclude_self=not ref, tn=tn,
                                 sn=sn)[:2]
    Mo = pyoracle.oracle_expansions(0)
    tol = 100 * ((p + 1) ** 2 + nj) * 2.0 ** -53
    assert np.linalg.norm(M - Mo) <= tol * np.linalg.norm(Mo)
    if ref:
        tol = 1e-6
    assert np.linalg.norm(pot - po) <= tol * np.linalg.norm(po)
    if kernel == ob.LAPLACE_G:
        assert np.linalg.norm(grad.reshape(3, -1) - go) <= tol * np.linalg.norm(go)
