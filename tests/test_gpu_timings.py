"""fmmb_get_timings runs the last evaluate's launches once more: with that evaluate's charges, in its stream layout, and
without a trace in what the plan holds; fmmb_set_overlap runs nothing."""
import numpy as np
import pytest

import old_fmm_bem_b200 as ob

pytestmark = pytest.mark.gpu
N = 3001


def _case(kernel, precision, nrhs):
    rng = np.random.default_rng(5)
    helm = kernel in (ob.HELMHOLTZ_G, ob.YUKAWA)
    x = rng.random((3, N)).astype(np.float32)
    q = [rng.standard_normal(N * k).astype(np.float32) for k in (nrhs, 1)]
    if kernel == ob.HELMHOLTZ_G:
        q = [v.astype(np.complex64) for v in q]
    pl = ob.Plan(kernel=kernel, p=6, lmax=3, precision=precision, semantics=ob.SEM_ACCURATE, exclude_self=True, nrhs=nrhs,
                 **(dict(wavenumber=2.0) if helm else {}))
    pl.set_geometry(x, x, bbox=(0, 0, 0, 1))
    return pl, x, q


@pytest.mark.parametrize("kernel,precision,nrhs", [(ob.LAPLACE_G, ob.FP64, 1), (ob.LAPLACE_G, ob.FP64, 3),
                                                   (ob.LAPLACE_G, ob.MIXED, 1), (ob.LAPLACE_G, ob.MIXED, 3),
                                                   (ob.HELMHOLTZ_G, ob.MIXED, 1), (ob.YUKAWA, ob.FP64, 2)])
@pytest.mark.parametrize("switch", [False, True])
@pytest.mark.parametrize("evaluates", [1, 3])
def test_expansions_stay_the_last_evaluates(kernel, precision, nrhs, switch, evaluates):
    # not even their last bits (the atomics' order) change: nothing writes them
    pl, x, q = _case(kernel, precision, nrhs)
    with pl:
        for _ in range(evaluates):
            pl.evaluate(q[0], f64=True)
        want = [pl.expansions(w) for w in (0, 1)]
        pl.direct(q[1])  # other charges
        if switch:
            pl.set_overlap(False)
        ph = pl.timings()
        assert all(ph[k] > 0 for k in ph if k != "p2p") and (ph["p2p"] > 0) != (nrhs > 1 and precision == ob.MIXED)
        assert pl.timings() == ph  # measured once
        for w in (0, 1):
            assert np.array_equal(pl.expansions(w), want[w])


def test_set_overlap_runs_nothing():
    # it changes the plan's state and returns while the plan's stream is busy (here for some 0.2 s)
    torch = pytest.importorskip("torch")
    pl, x, q = _case(ob.LAPLACE_G, ob.MIXED, 1)
    s, e = torch.cuda.Stream(), torch.cuda.Event()
    with pl:
        pl.set_stream(s)
        pl.evaluate(q[0])
        s.synchronize()
        with torch.cuda.stream(s):
            torch.cuda._sleep(400_000_000)
            e.record(s)
            pl.set_overlap(False)
            assert not e.query()
        s.synchronize()
        assert all(v > 0 for v in pl.timings().values())


@pytest.mark.parametrize("read", [False, True])
def test_phases_after_a_new_geometry(read):
    # the last evaluate's where they were read in time, else 0; never another geometry's
    pl, x, q = _case(ob.LAPLACE_G, ob.MIXED, 1)
    with pl:
        pl.evaluate(q[0])
        before = pl.timings() if read else None
        pl.set_geometry(x, x, bbox=(0, 0, 0, 1))
        ph = pl.timings()
        assert ph == before if read else ph.pop("total") > 0 and not any(ph.values())
        pl.evaluate(q[0])
        now = pl.timings()
        assert all(v > 0 for v in now.values()) and now != before


def test_a_refused_geometry_keeps_the_phases():
    pl, x, q = _case(ob.LAPLACE_G, ob.MIXED, 1)
    with pl:
        pl.evaluate(q[0])
        with pytest.raises(ob.FMMError):
            pl.set_geometry(x, x, bbox=(0, 0, 0, -1))
        assert all(v > 0 for v in pl.timings().values())
