"""The resident loop in every precision, and its grid barrier's sums: each CTA
adds its partials as fixed-point words (exact in their units, at the scale of
the previous total), and every CTA takes an extra barrier with sums through
memory when a partial is out of the words' range or a total is too small."""
import numpy as np
import pytest

import fsim
from _util import rel_l2
from test_gpu_pcg import _prepared
from test_gpu_pcg_cluster import _first_leaves, _system

pytestmark = pytest.mark.gpu

PRECS = [fsim.PREC_FP32, fsim.PREC_MIXED, fsim.PREC_FP64]


@pytest.fixture(autouse=True)
def _defaults(monkeypatch):
    monkeypatch.delenv("FSIM_PCG_RES", raising=False)
    monkeypatch.delenv("FSIM_PCG_CG1", raising=False)


def _solve(sim, prm):
    sim.set_profiling(True)
    sim.reset_kernel_times()
    st = sim.pcg_solve(prm)
    names = set(sim.kernel_times())
    sim.set_profiling(False)
    return st, any(k.startswith("pcg_resident") for k in names)


def _fixed(prec, it):
    if prec != fsim.PREC_MIXED:
        return fsim.pcg_params(fsim.PCG_FIXED, prec, it)
    return fsim.pcg_params(fsim.PCG_RELATIVE, prec, it, tolerance=1e-14, inner_tolerance=1e-14,
                           max_refinements=1)


# 1: most CTAs hold nothing; 152, 153: one leaf per SM and the first with two;
# 700: several half leaves per warp for FP64
@pytest.mark.parametrize("n", [1, 2, 152, 153, 305, 700])
@pytest.mark.parametrize("prec", PRECS)
def test_tracks_the_pair(monkeypatch, n, prec):
    dims = (77, 80, 51)
    make = _system(dims, _first_leaves(dims, n), seed=n)
    got = {}
    for res in ("1", "0"):
        with monkeypatch.context() as m:
            m.setenv("FSIM_PCG_RES", res)
            sim = make()
        assert sim.leaves().shape[0] == n
        for it in (1, 12):
            st, resident = _solve(sim, _fixed(prec, it))
            assert resident == (res == "1") and st.iterations == it
            got[res, it] = (st.rr, sim.field(fsim.FIELD_PRESSURE)[0])
        sim.close()
    tol = 1e-6 if prec == fsim.PREC_FP64 else 1e-5  # pressures are fp32 fields
    for it in (1, 12):
        (rr, x), (rr0, x0) = got["1", it], got["0", it]
        assert rel_l2(x, x0) <= tol and abs(rr - rr0) <= 1e-3 * rr0, it


@pytest.mark.parametrize("prec", PRECS)
def test_converged_and_repeatable(monkeypatch, prec):
    monkeypatch.setenv("FSIM_PCG_RES", "1")
    orc, sim = _prepared(n=48, scene="sphere_drop")
    tol = {fsim.PREC_FP32: 1e-5, fsim.PREC_MIXED: 1e-9, fsim.PREC_FP64: 1e-12}[prec]
    prm = fsim.pcg_params(fsim.PCG_RELATIVE, prec, 20000, tolerance=tol, inner_tolerance=1e-3,
                          max_refinements=20)
    st, resident = _solve(sim, prm)
    assert resident and st.status == 0 and np.sqrt(st.rr / st.bb) <= tol
    x = sim.field(fsim.FIELD_PRESSURE)[0]
    st2, _ = _solve(sim, prm)
    assert (st2.iterations, st2.rr) == (st.iterations, st.rr)
    assert np.array_equal(sim.field(fsim.FIELD_PRESSURE)[0], x)
    orc.pcg_solve(mode=1, precision=0, max_iterations=20000, tol=1e-5)
    x32 = orc.field(4)[0]
    ost = orc.pcg_solve(mode=1, precision=2, max_iterations=20000, tol=1e-13)
    x64 = orc.pressure_f64()
    # FP32 stops at a residual of 1e-5: its error is the solver's own, as the oracle's
    bar = {fsim.PREC_FP32: max(1e-5, 1.5 * rel_l2(x32, x64)), fsim.PREC_MIXED: 1e-6,
           fsim.PREC_FP64: 1e-7}[prec]
    assert rel_l2(x, x64) <= bar
    if prec == fsim.PREC_FP64:
        assert st.iterations <= ost.iterations + 2
    sim.close()


@pytest.mark.parametrize("prec", PRECS)
def test_totals_out_of_the_words_range(monkeypatch, prec):
    """Isolated fluid cells converge in one iteration: r.r drops to rounding
    (far more than 2^7 at once) and then stays or hits 0, so every later
    barrier sums through memory.  Status and iterations are the pair's."""
    n = 32
    fill = np.zeros((n, n, n), bool)
    fill[2::4, 2::4, 2::4] = True
    make = _system((n, n, n), fill, seed=3)
    got = []
    for res in ("1", "0"):
        with monkeypatch.context() as m:
            m.setenv("FSIM_PCG_RES", res)
            sim = make()
        st, resident = _solve(sim, fsim.pcg_params(fsim.PCG_RELATIVE, prec, 50, tolerance=1e-5))
        assert resident == (res == "1") and st.status == 0
        x = sim.field(fsim.FIELD_PRESSURE)[0]
        more, _ = _solve(sim, _fixed(prec, 4))
        got.append((st.iterations, x, more.status in (fsim.OK, fsim.ERR_BREAKDOWN,
                                                       fsim.ERR_NOT_CONVERGED)))
        sim.close()
    assert got[0][0] == got[1][0] and got[0][2] and got[1][2]
    assert rel_l2(got[0][1], got[1][1]) <= 1e-6


def test_default_choice():
    """48^3 (84 leaves): the cluster loop for FP32 and MIXED, the resident loop
    for FP64; a system of about 700 leaves: the resident loop for all three."""
    orc, sim = _prepared(n=48, scene="sphere_drop")
    assert [_solve(sim, _fixed(p, 2))[1] for p in PRECS] == [False, False, True]
    sim.close()
    dims = (77, 80, 51)
    sim = _system(dims, _first_leaves(dims, 700))()
    assert [_solve(sim, _fixed(p, 2))[1] for p in PRECS] == [True, True, True]
    sim.close()
