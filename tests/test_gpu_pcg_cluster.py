"""The cluster loop: FP32 and MIXED solves of at most 192 particle leaves run
every iteration inside one 16-CTA thread-block cluster.
Its element-wise arithmetic is the spmv / update pair's and its dot products
are summed in another order, so the bars are the solver's own, as for the
resident loop: fixed iteration counts track the oracle and the pair, relative
solves are no further from the converged solution than the oracle's."""
import numpy as np
import pytest

import fsim
from _util import rel_l2
from test_gpu_pcg import _pressures, _prepared

pytestmark = pytest.mark.gpu


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
    return st, any("cluster" in k for k in names)


def _system(dims, fill, seed=0):
    """A noisy system in box dims whose particles fill the cells where fill is
    true, assembled on the handle."""
    rng = np.random.default_rng(seed)
    cells = np.argwhere(fill)
    pos = (np.repeat(cells, 4, axis=0) + rng.uniform(0.01, 0.99, (4 * len(cells), 3)))
    pos = pos.astype(np.float32)
    vel = rng.normal(0, 5.0, pos.shape).astype(np.float32)
    g, f = fsim.physical_gravity(dims[1])

    def make():
        sim = fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f)
        sim.upload_particles(pos, vel, vel)
        sim.transfer_particles_to_grid()
        sim.apply_boundary_conditions()
        sim.add_gravity(0.01)
        sim.apply_boundary_conditions()
        sim.compute_divergence()
        return sim

    return make


def _first_leaves(dims, n):
    """The cells of n leaves: x-major columns of the box's leaves."""
    lv = [-(-d // 8) for d in dims]
    on = np.zeros(lv, bool)
    on.reshape(-1)[:n] = True
    full = on.repeat(8, 0).repeat(8, 1).repeat(8, 2)
    return full[: dims[0], : dims[1], : dims[2]]


# 1, 2: most CTAs hold nothing; 15 - 17: one and two leaves per CTA; 192: the
# largest; 193 and above: past it
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 45, 159, 192, 193, 209, 256, 257])
@pytest.mark.parametrize("prec", [fsim.PREC_FP32, fsim.PREC_MIXED])
def test_tracks_the_pair_over_leaf_counts(monkeypatch, n, prec):
    dims = (61, 64, 51)
    make = _system(dims, _first_leaves(dims, n), seed=n)
    got = {}
    for res in (None, "0"):
        with monkeypatch.context() as m:
            if res is not None:
                m.setenv("FSIM_PCG_RES", res)
            sim = make()
        assert sim.leaves().shape[0] == n
        for it in (1, 12):
            prm = (fsim.pcg_params(fsim.PCG_FIXED, prec, it) if prec == fsim.PREC_FP32 else
                   fsim.pcg_params(fsim.PCG_RELATIVE, prec, it, tolerance=1e-14,
                                   inner_tolerance=1e-14, max_refinements=1))
            st, cluster = _solve(sim, prm)
            assert cluster == (res is None and n <= 192)
            assert st.iterations == it
            got[res, it] = (st.rr, sim.field(fsim.FIELD_PRESSURE)[0])
        sim.close()
    for it in (1, 12):
        rr, x = got[None, it]
        rr0, x0 = got["0", it]
        # same operations; the dot products' order differs
        assert rel_l2(x, x0) <= 1e-5 and abs(rr - rr0) <= 1e-3 * rr0, it


@pytest.mark.parametrize("n,scene", [(24, "sphere_drop"), (32, "dam_break"), (64, "sphere_drop")])
def test_against_oracle(n, scene):
    orc, sim = _prepared(n=n, scene=scene)
    assert sim.leaves().shape[0] <= 192
    for it in (1, 5, 25):
        st, cluster = _solve(sim, fsim.pcg_params(fsim.PCG_FIXED, fsim.PREC_FP32, it))
        ost = orc.pcg_solve(mode=2, precision=0, max_iterations=it)
        assert cluster and st.status == 0 and st.iterations == it
        a, b = _pressures(sim, orc)
        assert rel_l2(a, b) <= 1e-5, it
        assert abs(st.rr - ost.rr) <= 1e-3 * ost.rr + 1e-30, it
    prm = fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_FP32, 3000, tolerance=1e-5)
    st, _ = _solve(sim, prm)
    a = sim.field(fsim.FIELD_PRESSURE)[0]
    again, _ = _solve(sim, prm)  # fixed-order sums: the same bits
    assert (again.iterations, again.rr) == (st.iterations, st.rr)
    assert np.array_equal(sim.field(fsim.FIELD_PRESSURE)[0], a)
    ost = orc.pcg_solve(mode=1, precision=0, max_iterations=3000, tol=1e-5)
    b = orc.field(4)[0]
    assert st.status == 0 and st.iterations <= 1.1 * ost.iterations + 2
    mixed, _ = _solve(sim, fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_MIXED, 3000,
                                           tolerance=1e-9, inner_tolerance=1e-3,
                                           max_refinements=20))
    c = sim.field(fsim.FIELD_PRESSURE)[0]
    orc.pcg_solve(mode=1, precision=2, max_iterations=20000, tol=1e-13)
    x64 = orc.pressure_f64()
    assert rel_l2(a, x64) <= max(1e-5, 1.5 * rel_l2(b, x64))
    assert mixed.status == 0 and mixed.refinements >= 2 and np.sqrt(mixed.rr / mixed.bb) <= 1e-9
    assert rel_l2(c, x64) <= 1e-6
    sim.close()


def test_rules_and_statuses():
    orc, sim = _prepared()
    prm = sim.default_pcg_params()  # the reference's absolute rule
    st, cluster = _solve(sim, prm)
    ost = orc.pcg_solve(mode=0, precision=0, max_iterations=1500, threshold=prm.threshold)
    assert cluster and st.status == 0 and st.rr < prm.threshold
    assert abs(st.iterations - ost.iterations) <= 2 + ost.iterations // 20
    st, _ = _solve(sim, fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_FP32, 3, tolerance=1e-12))
    assert st.status == fsim.ERR_NOT_CONVERGED and st.iterations == 3
    st, _ = _solve(sim, fsim.pcg_params(fsim.PCG_FIXED, fsim.PREC_FP32, 0))
    assert st.iterations == 0 and not sim.field(fsim.FIELD_PRESSURE)[0].any()
    sim.close()
    # no fluid at all (one particle inside a solid): converged at once, or a
    # breakdown of 0 / 0 when iterations are forced
    g, f = fsim.physical_gravity(16)
    with fsim.Simulation((16, 16, 16), fsim.BOUNDARY_BOX, g, f) as sim:
        sim.add_solid_cuboid((4, 4, 4), (9, 9, 9))
        pos = np.full((1, 3), 6.5, np.float32)
        sim.upload_particles(pos, 0 * pos, 0 * pos)
        sim.transfer_particles_to_grid()
        sim.apply_boundary_conditions()
        sim.compute_divergence()
        st, cluster = _solve(sim, sim.default_pcg_params())
        assert cluster and st.status == 0 and st.iterations == 0 and st.n_rows == 0
        st, _ = _solve(sim, fsim.pcg_params(fsim.PCG_FIXED, fsim.PREC_FP32, 3))
        assert st.status == fsim.ERR_BREAKDOWN


def test_wait_gives_up_and_recovers(monkeypatch):
    """With FSIM_PCG_RES_WITHHOLD=1 CTA 0 pushes nothing in the first solve's
    first round (and the limit is 256 polls): every CTA's wait gives up, the
    solve reports FSIM_ERR_TIMEOUT, and the next one is a clean handle's."""
    prm = fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_FP32, 3000, tolerance=1e-5)
    _, ref = _prepared()
    st_ref = ref.pcg_solve(prm)
    x_ref = ref.field(fsim.FIELD_PRESSURE)[0]
    ref.close()
    with monkeypatch.context() as m:
        m.setenv("FSIM_PCG_RES_WITHHOLD", "1")
        _, sim = _prepared()
    with pytest.raises(fsim.FsimError) as err:
        sim.pcg_solve(prm)
    assert err.value.code == fsim.ERR_TIMEOUT
    st, cluster = _solve(sim, prm)
    assert cluster and (st.iterations, st.rr) == (st_ref.iterations, st_ref.rr)
    assert np.array_equal(sim.field(fsim.FIELD_PRESSURE)[0], x_ref)
    sim.close()
