"""A step whose pressure solve gives up (FSIM_ERR_TIMEOUT) applies nothing of
it: the particles are moved and keep their velocities, the grid keeps the
velocities from before the projection, no pressure is reported, time stands
still, and a fresh upload steps as on a handle that never timed out."""
import numpy as np
import pytest

import fsim

pytestmark = pytest.mark.gpu

DT = 0.01


def _state(n):
    """The cells of a dam break, eight particles each, with noisy velocities."""
    cells = np.argwhere(np.ones((n // 2, n // 2, n), bool))
    rng = np.random.default_rng(n)
    pos = (np.repeat(cells, 8, axis=0) + rng.uniform(0.01, 0.99, (8 * len(cells), 3)))
    vel = rng.normal(0, 0.3 * n, pos.shape).astype(np.float32)
    return pos.astype(np.float32), vel, vel


def _sim(n, tank):
    g, f = fsim.physical_gravity(n)
    return fsim.Simulation((n, n, n), fsim.BOUNDARY_TANK if tank else fsim.BOUNDARY_BOX, g, f)


# the cluster loop, the resident loop's register kernel and its FP64 form
@pytest.mark.parametrize("prec,res", [(fsim.PREC_FP32, None), (fsim.PREC_FP32, "1"),
                                      (fsim.PREC_FP64, "1")])
@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("tank", [False, True])
def test_nothing_of_the_solve_is_applied(monkeypatch, prec, res, host, tank):
    n = 32
    prm = fsim.pcg_params(fsim.PCG_RELATIVE, prec, 2000, tolerance=1e-5)
    state = _state(n)
    monkeypatch.delenv("FSIM_PCG_CG1", raising=False)
    monkeypatch.delenv("FSIM_PCG_RES", raising=False)
    if res is not None:
        monkeypatch.setenv("FSIM_PCG_RES", res)
    with _sim(n, tank) as ref:
        ref.upload_particles(*state)
        ref.move_particles(DT)
        pos1, vel1, _ = ref.download_particles()
        ref.upload_particles(*state)
        ref.step(DT, prm)
        want = ref.download_particles()
    with monkeypatch.context() as m:
        m.setenv("FSIM_PCG_RES_WITHHOLD", "1")
        sim = _sim(n, tank)
    sim.upload_particles(*state)
    with pytest.raises(fsim.FsimError) as err:
        if host:
            sim.step_host(DT, prm, *state)
        else:
            sim.step(DT, prm)
    assert err.value.code == fsim.ERR_TIMEOUT
    p, v, _ = sim.download_particles()
    assert np.array_equal(p, pos1) and np.array_equal(v, vel1)
    assert not sim.field(fsim.FIELD_PRESSURE)[0].any() and sim.time == 0.0
    # nothing has been projected: the saved velocities are still those before gravity
    u, saved = sim.field(fsim.FIELD_VELOCITY)[0], sim.field(fsim.FIELD_VELOCITY_UPDATE)[0]
    assert np.array_equal(u[..., 0], saved[..., 0]) and np.array_equal(u[..., 2], saved[..., 2])
    sim.upload_particles(*state)
    sim.step(DT, prm)
    for got, ref_rows in zip(sim.download_particles(), want):
        assert np.array_equal(got, ref_rows)
    sim.close()
