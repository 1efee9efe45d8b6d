"""P2G pass 1 adds a term as two 32-bit pieces and falls back to 64-bit sums
per leaf when a term is 65,536 or more; small launches run one CTA per leaf and
component.  Both must give the exact fixed-point sums: faces are compared with
float64 sums of the kernel's own per-cell float32 sums, rounded to 2^-32."""
import numpy as np
import pytest

import fsim

pytestmark = pytest.mark.gpu


def _p2g(pos, vel, dims):
    """Fixed-point P2G of velocity component 0 on dense nodes [-1, N + 1]."""
    f32 = np.float32
    cell = np.floor(pos).astype(int)
    order = np.lexsort((np.arange(len(pos)), cell[:, 2], cell[:, 1], cell[:, 0]))
    shape = tuple(d + 3 for d in dims)
    mom, mass = np.zeros(shape, np.float64), np.zeros(shape, np.float64)
    boxes = {}
    for q in order:
        p, c = pos[q], tuple(cell[q])
        am, aw = boxes.setdefault(c, (np.zeros((2, 3, 3), f32), np.zeros((2, 3, 3), f32)))
        w = np.zeros((3, 3), f32)
        w[0, :2] = f32(1) - f32(p[0] - f32(c[0])), f32(p[0] - f32(c[0]))
        for ax in (1, 2):
            lo = f32(c[ax]) + f32(0.5)
            k = 0 if p[ax] < lo else 1
            f = f32(p[ax] - (lo - f32(1))) if k == 0 else f32(p[ax] - lo)
            w[ax, k], w[ax, k + 1] = f32(1) - f, f
        for i in range(2):
            for j in range(3):
                wij = f32(w[0, i] * w[1, j])
                ww = (wij * w[2]).astype(f32)
                am[i, j] = am[i, j] + (ww * vel[q, 0]).astype(f32)
                aw[i, j] = aw[i, j] + ww
    for c, (am, aw) in boxes.items():
        s = np.s_[c[0] + 1:c[0] + 3, c[1]:c[1] + 3, c[2]:c[2] + 3]
        mom[s] += np.rint(am.astype(np.float64) * 2.0 ** 32)
        mass[s] += np.rint(aw.astype(np.float64) * 2.0 ** 32)
    return mom * 2.0 ** -32, mass * 2.0 ** -32


# 1e3: pieces; 7e4 and 3e5: some and most leaves on the 64-bit path
@pytest.mark.parametrize("speed", [1e3, 7e4, 3e5])
@pytest.mark.parametrize("dims,n", [((8, 8, 8), 300), ((17, 9, 24), 900)])
def test_exact_sums(dims, n, speed):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * np.array(dims) * 0.999).astype(np.float32)
    vel = (rng.standard_normal((n, 3)) * speed).astype(np.float32)
    vel[: n // 2] *= np.float32(1e-3)
    g, f = fsim.physical_gravity(dims[1])
    with fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f) as sim:
        sim.upload_particles(pos, vel, vel)
        p, v, _ = sim.download_particles()
        sim.transfer_particles_to_grid()
        w, on = sim.field(fsim.FIELD_WEIGHT)
        u, _ = sim.field(fsim.FIELD_VELOCITY)
    mom, mass = _p2g(p, v, dims)
    mom, mass = (a[:-1, :-1, :-1] for a in (mom, mass))
    face = on.astype(bool) & (mass >= 2e-3)  # lower ones are summed again in float order
    assert face.sum() > 100
    assert np.array_equal(w[..., 0][face], mass[face].astype(np.float32))
    ref = mom[face].astype(np.float32) / mass[face].astype(np.float32)
    assert np.array_equal(u[..., 0][face], ref)
