"""The level set's gather over cell rings against a NumPy restatement of the
splat, bit for bit: odd box sizes, sparse particles (whole leaves empty),
particles on cell faces and box walls, bands up to the leaf neighbourhood's
reach (8 voxels) and past it (the splat), and particles that are deleted or
not binned yet."""
import numpy as np
import pytest

import fsim

pytestmark = pytest.mark.gpu


def _reference(pos, dims, radius, w):
    f32 = np.float32
    ax = [np.arange(-1, d + 1, dtype=f32) for d in dims]
    d2 = np.full([len(a) for a in ax], np.inf, f32)
    for p in pos:
        sq = [(a - q) * (a - q) for a, q in zip(ax, p)]
        d2 = np.minimum(d2, (sq[0][:, None, None] + sq[1][None, :, None]) + sq[2][None, None, :])
    return np.clip(np.sqrt(d2) - f32(radius), -f32(w), f32(w))


def _check(sim, pos, dims, radius, w):
    phi, act = sim.level_set(radius, w, 0)
    ref = _reference(pos, dims, radius, w)
    assert np.array_equal(phi, ref)
    assert np.array_equal(act, (np.abs(ref) < np.float32(w)).astype(np.uint8))


@pytest.mark.parametrize("radius,w", [(3.0, 3.0), (0.3, 0.4), (1.25, 2.5), (5.0, 3.0), (4.5, 4.0)])
@pytest.mark.parametrize("dims,n", [((17, 33, 9), 40), ((40, 8, 23), 1), ((16, 16, 16), 3000)])
def test_gather_matches_splat(dims, n, radius, w):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * np.array(dims)).astype(np.float32)
    pos[0] = [0.0, dims[1], 0.5]  # on the walls
    if n > 2:
        pos[1], pos[2] = [8.0, 8.0, 8.0], [7.9999995, 8.0, 3.0]  # leaf corner and face
    pos = np.minimum(pos, np.array(dims, np.float32))
    g, f = fsim.physical_gravity(dims[1])
    with fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f) as sim:
        z = np.zeros_like(pos)
        sim.upload_particles(pos, z, z)
        _check(sim, pos, dims, radius, w)


def test_deleted_and_appended_particles():
    dims = (16, 16, 16)
    g, f = fsim.physical_gravity(16)
    with fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f) as sim:
        sim.seed(fsim.scene_passes("sphere_drop", 16), seed=0)
        pos, vel, gvel = sim.download_particles()
        src = fsim.fsim_source()
        src.lo[:], src.hi[:] = (3.0, 1.0, 2.0), (9.0, 14.0, 12.0)
        sim.add_source(src)
        sim.delete_fluid_in_sources(0.0)
        kept = ~np.all((pos >= [3, 1, 2]) & (pos <= [8, 13, 11]), axis=1)
        assert 0 < kept.sum() < len(pos)
        # the packed download: the kept rows of every field, in order
        for got, ref in zip(sim.download_particles(), (pos, vel, gvel)):
            assert np.array_equal(got, ref[kept])
        _check(sim, pos[kept], dims, 3.0, 3.0)
        sim.add_contribution_from_sources(0.0)
        now = sim.download_particles()[0]
        assert len(now) > kept.sum()
        _check(sim, now, dims, 3.0, 3.0)


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 2500])
def test_packed_download_block_edges(n):
    """Deleted particles at the ends of the packing blocks."""
    dims = (16, 16, 16)
    g, f = fsim.physical_gravity(16)
    rng = np.random.default_rng(n)
    pos = np.sort(rng.random((n, 3)).astype(np.float32) * 8, axis=0)
    vel = rng.standard_normal((n, 3)).astype(np.float32)
    with fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f) as sim:
        sim.upload_particles(pos, vel, -vel)
        pos, vel, gvel = sim.download_particles()
        src = fsim.fsim_source()
        src.lo[:], src.hi[:] = (0.0, 0.0, 0.0), (9.0, 9.0, float(pos[n // 2, 2]) + 1.0)
        sim.add_source(src)
        sim.delete_fluid_in_sources(0.0)
        kept = pos[:, 2] > np.float32(src.hi[2]) - np.float32(1.0)  # the box's end less one
        for got, ref in zip(sim.download_particles(), (pos, vel, gvel)):
            assert np.array_equal(got, ref[kept])
