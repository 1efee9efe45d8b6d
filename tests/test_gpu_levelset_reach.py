"""Level-set bands whose radius + half width lies just above a whole number and
rounds to it: particles exactly that far from a voxel are inside the band by a
rounding, and the cell search must still reach them."""
import numpy as np
import pytest

import fsim
from test_gpu_levelset_gather import _check

pytestmark = pytest.mark.gpu

# (reach R, radius, half width) with fl(radius + w) = R and fl(R - radius) < w
BANDS = [(1, 0.73950356, 0.26049647), (2, 0.62280816, 1.3771919), (4, 3.2134106, 0.78658944),
         (7, 5.6242356, 1.3757645), (8, 3.3696191, 4.630381)]


@pytest.mark.parametrize("reach,radius,w", BANDS)
def test_band_edge_on_a_whole_number(reach, radius, w):
    f32 = np.float32
    radius, w = f32(radius), f32(w)
    assert f32(radius + w) == reach and f32(f32(reach) - radius) < w
    dims = (33, 20, 17)
    pos = np.array([[16.0, 9.0, 8.0]], f32)  # on a voxel point: whole distances
    g, f = fsim.physical_gravity(dims[1])
    with fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f) as sim:
        sim.upload_particles(pos, 0 * pos, 0 * pos)
        _check(sim, pos, dims, radius, w)


@pytest.mark.parametrize("radius,w", [(1e-23, 1e-23), (1e-20, 1e-20), (1e-23, 0.5), (7.0, 1e-9), (3.0, 1e-20)])
def test_bands_of_very_different_sizes(radius, w):
    dims = (17, 16, 9)
    pos = np.array([[8.0, 9.0, 4.0], [3.25, 9.0, 4.0]], np.float32)
    g, f = fsim.physical_gravity(dims[1])
    with fsim.Simulation(dims, fsim.BOUNDARY_BOX, g, f) as sim:
        sim.upload_particles(pos, 0 * pos, 0 * pos)
        _check(sim, pos, dims, radius, w)
