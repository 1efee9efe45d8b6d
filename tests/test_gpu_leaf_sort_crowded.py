"""Crowded cells in the rebinning's per-leaf sort: the order stays a stable sort
by (new cell, old cell, row), and its time does not grow with the square of a
cell's particles."""
import numpy as np
import pytest

import fsim
from test_gpu_leaf_sort import _cell_keys

pytestmark = pytest.mark.gpu

N = 24


def _rows(counts, rng):
    """counts[i] particles in cell i of the leaf at (8, 8, 8), rows shuffled."""
    c = np.repeat(np.arange(len(counts)), counts)
    pos = 8 + np.stack([c >> 6, (c >> 3) & 7, c & 7], 1) + rng.uniform(0.01, 0.99, (len(c), 3))
    return pos[rng.permutation(len(c))].astype(np.float32)


# cells around the lengths where another way of ordering takes over, alone and
# beside others; a leaf at its limit in 1, 2, 3 and 48 cells
CASES = {
    "ends": [0, 1, 31, 32, 33, 47, 48, 49, 50, 63, 64, 65, 66, 127, 128, 129, 255, 256, 257],
    "wide": [1023, 1024, 1025, 5, 1026, 0, 2047, 2048, 2049, 64, 65],
    "one": [12288],
    "two": [6144, 6144],
    "three": [1, 12286, 1],
    "many": [256] * 48,
}


def _sim():
    g, f = fsim.physical_gravity(N)
    return fsim.Simulation((N, N, N), fsim.BOUNDARY_BOX, g, f)


@pytest.mark.parametrize("case", sorted(CASES))
def test_order(case):
    rng = np.random.default_rng(11)
    pos = _rows(CASES[case], rng)
    tag = np.arange(3 * len(pos), dtype=np.float32).reshape(-1, 3)
    zero = np.zeros_like(pos)
    with _sim() as sim:
        sim.upload_particles(pos, tag, zero)
        want = np.argsort(_cell_keys(pos), kind="stable")
        p, v, _ = sim.download_particles()
        assert np.array_equal(p, pos[want]) and np.array_equal(v, tag[want])
    # rows out of order before a move: old cells break ties in the new ones.
    # Every particle moves one cell along z, all from cells 0 .. 6 of a row.
    keep = (np.floor(pos[:, 2]).astype(int) & 7) < 7
    pos, tag = pos[keep], tag[keep]
    step = np.zeros_like(pos)
    step[:, 2] = 1.0
    moved = pos + step
    order = np.lexsort((np.arange(len(pos)), _cell_keys(pos), _cell_keys(moved)))
    with _sim() as sim:
        out = [np.empty_like(pos) for _ in range(3)]
        sim.step_host(1.0, fsim.pcg_params(fsim.PCG_FIXED, fsim.PREC_FP32, 1), pos, tag, step,
                      out=out)
        assert np.array_equal(out[0], moved[order])


@pytest.mark.parametrize("case", ["two", "three", "many"])
def test_time(case):
    """A leaf at its limit in a few cells, against the same number of rows with
    24 in every cell: a cell of m rows ordered by m log^2 m operations takes
    (1 + log2 12,288)^2 / 2 or about 110 passes over its rows at the most,
    which are a few times the other phases; m^2 of them take hundreds."""
    rng = np.random.default_rng(12)
    us = {}
    for name, counts in (("even", [24] * 512), (case, CASES[case])):
        pos = _rows(counts, rng)
        zero = np.zeros_like(pos)
        with _sim() as sim:
            sim.upload_particles(pos, zero, zero)  # first launches
            sim.set_profiling(True)
            best = []
            for _ in range(5):
                sim.reset_kernel_times()
                sim.upload_particles(pos, zero, zero)
                best.append(sim.kernel_times()["sort_leaves"][0])
            us[name] = min(best)
    assert us[case] <= 8 * us["even"], us
