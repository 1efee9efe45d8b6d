"""The rebinning's stable sort by leaf bins: the order is that of a stable sort
by cell, whatever the upload's order, and a state with a leaf too full for the
per-leaf sort (12,288 particles) takes the library's sort to the same order."""
import numpy as np
import pytest

import fsim

pytestmark = pytest.mark.gpu

N = 24


def _cell_keys(pos):
    """OpenVDB order of the cells of a domain inside one 64^3 block."""
    c = np.floor(pos).astype(np.int64)
    leaf = ((c[:, 0] >> 3) << 6) | ((c[:, 1] >> 3) << 3) | (c[:, 2] >> 3)
    return leaf * 512 + (((c[:, 0] & 7) << 6) | ((c[:, 1] & 7) << 3) | (c[:, 2] & 7))


def _positions(case, rng):
    if case == "one":
        return np.array([[3.5, 4.5, 5.5]])
    if case == "two_leaves":
        return rng.uniform(0.01, 15.99, (40, 3)) * np.array([1, 0.4, 0.4])
    if case == "even":  # every leaf a few thousand
        return rng.uniform(0.01, N - 0.01, (60000, 3))
    if case == "full_cells":  # cells at and around the single-thread length
        cells = np.repeat(np.arange(40), [47, 48, 49, 50, 200] * 8)
        base = np.stack([cells % 8, cells // 8, np.full(cells.size, 9)], 1)
        return base + rng.uniform(0.01, 0.99, (cells.size, 3))
    n = {"most": 12288, "over": 12289, "one_cell": 12288, "far_over": 40000}[case]
    hi = 0.98 if case == "one_cell" else 7.98
    return np.concatenate([8 + rng.uniform(0.01, hi, (n, 3)), rng.uniform(0.01, 7.9, (500, 3)),
                           16 + rng.uniform(0.01, 7.9, (1033, 3))])


@pytest.mark.parametrize("case", ["one", "two_leaves", "even", "full_cells", "most", "over",
                                  "one_cell", "far_over"])
@pytest.mark.parametrize("ordered", [False, True])
def test_order_is_a_stable_sort(case, ordered):
    rng = np.random.default_rng(5)
    pos = _positions(case, rng).astype(np.float32)
    pos = pos[rng.permutation(len(pos))]
    if ordered:
        pos = pos[np.argsort(_cell_keys(pos), kind="stable")]
    tag = np.arange(3 * len(pos), dtype=np.float32).reshape(-1, 3)
    zero = np.zeros_like(pos)
    g, f = fsim.physical_gravity(N)
    sim = fsim.Simulation((N, N, N), fsim.BOUNDARY_BOX, g, f)
    sim.upload_particles(pos, tag, zero)
    p, v, _ = sim.download_particles()
    want = np.argsort(_cell_keys(pos), kind="stable")
    assert np.array_equal(p, pos[want]) and np.array_equal(v, tag[want])
    # a move: old order first, then the new cells
    gvel = rng.normal(0, 1.0, pos.shape).astype(np.float32)
    sim.upload_particles(pos, tag, gvel)
    sim.move_particles(0.5)
    p, v, _ = sim.download_particles()
    moved = (pos + gvel * np.float32(0.5)).astype(np.float32)
    keep = np.all((moved >= 0) & (moved < N), axis=1)  # clamped rows may leave the fluid
    want = want[keep[want]]
    want = want[np.argsort(_cell_keys(moved[want]), kind="stable")]
    mine = np.isin(v[:, 0], tag[keep][:, 0])
    assert np.array_equal(v[mine], tag[want]) and np.array_equal(p[mine], moved[want])
    sim.close()


@pytest.mark.parametrize("case", ["two_leaves", "even", "full_cells", "most", "over"])
def test_step_on_unsorted_rows(case):
    """fsim_step_host on shuffled rows orders them by (new cell, old cell,
    row): as uploading, moving and rebinning in sequence."""
    rng = np.random.default_rng(6)
    pos = _positions(case, rng).astype(np.float32)
    pos = pos[rng.permutation(len(pos))]
    vel = rng.normal(0, 0.5, pos.shape).astype(np.float32)
    g, f = fsim.physical_gravity(N)
    out = []
    for whole in (True, False):
        sim = fsim.Simulation((N, N, N), fsim.BOUNDARY_BOX, g, f)
        prm = sim.default_pcg_params()
        if whole:
            buf = [np.empty_like(pos) for _ in range(3)]
            st, n = sim.step_host(0.01, prm, pos, vel, vel, out=buf)
            out.append([b[:n] for b in buf])
        else:
            sim.upload_particles(pos, vel, vel)
            sim.step(0.01, prm)
            out.append(sim.download_particles())
        sim.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
