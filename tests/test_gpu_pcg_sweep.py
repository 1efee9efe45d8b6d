"""The pipelined pair on a system of two kinds of columns (all cells inside
the fluid, and not) around the leaf count above which the update sweeps
downwards: fixed iteration counts against the unpipelined kernels, which do
neither.  Only the order of the dot products' sums differs, so the bar is the
one fixed iterations hold against the oracle."""
import numpy as np
import pytest

import fsim
from _util import rel_l2
from test_gpu_pcg_cluster import _first_leaves, _system

pytestmark = pytest.mark.gpu


# 300: several half leaves for some warps only; 16,384 / 16,385: both sides of
# the line; 17,001: a ragged last round
@pytest.mark.parametrize("n", [300, 16384, 16385, 17001])
@pytest.mark.parametrize("prec", [fsim.PREC_FP32, fsim.PREC_MIXED])
def test_pipelined_kernels_track_the_plain_ones(monkeypatch, n, prec):
    dims = (256, 256, 136)
    rng = np.random.default_rng(n)
    fill = rng.random(dims) < 0.02
    fill[4::8, 4::8, 4::8] = True
    fill[:40, :44, :60] = True
    make = _system(dims, fill & _first_leaves(dims, n), seed=n)
    prm = (fsim.pcg_params(fsim.PCG_FIXED, prec, 25) if prec == fsim.PREC_FP32 else
           fsim.pcg_params(fsim.PCG_RELATIVE, prec, 25, tolerance=1e-14,
                           inner_tolerance=1e-14, max_refinements=1))
    got = {}
    for pipe in ("1", "0"):
        with monkeypatch.context() as m:
            m.setenv("FSIM_PCG_RES", "0")
            m.setenv("FSIM_PCG_CG1", "0")
            m.setenv("FSIM_PCG_PIPE", pipe)
            sim = make()
            st = sim.pcg_solve(prm)
            assert st.iterations == 25
            assert sim.leaves().shape[0] >= n
            got[pipe] = (st.rr, sim.field(fsim.FIELD_PRESSURE)[0])
            sim.close()
    assert rel_l2(got["1"][1], got["0"][1]) <= 1e-5
    assert abs(got["1"][0] - got["0"][0]) <= 1e-3 * got["0"][0]
