"""The resident loop's kernels for fp32 vectors, around the sizes where one
takes over from another: up to eight leaves per SM a warp holds one half leaf
in registers, up to sixteen two (MIXED from eleven on), above that up to four
in tensor and shared memory.  Fixed
iteration counts against the spmv / update pair, whose element-wise operations
are the same; only the order of the dot products' sums differs."""
import numpy as np
import pytest

import fsim
from _util import rel_l2
from test_gpu_pcg_cluster import _first_leaves, _system

pytestmark = pytest.mark.gpu


# leaves per SM on 152 SMs: 2, 8 (one CTA short of a leaf, then all full), 9, 10,
# 11, 14, 15, 16, 17
@pytest.mark.parametrize("n", [300, 1215, 1216, 1217, 1520, 1521, 2128, 2200, 2432, 2433])
@pytest.mark.parametrize("prec", [fsim.PREC_FP32, fsim.PREC_MIXED])
def test_tracks_the_pair(monkeypatch, n, prec):
    dims = (125, 120, 88)
    make = _system(dims, _first_leaves(dims, n), seed=n)
    got = {}
    for res in ("1", "0"):
        with monkeypatch.context() as m:
            m.setenv("FSIM_PCG_RES", res)
            m.setenv("FSIM_PCG_CG1", "0")
            sim = make()
        assert sim.leaves().shape[0] >= n
        for it in (1, 12):
            prm = (fsim.pcg_params(fsim.PCG_FIXED, prec, it) if prec == fsim.PREC_FP32 else
                   fsim.pcg_params(fsim.PCG_RELATIVE, prec, it, tolerance=1e-14,
                                   inner_tolerance=1e-14, max_refinements=1))
            sim.set_profiling(True)
            sim.reset_kernel_times()
            st = sim.pcg_solve(prm)
            assert any("resident" in k for k in sim.kernel_times()) == (res == "1")
            sim.set_profiling(False)
            assert st.iterations == it
            got[res, it] = (st.rr, sim.field(fsim.FIELD_PRESSURE)[0])
        sim.close()
    for it in (1, 12):
        (rr, x), (rr0, x0) = got["1", it], got["0", it]
        assert rel_l2(x, x0) <= 1e-5 and abs(rr - rr0) <= 1e-3 * rr0, it
