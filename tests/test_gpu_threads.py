"""Handles used from several threads do not disturb one another's launches."""
import threading

import numpy as np
import pytest

import fsim
from test_gpu_pcg_cluster import _system

pytestmark = pytest.mark.gpu


def test_resident_sizes_side_by_side(monkeypatch):
    """Two threads solve systems of 9 and of 16 leaves per SM, which take the
    same kernel with different amounts of shared memory: no launch is refused
    (a refused one would leave its handle on the pair), and every solve gives
    the bits of a solve alone."""
    import torch

    monkeypatch.delenv("FSIM_PCG_RES", raising=False)
    monkeypatch.delenv("FSIM_PCG_CG1", raising=False)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    dims = (128, 128, 88)
    fill = np.zeros(dims, bool)
    sims, want = [], []
    prm = fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_FP32, 50, tolerance=1e-4)
    for per in (9, 16):
        n = per * sms - 40
        lv = [d // 8 for d in dims]
        on = np.zeros(lv, bool)
        on.reshape(-1)[:n] = True
        fill = on.repeat(8, 0).repeat(8, 1).repeat(8, 2)
        x, y, z = np.indices(dims) & 7
        fill &= (x >= 3) & (x < 5) & (y >= 3) & (y < 5) & (z >= 3) & (z < 5)
        sim = _system(dims, fill, seed=per)()
        assert sim.leaves().shape[0] == n
        st = sim.pcg_solve(prm)
        want.append((st.iterations, st.rr, sim.field(fsim.FIELD_PRESSURE)[0]))
        sims.append(sim)
    bad = []

    def work(i):
        for _ in range(600):
            st = sims[i].pcg_solve(prm)
            if (st.iterations, st.rr) != want[i][:2]:
                bad.append((i, st.iterations, st.rr))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:3]
    for sim, w in zip(sims, want):
        assert np.array_equal(sim.field(fsim.FIELD_PRESSURE)[0], w[2])
        sim.set_profiling(True)
        sim.reset_kernel_times()
        sim.pcg_solve(prm)
        assert "pcg_resident" in sim.kernel_times()
        sim.close()
