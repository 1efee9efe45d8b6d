"""What the on-chip loops share with the spmv / update pair bit for bit.  A MIXED
solve's vectors are the pair's operations on the same cells, and its alpha and
beta are fp32 roundings of quotients of totals that both hold to some 2^-44, so
the vectors are equal unless a quotient lies that close to a rounding boundary;
r.r is a sum of the same exact products in another order.  FP64 forms products
and sums in one rounding where the pair takes two."""
import numpy as np
import pytest

import fsim
from _util import rel_l2
from test_gpu_pcg_cluster import _first_leaves, _system
from test_gpu_pcg_resident_precisions import _fixed, _solve

pytestmark = pytest.mark.gpu

DIMS = (77, 80, 51)


def _arms(monkeypatch, make, run, other):
    """run(sim) on a handle that takes the on-chip loop (FSIM_PCG_RES = other,
    None: by size) and on one that takes the pair."""
    out = []
    monkeypatch.delenv("FSIM_PCG_CG1", raising=False)
    for res in (other, "0"):
        with monkeypatch.context() as m:
            m.delenv("FSIM_PCG_RES", raising=False)
            if res is not None:
                m.setenv("FSIM_PCG_RES", res)
            sim = make()
        out.append(run(sim))
        sim.close()
    return out


# the cluster; one and two half leaves per warp, the general kernel
@pytest.mark.parametrize("n,res", [(3, None), (45, None), (192, None), (2, "1"), (305, None),
                                   (700, None), (1700, None), (2600, None)])
def test_mixed_is_the_pair(monkeypatch, n, res):
    dims = DIMS if n <= 700 else (128, 128, 88)
    make = _system(dims, _first_leaves(dims, n), seed=n)

    def run(sim):
        got = []
        for it in (1, 2, 12):
            st, _ = _solve(sim, _fixed(fsim.PREC_MIXED, it))
            got.append((st.iterations, st.rr, sim.field(fsim.FIELD_PRESSURE)[0]))
        st, _ = _solve(sim, fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_MIXED, 4000,
                                            tolerance=1e-9, inner_tolerance=1e-3,
                                            max_refinements=30))
        got.append((st.iterations, st.rr, sim.field(fsim.FIELD_PRESSURE)[0]))
        return got

    for a, b in zip(*_arms(monkeypatch, make, run, res)):
        assert a[0] == b[0] and np.array_equal(a[2], b[2])
        assert abs(a[1] - b[1]) <= 1e-11 * b[1]


@pytest.mark.parametrize("n", [1, 152, 305, 700])
def test_fp64_sums(monkeypatch, n):
    """12 iterations of rounding errors of 2^-53 each, against the second word
    of the fixed-point sums (2^-40 of the first's units)."""
    make = _system(DIMS, _first_leaves(DIMS, n), seed=n)

    def run(sim):
        return [_solve(sim, _fixed(fsim.PREC_FP64, it))[0].rr for it in (1, 12)]

    a, b = _arms(monkeypatch, make, run, "1")
    for x, y in zip(a, b):
        assert abs(x - y) <= 1e-10 * y


def test_totals_through_memory(monkeypatch):
    """Isolated fluid cells converge in one iteration: r.r falls by far more
    than the words hold (2^7), so the barrier sums through memory.  MIXED's
    vectors being the pair's, its status, iterations and tiny totals are too."""
    n = 32
    fill = np.zeros((n, n, n), bool)
    fill[2::4, 2::4, 2::4] = True
    make = _system((n, n, n), fill, seed=3)

    def run(sim):
        st, _ = _solve(sim, fsim.pcg_params(fsim.PCG_RELATIVE, fsim.PREC_MIXED, 50,
                                            tolerance=1e-5))
        got = [(st.status, st.iterations, st.rr, sim.field(fsim.FIELD_PRESSURE)[0])]
        for it in (1, 2):
            st, _ = _solve(sim, _fixed(fsim.PREC_MIXED, it))
            got.append((st.status, st.iterations, st.rr, sim.field(fsim.FIELD_PRESSURE)[0]))
        return got, st.bb

    (a, bb), (b, _) = _arms(monkeypatch, make, run, "1")
    assert a[0][2] < 2.0 ** -30 * bb  # the drop of one iteration
    for x, y in zip(a, b):
        assert x[:2] == y[:2] and np.array_equal(x[3], y[3])
        assert abs(x[2] - y[2]) <= 1e-11 * y[2]
