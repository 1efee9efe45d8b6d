"""Refused launches and failed solves are told apart.  A child process whose
CUDA runtime calls go through a small C library that can refuse a launch, or
report an error from a stream synchronisation, without touching the GPU:

- a refused on-chip launch falls to the next loop, and only the refused kernel
  is out for the handle: other precisions and sizes keep theirs;
- an error after the launch is the solve's error, not a refusal: no other loop
  runs on the vectors of the failed one, and the next solve is as before."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
typedef struct { unsigned x, y, z; } dim;
int refuse_cooperative, refuse_cluster, fail_sync;  /* calls left to refuse or fail */
static void* real(const char* n) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), n); }
int cudaLaunchCooperativeKernel(const void* f, dim g, dim b, void** a, size_t m, void* s) {
  if (refuse_cooperative > 0 && refuse_cooperative--) return 720; /* too large */
  return ((int (*)(const void*, dim, dim, void**, size_t, void*))real(
      "cudaLaunchCooperativeKernel"))(f, g, b, a, m, s);
}
int cudaLaunchKernelExC(const void* c, const void* f, void** a) {
  if (refuse_cluster > 0 && refuse_cluster--) return 912; /* no such cluster */
  return ((int (*)(const void*, const void*, void**))real("cudaLaunchKernelExC"))(c, f, a);
}
int cudaStreamSynchronize(void* s) {
  const int e = ((int (*)(void*))real("cudaStreamSynchronize"))(s);
  if (fail_sync > 0 && fail_sync--) return 999; /* unknown */
  return e;
}
"""

CHILD = r"""
import ctypes, json, sys
shim = ctypes.CDLL(sys.argv[1], ctypes.RTLD_GLOBAL)
sys.path[:0] = sys.argv[2:5]
import numpy as np
import fsim
from test_gpu_pcg_cluster import _first_leaves, _system

FP32, MIXED, FP64 = fsim.PREC_FP32, fsim.PREC_MIXED, fsim.PREC_FP64


def arm(name, n):
    ctypes.c_int.in_dll(shim, name).value = n


def left(name):
    return ctypes.c_int.in_dll(shim, name).value


def solve(sim, prec, shim_arg=None):
    prm = fsim.pcg_params(fsim.PCG_RELATIVE, prec, 2000, tolerance=1e-5)
    sim.set_profiling(True)
    sim.reset_kernel_times()
    if shim_arg:
        arm(shim_arg, 1)
    try:
        st = sim.pcg_solve(prm)
        got = [st.status, st.iterations, st.rr]
    except fsim.FsimError as e:
        got = ["error", e.code]
    # the last loop tried (a refused launch has its name in the times too)
    names = [k for k in sim.kernel_times() if k.startswith("pcg")]
    loop = ["spmv"] if any("spmv" in k and "cluster" not in k for k in names) else []
    loop += [q for q in ("resident_f64", "resident_mixed", "resident", "cluster")
             if any(q in k for k in names)]
    sim.set_profiling(False)
    return (loop or ["none"])[0], got, sim.field(fsim.FIELD_PRESSURE)[0]


dims = (77, 80, 51)
small, large = (_system(dims, _first_leaves(dims, n), seed=n) for n in (40, 700))
out = {}
ref = {}
for name, make in (("small", small), ("large", large)):
    sim = make()
    for prec in (FP32, MIXED, FP64):
        ref[name, prec] = solve(sim, prec)
    sim.close()
    out[name] = [ref[name, p][0] for p in (FP32, MIXED, FP64)]

# one refused FP64 launch: that solve by the pair, every other loop stays
for name, make in (("small", small), ("large", large)):
    sim = make()
    out[name + "_refused"] = [solve(sim, FP64, "refuse_cooperative")[0],
                              *(solve(sim, p)[0] for p in (FP64, FP32, MIXED))]
    assert left("refuse_cooperative") == 0
    sim.close()
# a refused cluster: the resident loop
sim = small()
out["cluster_refused"] = [solve(sim, FP32, "refuse_cluster")[0], solve(sim, FP32)[0], solve(sim, MIXED)[0]]
sim.close()
# an error after the launch
for name, make, prec in (("small", small, FP32), ("large", large, FP32), ("large", large, FP64)):
    sim = make()
    failed = solve(sim, prec, "fail_sync")
    assert left("fail_sync") == 0
    again = solve(sim, prec)
    want = ref[name, prec]
    out["failed_%s_%d" % (name, prec)] = [failed[1], again[0] == want[0], again[1] == want[1],
                                          bool(np.array_equal(again[2], want[2]))]
    sim.close()
print(json.dumps(out))
"""


def test_refusals_and_failures(tmp_path):
    here = Path(__file__).resolve().parent
    (tmp_path / "shim.c").write_text(SHIM)
    shim = tmp_path / "shim.so"
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(shim), str(tmp_path / "shim.c"),
                    "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(shim), str(here),
                        str(here.parent / "fluid-sim-lb_gb300"), str(here.parent)],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    got = json.loads(r.stdout.splitlines()[-1])
    assert got["small"] == ["cluster", "cluster", "resident_f64"]
    assert got["large"] == ["resident", "resident_mixed", "resident_f64"]
    assert got["small_refused"] == ["spmv", "spmv", "cluster", "cluster"]
    assert got["large_refused"] == ["spmv", "spmv", "resident", "resident_mixed"]
    assert got["cluster_refused"] == ["resident", "resident", "cluster"]
    for case in ("failed_small_0", "failed_large_0", "failed_large_2"):
        assert got[case] == [["error", 2], True, True, True], case
