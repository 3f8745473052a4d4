"""What a one-launch solve needs from the runtime, and what is done without it.

A device that refuses the launch of a one-launch solve (blocks that do not fit
together: a share of the SMs, other work in the way): the call goes on with its
separate launches. The refusal comes from a stand-in for the runtime's launch
calls, preloaded into a child process, that returns
cudaErrorCooperativeLaunchTooLarge for every cooperative or cluster launch.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <cstdio>
static int refused = 0;
extern "C" cudaError_t cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  ++refused;
  return cudaErrorCooperativeLaunchTooLarge;
}
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* f, void** args) {
  for (unsigned i = 0; i < cfg->numAttrs; ++i)
    if (cfg->attrs[i].id == cudaLaunchAttributeCooperative || cfg->attrs[i].id == cudaLaunchAttributeClusterDimension) {
      ++refused;
      return cudaErrorCooperativeLaunchTooLarge;
    }
  using Fn = cudaError_t (*)(const cudaLaunchConfig_t*, const void*, void**);
  static Fn real = (Fn)dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
  return real(cfg, f, args);
}
extern "C" int refused_launches() { return refused; }
"""

CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1] + "/tests")
sys.path.insert(0, sys.argv[1])
from test_gpu_csc_resident import _ctx, _laplacian
from test_gpu_resident_solve import _solve, _world
out = {}
A = _laplacian((9, 10, 11), 0.05)
b = np.random.default_rng(4).uniform(-1, 1, A.shape[0])
with _ctx() as ctx:
    out["csc"] = ctx.csc_solve(A.indptr, A.indices, A.data, b)
for n in (17, 63):  # one cluster, the grid
    got, st, launched = _solve(_world(n, 0.5), "mgpcg64", False)
    out["p%d" % n] = got.f64["p"] * got.exists
    out["launches%d" % n] = launched
try:
    out["refused"] = ctypes.CDLL(None).refused_launches()
except AttributeError:
    out["refused"] = 0
np.savez(sys.argv[2], **out)
"""


def _child(tmp_path, name, env):
    out = str(tmp_path / (name + ".npz"))
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, out], env=dict(os.environ, **env), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(out)


def test_refused_launches_take_the_separate_ones(tmp_path):
    from mac_b200.gpu import load
    load()
    cudart = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l)
    src, so = tmp_path / "refuse.cpp", str(tmp_path / "refuse.so")
    src.write_text(FAKE)
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", "-o", so, str(src),
                    "-Wl,--no-as-needed", cudart, "-Wl,-rpath," + os.path.dirname(cudart), "-ldl"], check=True)
    plain = _child(tmp_path, "plain", {})
    refused = _child(tmp_path, "refused", {"LD_PRELOAD": so})
    assert plain["refused"] == 0 and refused["refused"] >= 3
    for k in ("csc", "p17", "p63"):  # both solved to 1e-12
        assert np.linalg.norm(plain[k] - refused[k]) <= 1e-8 * np.linalg.norm(plain[k]), k
    for n in (17, 63):
        assert refused["launches%d" % n] > plain["launches%d" % n]


RESET = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1] + "/tests")
sys.path.insert(0, sys.argv[1])
from test_gpu_resident_solve import _solve, _world
s = _world(63, 0.5)
a, sa, la = _solve(s, "mgpcg64", False)
cudart = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l)
assert ctypes.CDLL(cudart).cudaDeviceReset() == 0
b, sb, lb = _solve(s, "mgpcg64", False)
assert (la, sa["iterations"]) == (lb, sb["iterations"]), (la, lb)
assert np.array_equal(a.f64["p"], b.f64["p"])
"""


def test_device_reset_by_the_host_program():
    """The kernel's shared memory and cluster size are allowed again for a context
    made after the reset: the solve is one launch as before."""
    r = subprocess.run([sys.executable, "-c", RESET, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
