"""A launch that the device refuses (no room for the CTAs of a cluster) leaves the system to the next
kernel: Jacobi-PCG falls from the register kernel to the 16-CTA cluster and from that to the grid.  The
refusal comes from a stand-in for cudaLaunchKernelExC in a child process."""
import json
import os
import shutil
import subprocess
import sys

import pytest
from test_gpu_jacobi_sizes import ladder, solve

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
#include <cstdlib>
extern "C" int cudaLaunchKernelExC(const unsigned* config, const void* f, void** args) {  // config: gridDim.x first
    if (config[0] <= (unsigned)atoi(getenv("REFUSE_CTAS"))) return 701;                    // cudaErrorLaunchOutOfResources
    static auto real = (int (*)(const unsigned*, const void*, void**))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaLaunchKernelExC");
    return real(config, f, args);
}
"""
CHILD = """
import json, sys
from test_gpu_jacobi_sizes import ladder, solve
cfg, net = ladder(int(sys.argv[1]))
solves, r, _ = solve(net, cfg, True)
print(json.dumps([solves, r]))
"""


@pytest.mark.parametrize("rungs", [100, 900])  # one CTA, a cluster of four
@pytest.mark.parametrize("refused,kernel", [(8, 1), (16, 0)])
def test_refused_launch(cuda_ok, tmp_path, rungs, refused, kernel):
    (tmp_path / "shim.cpp").write_text(SHIM)
    lib = str(tmp_path / "shim.so")
    subprocess.run([shutil.which("g++") or "c++", "-shared", "-fPIC", "-O1", str(tmp_path / "shim.cpp"), "-o", lib, "-ldl"], check=True)
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, LD_PRELOAD=lib, REFUSE_CTAS=str(refused), PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    out = subprocess.run([sys.executable, "-c", CHILD, str(rungs)], env=env, check=True, capture_output=True, text=True, timeout=300).stdout
    solves, r = json.loads(out.strip().splitlines()[-1])
    cfg, net = ladder(rungs)
    general, r_general, _ = solve(net, cfg, False)
    assert [s[2] for s in solves] == [kernel] * len(solves) and [s[0] for s in solves] == [s[0] for s in general]
    assert all(s[1] <= 1e-10 for s in solves) and abs(r - r_general) <= 1e-9 * r_general
