"""Contexts in several threads at once, on networks whose multigrid hierarchies end in dense levels of
different sizes: the shared-memory limits that one thread sets have to hold for the others' launches, so
a kernel's limit is always set to the same value."""
import os
import shutil
import subprocess
import sys
import threading

import pytest
from test_gpu_jacobi_sizes import ladder

from cicy_geom_b200.device import Context

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
#include <map>
static std::map<const void*, int> limits;
static int changes = 0;
extern "C" int limit_changes() { return changes; }
extern "C" int cudaFuncSetAttribute(const void* f, int attr, int value) {
    if (attr == 8) changes += limits.emplace(f, value).first->second != value;  // cudaFuncAttributeMaxDynamicSharedMemorySize
    static auto real = (int (*)(const void*, int, int))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), "cudaFuncSetAttribute");
    return real(f, attr, value);
}
"""
CHILD = """
import ctypes, os
from cicy_geom_b200.device import Context
from test_gpu_jacobi_sizes import ladder
for rungs in (50, 60, 70, 150, 400, 1000):
    for pre, cluster in ((0, True), (3, True), (3, False)):
        cfg, net = ladder(rungs)
        with Context(0) as ctx:
            ctx.set_solver(preconditioner=pre, cluster=cluster)
            ctx.upload(net)
            ctx.network_to_conductance(cfg.params())
print("changes", ctypes.CDLL(os.environ["LD_PRELOAD"]).limit_changes())
"""


def test_limits_do_not_change(cuda_ok, tmp_path):
    (tmp_path / "shim.cpp").write_text(SHIM)
    lib = str(tmp_path / "shim.so")
    subprocess.run([shutil.which("g++") or "c++", "-shared", "-fPIC", "-O1", str(tmp_path / "shim.cpp"), "-o", lib, "-ldl"], check=True)
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    out = subprocess.run([sys.executable, "-c", CHILD], env=env, check=True, capture_output=True, text=True, timeout=300).stdout
    assert out.split()[-2:] == ["changes", "0"]


@pytest.mark.parametrize("cluster", [True, False])
def test_dense_levels_of_different_sizes(cuda_ok, cluster):
    sizes = [40, 48, 56, 64, 70, 74] if cluster else [50, 60, 70, 80, 90, 100]
    expected, got, errors = {}, {}, []

    def context(rungs):
        cfg, net = ladder(rungs)
        ctx = Context(0)
        ctx.set_solver(preconditioner=3, cluster=cluster)
        ctx.upload(net)
        return ctx, cfg.params()

    def work(rungs):
        try:
            ctx, p = context(rungs)
            got[rungs] = [list(ctx.network_to_conductance(p).resistances) for _ in range(60)]
            ctx.close()
        except Exception as e:  # reported by the main thread
            errors.append((rungs, str(e)))

    for rungs in sizes:
        ctx, p = context(rungs)
        expected[rungs] = list(ctx.network_to_conductance(p).resistances)
        ctx.close()
    threads = [threading.Thread(target=work, args=(r,)) for r in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(r == expected[k] for k in sizes for r in got[k])
