"""A bounded wait of the FP64 stage that gives up has to reach the caller of
every entry point that steps or copies out.  The stage is replaced, in a child
process, by one that does nothing but set the context's status word, on the
host or in stream order, as the kernel does."""
import pytest

import preload

pytestmark = pytest.mark.gpu

STAGE = '''
#include <cuda_runtime.h>
#include "dg_internal.hpp"
static int mode = 0;         // 0: no report, 1: at once, 2: in stream order
static int* word = nullptr;  // of the last stage
extern "C" void stage_mode(int m) { mode = m; }
extern "C" void land() { *(volatile int*)word = 1; }
static void set(void* w) { *(volatile int*)w = 1; }
namespace dgk {
cudaError_t launch_euler_fp64(int, const EulerArgs&, const OzPlan& plan, cudaStream_t s) {
    word = plan.h_status;
    if (mode == 1) set(word);
    return mode == 2 ? cudaLaunchHostFunc(s, set, word) : cudaSuccess;
}
}
'''

CALLS = '''
import ctypes, sys
import numpy as np
import torch
from hopefoam_gb300 import _lib as L, euler
from hopefoam_gb300.mesh import periodic_square

shim, lib = ctypes.CDLL(sys.argv[1]), L.lib()
m = periodic_square(4, 4, 10.0, 10.0, perturb=0.1, seed=1)
ctx = euler.EulerContext(m, 2)
other = euler.EulerContext(m, 3)
ops = euler.reference_operators(2)
q = euler.isentropic_vortex(*euler.node_coords(m, ops["r"], ops["s"]), x0=5.0, y0=5.0)
ops3 = euler.reference_operators(3)
other.upload(euler.isentropic_vortex(*euler.node_coords(m, ops3["r"], ops3["s"]), x0=5.0, y0=5.0))
ctx.upload(q)
dev = torch.zeros(q.size, dtype=torch.float64, device="cuda")
host = np.zeros(q.size)
p = ctypes.c_void_p(dev.data_ptr())
h, F, PREC = ctx.h, 0, L.DG_PREC_FP64
none = np.zeros(1)
assert lib.dg_set_boundary_kinds(h, None, None) == L.DG_OK  # the limiter, no boundary faces
steps = {
    "rhs": lambda: lib.dg_euler_rhs(h, F, PREC, L.dptr(host)),
    "rhs_device": lambda: lib.dg_euler_rhs_device(h, F, PREC, p),
    "forward_euler": lambda: lib.dg_forward_euler_stage(h, 1e-3, F, PREC),
    "lserk4": lambda: lib.dg_lserk4_step(h, 1e-3, 1, F, PREC),
    "ssprk2": lambda: lib.dg_ssprk2_step(h, 1e-3, 1, F, PREC),
    "limited_ssprk2": lambda: lib.dg_limited_ssprk2_step(h, 1e-3, L.dptr(none), F, PREC),
}
for name, call in steps.items():
    ctx.upload(q)
    shim.stage_mode(0)
    assert call() == L.DG_OK, name
    shim.stage_mode(1)
    assert call() == L.DG_ERR_TIMEOUT, name + ": report at once"
    shim.stage_mode(0)
    assert call() == L.DG_OK, name + ": reported once"
copies = {
    "download": lambda: lib.dg_download_state(h, L.dptr(host)),
    "download_device": lambda: lib.dg_download_state_device(h, p),
    "sync": lambda: lib.dg_sync(h),
    "cfl_dt": lambda: lib.dg_cfl_dt(h, 0.5, L.dptr(none)),
    "noalloc": lambda: lib.dg_euler_rhs_noalloc(h, p, p, F),
}
for name, call in {**copies, **steps}.items():  # landed after the call that queued the stage
    ctx.upload(q)
    shim.land()
    assert call() == L.DG_ERR_TIMEOUT, name + ": landed before"
    ctx.upload(q)
    assert call() == L.DG_OK, name
groups = (ctypes.c_void_p * 2)(other.h.value, ctx.h.value)
b = ctypes.c_void_p()
assert lib.dg_batch_create(groups, 2, ctypes.byref(b)) == L.DG_OK
for schedule in (0, 1):
    assert lib.dg_batch_set_schedule(b, schedule, PREC) == L.DG_OK
    shim.stage_mode(0)
    assert lib.dg_batch_run(b, 1e-3, 1, F, PREC, None) == L.DG_OK
    shim.stage_mode(2)
    assert lib.dg_batch_run(b, 2e-3, 1, F, PREC, None) == L.DG_ERR_TIMEOUT, "batch"
    lib.dg_sync(ctx.h)
    lib.dg_sync(other.h)
shim.stage_mode(2)
assert lib.dg_batch_tune(b, 1e-3, F, PREC, 1, None) == L.DG_ERR_TIMEOUT, "tune"
lib.dg_batch_destroy(b)
print("all reported")
'''


def test_every_call_reports_a_timeout_of_the_fp64_stage(gpu_lib, tmp_path):
    so = preload.compile_host(STAGE, tmp_path / "stage.so", "-L/usr/local/cuda/lib64", "-lcudart")
    assert "all reported" in preload.run(so, CALLS, so)
