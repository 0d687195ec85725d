"""The shape search of a shadow map looks at the kernel that a map of its size runs: a trajectory a
lane (ucb_lle_split_kernel) while few cells leave schedulers idle, else the pair form; each has
its own shapes. A build prepared at one size still serves every other."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import ucb
from helpers import engine_request, lle2d_case

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

REGISTERS = """
import sys
sys.path.insert(0, {pkg!r}); sys.path.insert(0, {tests!r})
import ucb
from helpers import engine_request, lle2d_case
block, regs, unroll = map(int, sys.argv[1:])
ucb.precompile(engine_request(ucb, lle2d_case(n=8, t_max=1.0, transient=1.0), precision=ucb.PREC_F64,
                              mode=ucb.MODE_NATIVE, block_threads=block, max_registers=regs, unroll=unroll))
"""


def compiled_registers(rep, cache):
    """Registers of both kernels of the build in the reported shape, of a file compiled for it alone."""
    code = REGISTERS.format(pkg=str(ROOT / "u-cuda_b200"), tests=str(ROOT / "tests"))
    env = dict(os.environ, UCB_CUBIN_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", code, *(str(rep[k]) for k in ("block_threads", "max_registers", "unroll"))],
                       env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    (cubin,) = cache.iterdir()
    cuda = C.CDLL("libcuda.so.1")  # (the engine's context is current)
    module, function, value, out = C.c_void_p(), C.c_void_p(), C.c_int(), {}
    assert cuda.cuModuleLoad(C.byref(module), str(cubin).encode()) == 0
    for name in ("ucb_lle_kernel", "ucb_lle_split_kernel"):
        assert cuda.cuModuleGetFunction(C.byref(function), module, name.encode()) == 0
        assert cuda.cuFuncGetAttribute(C.byref(value), 4, function) == 0  # CU_FUNC_ATTRIBUTE_NUM_REGS
        out[name] = value.value
    assert cuda.cuModuleUnload(module) == 0
    return out


def test_each_form_is_tuned_by_its_own_kernel(tmp_path, monkeypatch):
    monkeypatch.setenv("UCB_TUNE_TABLE", str(tmp_path / "tuned.tsv"))
    eng = ucb.Engine(0)
    reps = {}
    for n, kernel in ((40, "ucb_lle_split_kernel"), (120, "ucb_lle_kernel")):
        req = engine_request(ucb, lle2d_case(n=n, t_max=2.0, transient=1.0), precision=ucb.PREC_F64,
                             mode=ucb.MODE_NATIVE)
        reps[kernel] = rep = eng.autotune(req, force=True)
        regs = compiled_registers(rep, tmp_path / kernel)
        assert rep["registers"] == regs[kernel], (rep, regs)
    assert reps["ucb_lle_kernel"]["key"] != reps["ucb_lle_split_kernel"]["key"]
    eng.close()


@pytest.mark.parametrize("prepared,called", [(40, 120), (120, 40)])
def test_a_prepared_build_serves_both_forms(prepared, called):
    import torch
    eng = ucb.Engine(0)

    def request(n):
        return engine_request(ucb, lle2d_case(n=n, t_max=2.0, transient=1.0), precision=ucb.PREC_F64,
                              mode=ucb.MODE_NATIVE)

    ref, rflags, _ = eng.run_lle2d(request(called))
    eng.prepare_lle2d(request(prepared))
    v = torch.empty(called ** 2, dtype=torch.float64, device="cuda")
    f = torch.empty(called ** 2, dtype=torch.int32, device="cuda")
    eng.lle2d_device_noalloc(request(called), v.data_ptr(), f.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(v.cpu().numpy(), ref)
    np.testing.assert_array_equal(f.cpu().numpy(), rflags)
    eng.close()
