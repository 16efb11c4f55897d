"""Small kernels for tests, compiled with the library's device headers as its run-time model
code is (csrc/jit.cpp: NVRTC, the same options)."""
import ctypes as C
import os
import re

import pytest

from inchman_b200 import build


def compile_cubin(src):
    nvrtc = pytest.importorskip("cuda.bindings.nvrtc")
    jit = open(os.path.join(build.CSRC, "jit.cpp")).read()
    prelude = re.search(r'kPrelude = R"GPGMPJIT\((.*?)\)GPGMPJIT"', jit, re.S).group(1)
    names = [n.encode() for n, _ in build.JIT_HEADERS] + [b"gpgmp_rtc_prelude.h"]
    texts = [open(p, "rb").read() for _, p in build.JIT_HEADERS] + [prelude.encode()]
    opts = [b"-arch=sm_100a", b"-fmad=false", b"-std=c++17", b"-default-device", b"-DGPGMP_JIT"]
    err, prog = nvrtc.nvrtcCreateProgram(src.encode(), b"test.cu", len(names), texts, names)
    assert err == nvrtc.nvrtcResult.NVRTC_SUCCESS
    (rc,) = nvrtc.nvrtcCompileProgram(prog, len(opts), opts)
    _, n = nvrtc.nvrtcGetProgramLogSize(prog)
    log = b" " * n
    nvrtc.nvrtcGetProgramLog(prog, log)
    assert rc == nvrtc.nvrtcResult.NVRTC_SUCCESS, log.decode(errors="replace")
    _, n = nvrtc.nvrtcGetCUBINSize(prog)
    cubin = b" " * n
    nvrtc.nvrtcGetCUBIN(prog, cubin)
    nvrtc.nvrtcDestroyProgram(prog)
    return cubin


class Kernels:
    def __init__(self, src):
        import torch
        drv = pytest.importorskip("cuda.bindings.driver")
        cubin = compile_cubin(src)
        torch.zeros(1, device="cuda")      # the primary context
        self.drv = drv
        err, self.mod = drv.cuModuleLoadData(cubin)
        assert err == drv.CUresult.CUDA_SUCCESS

    def launch(self, name, blocks, threads, *args, smem=0, stream=None):
        """args: tensors (their pointers) and integers (32 bits)."""
        import torch
        drv = self.drv
        err, fn = drv.cuModuleGetFunction(self.mod, name.encode())
        assert err == drv.CUresult.CUDA_SUCCESS
        if smem > 48 * 1024:
            (err,) = drv.cuFuncSetAttribute(
                fn, drv.CUfunction_attribute.CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, smem)
            assert err == drv.CUresult.CUDA_SUCCESS
        values = tuple(a if isinstance(a, int) else a.data_ptr() for a in args)
        kinds = tuple(C.c_int if isinstance(a, int) else C.c_void_p for a in args)
        st = (stream or torch.cuda.current_stream()).cuda_stream
        (err,) = drv.cuLaunchKernel(fn, blocks, 1, 1, threads, 1, 1, smem, st, (values, kinds), 0)
        assert err == drv.CUresult.CUDA_SUCCESS

    def close(self):
        self.drv.cuModuleUnload(self.mod)
