"""Launchers that raise a kernel's limit of dynamic shared memory do so on every device that they launch on.  The sources are
linked against a fake of the CUDA runtime that keeps the limits by device and refuses a launch above them, as the runtime does;
no GPU takes part."""
import ctypes
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

from inf_engine_b200.csrc.build import SRC_DIR, find_nvcc

FAKE = r"""
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <map>
#include <utility>
static int g_device = 0, g_launches = 0;
static std::map<std::pair<int, const void*>, int> g_limit;
extern "C" {
void fake_device(int d) { g_device = d; }
int fake_launches() { return g_launches; }
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int bytes) { g_limit[{g_device, f}] = bytes; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  const auto it = g_limit.find({g_device, f});
  if (c->dynamicSmemBytes > (it == g_limit.end() ? 48 * 1024 : (size_t)it->second)) return cudaErrorInvalidValue;
  ++g_launches;
  return cudaSuccess;
}
static CUresult fake_encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                            const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *f = (void*)fake_encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorUnknown; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaMemcpyFromSymbol(void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaErrorUnknown; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaErrorUnknown; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaErrorUnknown; }
char __cudaInitModule(void**) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* p; return &p; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
"""
SOURCES = ["gemm_simt", "gemm_f32", "attention_general", "gemm_stream_tma", "gated_delta", "gemm_tcgen05", "attention_tcgen05", "attention_mma"]
P, I, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_float


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("devices")
    nvcc = find_nvcc()
    (d / "fake.cpp").write_text(FAKE)

    def run(*cmd):
        r = subprocess.run(list(map(str, cmd)), capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-2000:]

    def compile_one(name):     # the host side is what is looked at: device code stays unoptimised and unassembled
        run(nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-Xcompiler", "-fPIC",
            "--expt-relaxed-constexpr", "-DIE_GD_DK=64", "-DIE_GD_DV=64", "-DIE_HD=128", f"-I{SRC_DIR}",
            "-c", SRC_DIR / f"{name}.cu", "-o", d / f"{name}.o")

    with ThreadPoolExecutor(8) as ex:
        list(ex.map(compile_one, SOURCES))
    run("g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", Path(nvcc).resolve().parent.parent / "include", d / "fake.cpp",
        *[d / f"{n}.o" for n in SOURCES], "-o", d / "devices.so")
    lib = ctypes.CDLL(str(d / "devices.so"))
    lib.ie_gemm_simt.argtypes = [P, I, P, I, P, I, I, I, I, I, I, I, P]
    lib.ie_attention_ordered_rows.argtypes = [P] * 7 + [I] * 11 + [F, I, P, I, P, I, P]
    lib.ie_moe_ring.argtypes = [P] * 5 + [I] * 10 + [F] * 4 + [P]
    lib.ie_gated_delta.argtypes = [P, P, P, I, I, P, P, I, P, I, P, P, P, I, P, P, I, P, P, I, I, I, I, I, F, F, I, I, P, I, I, P]
    lib.ie_gemm_stream_tma.argtypes = [P, P, P, P, I, P, I, I, I, I, I, I, F, I, I, I, P, I, P, I, P, I, F, F, F, F, P]
    lib.ie_gemm_tcgen05.argtypes = [P] * 3 + [I] * 9 + [P]
    lib.ie_attention_tcgen05.argtypes = [P] * 9 + [I] * 9 + [F] + [P] * 4
    lib.ie_attention_prefill.argtypes = [P] * 9 + [I] * 9 + [F, I, P]
    lib.ie_attention_decode.argtypes = [P] * 8 + [I] * 10 + [F, I, I, P]
    return lib


A = 4096      # addresses that nobody reads
CALLS = {
    "float32 product, few rows": lambda L: L.ie_gemm_simt(A, 0, A, 0, A, 0, 16, 32768, 2048, 2048, 2048, 32768, None),
    "float32 product, tiles": lambda L: L.ie_gemm_simt(A, 0, A, 0, A, 0, 300, 2048, 2048, 2048, 2048, 2048, None),
    "float32 attention": lambda L: L.ie_attention_ordered_rows(*[A] * 7, 512, 512, 4, 2, 2, 16, 8, 8, 64, 16, 0, 0.1, 0, None, 0, None, 64, None),
    "experts": lambda L: L.ie_moe_ring(*[A] * 5, 8, 1024, 512, 512, 1024, 2, 1, 0, 1, 148, 1.0, 0.0, 0.0, 0.0, None),
    "delta rule in chunks": lambda L: L.ie_gated_delta(A, A, A, 128, 128, A, A, 4, A, 128, A, A, A, 0, A, A, 128, A, A, 1, 2, 2, 64, 64,
                                                       1e-6, 1e-5, 1, 0, A, 300, 300, None),
    "streaming product, bulk copies": lambda L: L.ie_gemm_stream_tma(A, A, A, None, 0, None, 8, 520, 2304, 2304, 2304, 520, 0.0, 0, 0, 148, None, 0,
                                                                     None, 0, None, 0, 1.0, 0.0, 0.0, 0.0, None),
    "streaming product, rings of warps": lambda L: L.ie_gemm_stream_tma(A, A, A, None, 0, None, 8, 520, 2048, 2048, 2048, 520, 0.0, 0, 0, 148, None,
                                                                        0, None, 0, None, 0, 1.0, 0.0, 0.0, 0.0, None),
    "tcgen05 product": lambda L: L.ie_gemm_tcgen05(A, A, A, 256, 512, 256, 256, 256, 512, 0, 128, 148, None),
    "tcgen05 attention": lambda L: L.ie_attention_tcgen05(*[A] * 9, 512, 512, 4, 2, 8, 2, 64, 16, 8, 0.1, None, None, None, None),
    "prompt attention": lambda L: L.ie_attention_prefill(*[A] * 9, 1024, 1024, 4, 2, 8, 2, 128, 16, 0, 0.1, 64, None),
    "decode attention": lambda L: L.ie_attention_decode(*[A] * 8, 1024, 1024, 4, 2, 2, 8, 2, 128, 16, 0, 0.1, 6, 32, None),
}


@pytest.mark.parametrize("name", CALLS)
def test_a_second_device_is_set_up_as_the_first(lib, name):
    for device in (0, 1, 0, 3):
        lib.fake_device(device)
        before = lib.fake_launches()
        assert CALLS[name](lib) == 0, f"device {device}"
        assert lib.fake_launches() > before
