"""The decode attention for heads of 64 finds room beside a block of the streaming product ahead of it, and two blocks of one product do
not share an SM.  The launchers are linked against a fake of the CUDA runtime that notes the dynamic shared memory they ask for."""
import ctypes
import subprocess
from pathlib import Path

import pytest

from inf_engine_b200.csrc.build import SRC_DIR, find_nvcc
from test_several_devices import FAKE

P, I, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
A = 4096                     # an address that nobody reads
SM_BYTES = 228 * 1024        # shared memory of an SM; a block takes 1 KB beside its own
BLOCK = 1024


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("share")
    nvcc = find_nvcc()
    fake = FAKE.replace("  ++g_launches;\n", "  ++g_launches;\n  g_smem = (int)c->dynamicSmemBytes;\n")
    fake = fake.replace("static int g_device = 0,", """static int g_smem = 0;
extern "C" int fake_smem() { return g_smem; }
static int g_device = 0,""")
    assert fake.count("g_smem") == 3
    (d / "fake.cpp").write_text(fake)

    def run(*cmd):
        r = subprocess.run(list(map(str, cmd)), capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-2000:]

    for name in ("gemm_stream_tma", "attention_mma"):
        run(nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-Xcompiler", "-fPIC",
            "--expt-relaxed-constexpr", "-DIE_HD=64", f"-I{SRC_DIR}", "-c", SRC_DIR / f"{name}.cu", "-o", d / f"{name}.o")
    run("g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", Path(nvcc).resolve().parent.parent / "include", d / "fake.cpp",
        d / "gemm_stream_tma.o", d / "attention_mma.o", "-o", d / "share.so")
    lib = ctypes.CDLL(str(d / "share.so"))
    lib.ie_gemm_stream_tma.argtypes = [P, P, P, P, I, P, I, I, I, I, I, I, F, I, I, I, P, I, P, I, P, I, F, F, F, F, P]
    lib.ie_attention_decode.argtypes = [P] * 8 + [I] * 10 + [F, I, I, P]
    return lib


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("K", [1024, 2048, 3072])
@pytest.mark.parametrize("N", [3072, 16384])
def test_decode_attention_beside_a_product(lib, M, N, K):
    assert lib.ie_attention_decode(*[A] * 8, 512, 512, 4, 2, 2, 8, 2, 64, 16, 0, 0.1, 6, 32, None) == 0
    attention = lib.fake_smem() + 512 + BLOCK                     # the rotation's tables are static
    assert lib.ie_gemm_stream_tma(A, A, A, None, 0, None, M, N, K, K, K, N, 0.0, 0, 0, 148, None, 0, None, 0, None, 0, 1.0, 0.0, 0.0, 0.0, None) == 0
    sums = (16 if N >= 16 * 4 * 148 else 8) * 1024 + 64           # two buffers of eight warps' sums and the 1/rms, static
    product = lib.fake_smem() + sums + BLOCK
    assert attention + product <= SM_BYTES < 2 * product
