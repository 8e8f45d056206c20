"""The streaming product takes and refuses the same pairs of prologue and epilogue whatever K, and so whatever kernel, it would run.
The launcher is linked against a fake of the CUDA runtime, so a call that is taken wrongly launches nothing."""
import ctypes
import subprocess
from pathlib import Path

import pytest
import torch

from inf_engine_b200 import kernels
from inf_engine_b200.csrc.build import SRC_DIR, find_nvcc
from test_several_devices import FAKE

P, I, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
A = 4096      # an address that nobody reads
PLAIN, NORM, PRENORMED = 0, 1, 2
BF16, F32, RESIDUAL, SILU_MUL, RESIDUAL_NORMOUT, RELU2, GLU = range(7)
TAKEN = {PLAIN: {BF16, F32, RESIDUAL, SILU_MUL, RESIDUAL_NORMOUT, RELU2, GLU}, NORM: {BF16, F32, SILU_MUL}, PRENORMED: {BF16, F32, SILU_MUL}}
BAD_DTYPE = -1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("stream")
    nvcc = find_nvcc()
    (d / "fake.cpp").write_text(FAKE)

    def run(*cmd):
        r = subprocess.run(list(map(str, cmd)), capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-2000:]

    # the host side is what is looked at: device code stays unoptimised and unassembled
    run(nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-Xcompiler", "-fPIC",
        "--expt-relaxed-constexpr", f"-I{SRC_DIR}", "-c", SRC_DIR / "gemm_stream_tma.cu", "-o", d / "stream.o")
    run("g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", Path(nvcc).resolve().parent.parent / "include", d / "fake.cpp",
        d / "stream.o", "-o", d / "stream.so")
    lib = ctypes.CDLL(str(d / "stream.so"))
    lib.ie_gemm_stream_tma.argtypes = [P, P, P, P, I, P, I, I, I, I, I, I, F, I, I, I, P, I, P, I, P, I, F, F, F, F, P]
    return lib


def call(lib, m, n, k, pro, epi):
    """Status of the call, and whether it launched; every buffer that a pair could ask for is given."""
    before = lib.fake_launches()
    rc = lib.ie_gemm_stream_tma(A, A, A, A, 0, None, m, n, k, k, k, n, 1e-5, pro, epi, 148, A, n, A, 0, A, 148, 1.0, 0.0, 0.0, 0.0, None)
    return rc, lib.fake_launches() - before


# bulk copies: 512, 2,304, 5,120; rings of warps: 1,024, 2,048, 3,072, 4,096; units of 8 and of 16 rows
@pytest.mark.parametrize("K", [512, 1024, 2048, 2304, 3072, 4096, 5120])
@pytest.mark.parametrize("M,N", [(1, 520), (8, 9600), (9, 520), (16, 9600)])
def test_pairs_do_not_depend_on_the_kernel(lib, M, N, K):
    fits = (16 if M > 8 else 8) * (2 * K + 64) <= 100 * 1024      # a norm in the prologue wants its rows in shared memory
    for pro in (PLAIN, NORM, PRENORMED, 3, -1):
        for epi in (*range(7), 7, 9, -1):
            rc, launched = call(lib, M, N, K, pro, epi)
            if epi in TAKEN.get(pro, ()) and (pro == PLAIN or fits):
                assert (rc, launched) == (0, 1), (pro, epi)
            else:
                assert rc < 0 and launched == 0, (pro, epi)
                assert rc == BAD_DTYPE or (pro != PLAIN and not fits), (pro, epi)


def test_one_product_does_not_take_a_norm_and_hand_one_over():
    """Rows and sums of a norm that is taken are read while those of the next are written; each pair of buffers is named once."""

    class Lib:
        def ie_gemm_stream_tma_supports(self, *a):
            return 1

    x, w, c = torch.zeros(4, 2048, dtype=torch.bfloat16), torch.zeros(2048, 2048, dtype=torch.bfloat16), torch.zeros(4, 2048)
    xg, xg2, ssq, ssq2 = x.clone(), x.clone(), torch.zeros(16, 148), torch.zeros(16, 148)
    gain = torch.ones(2048, dtype=torch.bfloat16)
    for other in ((xg, gain, ssq), (xg2, gain, ssq2)):
        with pytest.raises(kernels.KernelError, match="prenormed and normout"):
            kernels.gemm_stream(x, w, c, 4, "residual", eps=1e-5, prenormed=(xg, ssq), normout=other, lib=Lib())
