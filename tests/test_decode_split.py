"""How a request's keys are cut in a decode attention launch: every key in one warp's part, the warps of its blocks evenly loaded,
and, where blocks wait for places on the SMs, no more blocks kept busy than the launch's own cut would keep."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parent.parent / "inf-engine_b200" / "csrc" / "decode_split.h"
SOURCE = """
#include "decode_split.h"
extern "C" void cut(int span, int launch_keys, int launch_blocks, int spread, int warps, int tile, int* out) {
  out[0] = decode_split_keys(span, launch_keys, launch_blocks, spread != 0, warps, tile);
  out[1] = decode_split_blocks(span, out[0], warps);
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "split.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", f"-I{HEADER.parent}", str(d / "split.cpp"), "-o", str(d / "split.so")], check=True)
    lib = ctypes.CDLL(str(d / "split.so"))

    def call(*args):
        out = (ctypes.c_int * 2)()
        lib.cut(*args, out)
        return out[0], out[1]

    return call


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("warps,tile", [(6, 32), (6, 16)])
@pytest.mark.parametrize("launch_keys,launch_blocks", [(64, 1), (512, 1), (32, 1), (64, 3), (512, 2), (96, 8), (320, 64)])
def test_cut(cut, spread, warps, tile, launch_keys, launch_blocks):
    longest = launch_keys * launch_blocks * warps
    for span in sorted({1, 2, 31, 32, 33, 63, 64, 65, longest // 7 + 1, longest // 3, longest // 2 + 1, longest - 1, longest, longest + 5000,
                        *range(1, longest, max(1, longest // 97))}):
        keys, blocks = cut(span, launch_keys, launch_blocks, spread, warps, tile)
        assert keys % tile == 0 and keys >= min(64, launch_keys) and 1 <= blocks <= launch_blocks
        assert (blocks - 1) * warps * keys < span <= blocks * warps * keys                   # those blocks hold all keys, and each some
        if span <= longest:
            most = launch_blocks if spread else -(-span // (launch_keys * warps))            # blocks that the launch's cut fills
            assert keys <= launch_keys and blocks <= most
            even = -(-span // (most * warps))
            assert keys <= max(min(64, launch_keys), -(-even // tile) * tile)                # nor a warp with more than its even part


def test_a_short_request_keeps_blocks_only_while_there_is_room(cut):
    # 21 requests of 512 to 3,500 keys, 8 kv heads: two blocks each do not find places at once, and a short request needs one
    assert cut(512, 320, 2, False, 6, 32) == (96, 1) and cut(3500, 320, 2, False, 6, 32) == (320, 2)
    # 4 requests, window 512: there is room for all
    assert cut(512, 64, 6, True, 6, 16) == (64, 2) and cut(512, 64, 2, True, 6, 16) == (64, 2)
