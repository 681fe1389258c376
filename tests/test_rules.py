"""The index rules that kernels and launchers share (csrc/rules.h), compiled for the CPU."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "rules.h"
extern "C" {
uint32_t row_block(uint32_t row, uint32_t rows) { return tnf::sf_row_block(row, rows); }
uint32_t tile_n(uint32_t m, uint32_t n, uint32_t sms) { return tnf::tile_n_rule(m, n, sms); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "librules.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "thinfer_b200", "csrc"), "-o", str(so),
                    str(d / "shim.cpp")], check=True)
    return C.CDLL(str(so))


def test_no_tile_copies_scales_past_the_weight(rules):
    """The scale layout of W ends with the 128-row block of its last row: whatever the tile's width, every block that it copies
    is one of those, and the right one wherever W has rows."""
    past = 0
    for m in (1, 128, 129, 256, 385, 512, 1000, 9345, 18817, 18944, 40000):
        for n in (8, 64, 128, 136, 256, 264, 384, 9216, 9224, 9344, 9352, 18688, 18696, 18816, 37632, 37640, 37760, 37888, 40000):
            width = rules.tile_n(m, n, 148)
            blocks = (n + 127) // 128
            assert width in (64, 128, 256)
            assert width <= 128 or n > 128  # half of a 256-wide tile would be padding in every CTA
            for n0 in range(0, n, width):
                for j in range(max(1, width // 128)):
                    row = n0 + 128 * j
                    block = rules.row_block(row, n)
                    assert block < blocks
                    if row < n:
                        assert block == row // 128
                    past += row // 128 >= blocks
    assert past > 0  # there are shapes here whose last tile hangs over by a whole block
