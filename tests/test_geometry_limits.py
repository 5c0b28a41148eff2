"""Sizes of streams with very many chunks, from the geometry header that host and
device share, compiled as C: nothing is cut to 32 bits."""
from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "zccl_gb300", "csrc")

SOURCE = r"""
#include <stdio.h>
#include "zgeom.h"
int main(void)
{
    const uint32_t Ts[] = {1, 72, 1u << 20, (1u << 29) - 1, 1u << 29, (1u << 30) + 7, 0x7fffffffu};
    for (int k = 0; k < 7; k++) {
        ZGeom g;
        ZTile z;
        if (zg_init(&g, (uint64_t)Ts[k] * 3 + 1, 32, Ts[k])) return 1;
        zg_tile(&g, g.ntiles - 1, &z);
        printf("%llu %llu %llu\n", (unsigned long long)zg_header_bytes(&g), (unsigned long long)zg_stream_worst(&g),
               (unsigned long long)z.e_end);
    }
    return 0;
}
"""


def test_many_chunks(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    src, exe = tmp_path / "limits.c", tmp_path / "limits"
    src.write_text(SOURCE)
    subprocess.run([cc, "-O2", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split("\n")
    for line, T in zip(out, [1, 72, 1 << 20, (1 << 29) - 1, 1 << 29, (1 << 30) + 7, 0x7FFFFFFF]):
        header, worst, end = map(int, line.split())
        n = 3 * T + 1
        assert header == 8 * T and end == n
        if T == 1:  # a head and a block of three floats (width 32)
            assert worst == 8 + 4 + 1 + 1 + 12
        else:  # heads, a block of two floats each, and a last segment of one float
            assert worst == 8 * T + T * (4 + 1 + 1 + 8) + 4


def test_header_size_has_one_definition():
    """No kernel forms the header's size by itself (the placers' was 32 bits wide)."""
    for f in ("zkern.cuh", "zk_compress.cu", "zk_homadd.cu", "zk_decompress.cu", "zk_walk.cu"):
        assert not re.search(r"\b8u \* \w+(\.|->)T\b", open(os.path.join(CSRC, f)).read()), f
