"""The block decoders read whole words of their staged bytes, some of them past
a block's end; the buffers' slack must cover all of it."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest


def test_reads_stay_within_the_slack(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    here = os.path.dirname(os.path.abspath(__file__))
    exe = tmp_path / "read_slack"
    subprocess.run([cc, "-O2", "-I", os.path.join(here, "..", "zccl_gb300", "csrc"), "-o", str(exe),
                    os.path.join(here, "native", "read_slack.c")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    checked, over = map(int, out.stdout.split())
    assert checked > 1_000_000 and over == 0
