"""Kernels' shared-memory limits only ever grow, on any number of devices and
from any thread: a call that wants less must not take from another thread's
launch what it counts on."""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "zccl_gb300", "csrc")


def test_limits_only_grow(tmp_path):
    cxx = shutil.which("g++")
    inc = next((d for d in ("/usr/local/cuda/include",) if os.path.exists(os.path.join(d, "cuda_runtime_api.h"))), None)
    if not cxx or not inc:
        pytest.skip("no C++ compiler or CUDA headers")
    exe = tmp_path / "launch_limits"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, "-I", inc, "-o", str(exe),
                    os.path.join(HERE, "native", "launch_limits.cpp"), "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.stdout.split() == ["0", "0", "0"]


def test_every_limit_goes_through_one_place():
    for f in glob.glob(os.path.join(CSRC, "*")):
        if not f.endswith("zlaunch.h"):
            assert "cudaFuncSetAttribute" not in open(f).read(), f


@pytest.mark.gpu
def test_threads_with_long_block_sides(port):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zccl_gb300.szp3d import Szp3D
    dims, eb, errors = (48, 40, 64), 1e-3, []
    v = np.random.default_rng(5).normal(0, 1, dims).astype(np.float32).ravel()
    want = {bs: port.szp3d_compress(v, dims, bs, eb) for bs in (12, 24, 32)}
    x = torch.from_numpy(v).cuda()
    torch.cuda.synchronize()

    def work(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                codecs = {bs: Szp3D(dims, bs) for bs in want}
                for i in range(40):
                    bs = (12, 24, 32)[(k + i) % 3]
                    out, size = codecs[bs].compress(x, eb)
                    n = codecs[bs].size(size)
                    codecs[bs].check()
                    assert out[:n].cpu().numpy().tobytes() == want[bs]
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
