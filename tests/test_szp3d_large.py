"""The 3-D compressor on values that are large against the bound: an offset of
thousands to millions of steps, amplitudes and differences around the limits of
its float forms (2^22 and 2^24), bounds that are no floats, and values next to
the middles between steps."""
from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest


def test_quantization_forms_match_double(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    here = os.path.dirname(os.path.abspath(__file__))
    exe = tmp_path / "sz3_large"
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-o", str(exe), os.path.join(here, "native", "sz3_large.c"), "-lm"],
                   check=True)
    out = subprocess.run([str(exe), "100000"], capture_output=True, text=True, timeout=200)
    b0, t0, b1, t1, b2, t2, n = map(int, out.stdout.split())
    assert b0 == b1 == b2 == 0
    assert n > 5_000_000 and t0 > n // 4 and t1 > n // 4 and t2 > n // 4


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
@pytest.mark.parametrize("dims", [(20, 36, 68), (9, 17, 131)])
def test_large_values(port, bs, dims):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zccl_gb300.szp3d import Szp3D
    rng = np.random.default_rng(bs)
    n = int(np.prod(dims))
    smooth = np.cumsum(rng.normal(0, 1, dims), axis=2)
    codec = Szp3D(dims, bs)
    for eb in (0.5, 1e-3, 0.0123456789012345):
        for off in (0.0, 3e3, 1.5e5, 6e5, 4.19e6, 4.2e6, 1.6e7, 1.7e7):
            for amp in (3.0, 2e3, 2e5, 3e6):
                q = off + amp * smooth / np.abs(smooth).max()
                if amp == 2e3:  # on the middles between steps, or next to them
                    q = np.floor(q) + 0.5
                x = np.ascontiguousarray(q * 2 * eb, np.float32).ravel()
                if amp == 3e6:
                    x[rng.integers(0, n, 5)] = 0  # a few far from their neighbours
                want = port.szp3d_compress(x, dims, bs, eb)
                out, size = codec.compress(torch.from_numpy(x).cuda(), eb)
                codec.check()
                assert out[: codec.size(size)].cpu().numpy().tobytes() == want, (eb, off, amp)


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
def test_values_that_cannot_be_quantized(bs):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import zccl_gb300 as Z
    from zccl_gb300.szp3d import Szp3D
    dims = (10, 11, 70)
    codec = Szp3D(dims, bs)
    x = torch.zeros(dims, device="cuda")
    for at in ((0, 0, 0), (9, 10, 69), (4, 5, 33)):
        for v in (float("nan"), float("inf"), -float("inf"), 1e30):
            y = x.clone()
            y[at] = v
            codec.compress(y.reshape(-1), 1e-3)
            with pytest.raises(Z.ZcclError):
                codec.check()
    codec.compress(x.reshape(-1), 1e-3)
    codec.check()
